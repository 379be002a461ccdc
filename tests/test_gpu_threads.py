"""The first device work of a thread is a kernel of this library into memory that is already there."""
import threading

import pytest
import torch

from open_transformers_b200.ops import functional as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["gemm", "attention"])
def test_first_call_of_a_thread(what):
    g = torch.Generator().manual_seed(0)
    a, b = (torch.randn(256, 128, generator=g).bfloat16().cuda() for _ in range(2))
    qk, qkv = (torch.randn(128, n * 64, generator=g).bfloat16().cuda() for n in (2, 3))

    def call():
        if what == "gemm":
            return (K.gemm(a, b, out=out),)
        return K.attn_fwd(qk, qkv, 1, 128, 1, 1, 64, 0)  # (its outputs come from the allocator's cache)

    out = torch.empty(256, 256, dtype=torch.bfloat16, device="cuda")
    want = [t.clone() for t in call()]
    torch.cuda.synchronize()
    got = []

    def run():
        try:
            got.append([t.clone() for t in call()])
            torch.cuda.synchronize()
        except Exception as e:
            got.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    assert not isinstance(got[0], Exception), got[0]
    assert all(torch.equal(x, y) for x, y in zip(got[0], want))
