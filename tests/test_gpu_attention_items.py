"""More attention work items than SMs on a GPU, so that every CTA walks several: bit for bit against the CPU twin, for any
order of the items."""
import pytest
import torch

from open_transformers_b200.ops import functional as K
from open_transformers_b200.ops.native import cuda_lib

pytestmark = pytest.mark.gpu


# one pair of tiles per head; a lone last tile (its partner's warps sit the item out); a window that skips key blocks; several
# items of a single key block, whole and ragged, on every CTA
@pytest.mark.parametrize("B,T,H,Hkv,D,window", [(90, 192, 4, 2, 64, 0), (40, 320, 4, 4, 64, 96), (33, 384, 6, 2, 128, 128), (200, 64, 4, 4, 64, 0),
                                                (120, 100, 4, 2, 128, 0)])
def test_many_items(B, T, H, Hkv, D, window):
    g = torch.Generator().manual_seed(T)
    qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).to(torch.bfloat16) for n in (H + Hkv, H + 2 * Hkv, H))

    def run(dev):
        a, b, d = qk.to(dev), qkv.to(dev), dO.to(dev)
        O, lse = K.attn_fwd(a, b, B, T, H, Hkv, D, window)
        dqk, dqkv = torch.zeros_like(a), torch.zeros_like(b)
        K.attn_bwd(a, b, O, d, lse, dqk, dqkv, B, T, H, Hkv, D, window)
        return [t.cpu() for t in (O, lse, dqk, dqkv)]

    want = run("cpu")
    try:
        for rotation in (0, 1, 2**31 - 1):  # (the last: the sum of item and rotation needs all 32 bits)
            assert cuda_lib().otb_set_attn_rotation(rotation) == 0
            for got, ref in zip(run("cuda"), want):
                assert torch.equal(got, ref)
    finally:
        cuda_lib().otb_set_attn_rotation(0)
    assert K.kernel_status("cuda") == 0
