"""Attention forward and backward where a step, a half step or a sequence ends: bit for bit against the CPU twin."""
import pytest
import torch

from open_transformers_b200.ops import functional as K

pytestmark = pytest.mark.gpu


# one row; just below and above a half step and a step; a window whose edge falls in either half of a step, and inside a 16-query piece
@pytest.mark.parametrize("T", [1, 16, 63, 65, 127, 129, 192, 255, 321, 515])
@pytest.mark.parametrize("H,Hkv,D,window", [(4, 2, 64, 0), (4, 4, 64, 96), (2, 1, 128, 0), (4, 2, 128, 64), (2, 2, 128, 160)])
def test_step_edges(T, H, Hkv, D, window):
    B = 2
    g = torch.Generator().manual_seed(T * 8 + D + window)
    qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).to(torch.bfloat16) for n in (H + Hkv, H + 2 * Hkv, H))

    def run(dev):
        a, b, d = qk.to(dev), qkv.to(dev), dO.to(dev)
        O, lse = K.attn_fwd(a, b, B, T, H, Hkv, D, window)
        dqk, dqkv = torch.zeros_like(a), torch.zeros_like(b)
        K.attn_bwd(a, b, O, d, lse, dqk, dqkv, B, T, H, Hkv, D, window)
        return [t.cpu() for t in (O, lse, dqk, dqkv)]

    for got, ref in zip(run("cuda"), run("cpu")):
        assert torch.equal(got, ref)
    assert K.kernel_status("cuda") == 0


def test_int8_probabilities_are_rounded_twice():
    """127 p is rounded before it is rounded to an integer: a fused multiply-add differs in a few of these 4 M probabilities."""
    B, T, H, D = 1, 1000, 4, 128
    g = torch.Generator().manual_seed(1)
    qk, qkv = torch.randn(B * T, 2 * H * D, generator=g).to(torch.bfloat16), torch.randn(B * T, 3 * H * D, generator=g).to(torch.bfloat16)
    for window in (0, 512):
        got = K.attn_fwd(qk.cuda(), qkv.cuda(), B, T, H, H, D, window, int8_pv=True)
        for x, ref in zip(got, K.attn_fwd(qk, qkv, B, T, H, H, D, window, int8_pv=True)):
            assert torch.equal(x.cpu(), ref)
