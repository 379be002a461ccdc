"""Exact fp32 family on a GPU at the edges of its tiles: bit for bit against the CPU twin."""
import pytest
import torch

from open_transformers_b200.ops import functional as K

pytestmark = pytest.mark.gpu


def _same(dev, host, what):
    assert torch.equal(dev.cpu(), host), what


# one shape per tile size (32, 64 and 128 wide: the rule counts tiles against the SMs), ragged in every direction; ``pad``
# makes the row pitch no multiple of four elements, which takes the scalar loads
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K_,pad", [(33, 31, 5, 0), (65, 130, 67, 3), (770, 900, 33, 0), (2309, 2311, 17, 0), (2309, 2311, 18, 1),
                                        (1180, 1155, 37, 0), (1180, 1155, 70, 1)])  # (64-wide tiles, three to an SM)
def test_gemm_tiles(a_mn, b_mn, M, N, K_, pad):
    g = torch.Generator().manual_seed(M + K_)

    def operand(r, c):
        return torch.randn(r, c + pad, generator=g)[:, :c]

    a = operand(K_, M) if a_mn else operand(M, K_)
    b = operand(K_, N) if b_mn else operand(N, K_)
    res, acc = torch.randn(M, N, generator=g), torch.randn(M, N, generator=g)
    da, db = (torch.empty(t.shape[0], t.shape[1] + pad, device="cuda")[:, : t.shape[1]].copy_(t) for t in (a, b))
    _same(K.gemm(da, db, a_mn=a_mn, b_mn=b_mn), K.gemm(a, b, a_mn=a_mn, b_mn=b_mn), "store")
    _same(K.gemm(da, db, a_mn=a_mn, b_mn=b_mn, epi=K.EPI_RESIDUAL, residual=res.cuda()),
          K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, epi=K.EPI_RESIDUAL, residual=res), "residual")
    _same(K.gemm(da, db, a_mn=a_mn, b_mn=b_mn, epi=K.EPI_ACC_F32, out=acc.cuda()),
          K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, epi=K.EPI_ACC_F32, out=acc.clone()), "accumulate")


@pytest.mark.parametrize("B,T,H,Hkv,D,window", [(1, 1, 1, 1, 4, 0), (2, 63, 2, 1, 64, 0), (1, 65, 4, 2, 48, 0), (1, 200, 2, 2, 128, 0),
                                                (1, 129, 2, 1, 72, 32), (2, 300, 2, 1, 64, 96), (1, 330, 1, 1, 6, 128),
                                                # one warp per row up to 31 (backward) and 40 (forward) tokens, tiles above; with more heads
                                                # than SMs up to 8 and 16
                                                (3, 5, 4, 2, 64, 0), (2, 31, 2, 1, 128, 8), (2, 32, 4, 1, 40, 0), (1, 40, 2, 2, 6, 32), (2, 41, 3, 1, 64, 16),
                                                (120, 8, 4, 2, 16, 0), (120, 9, 4, 2, 16, 3), (120, 16, 2, 1, 64, 0), (120, 17, 2, 2, 8, 0)])
def test_attention_tiles(B, T, H, Hkv, D, window):
    g = torch.Generator().manual_seed(T + D)
    qk = torch.randn(B * T, (H + Hkv) * D, generator=g)
    qkv = torch.randn(B * T, (H + 2 * Hkv) * D, generator=g)
    dO = torch.randn(B * T, H * D, generator=g)

    def both(qk_, qkv_, dO_):
        O, lse = K.attn_fwd(qk_, qkv_, B, T, H, Hkv, D, window)
        dqk, dqkv = torch.zeros_like(qk_), torch.zeros_like(qkv_)
        K.attn_bwd(qk_, qkv_, O, dO_, lse, dqk, dqkv, B, T, H, Hkv, D, window)
        return O, lse, dqk, dqkv

    for dev, host, what in zip(both(qk.cuda(), qkv.cuda(), dO.cuda()), both(qk, qkv, dO), ("O", "lse", "dqk", "dqkv")):
        _same(dev, host, what)
