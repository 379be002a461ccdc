"""Products that run on CTA pairs (256 x 256 tiles of two SMs) on a GPU: bit for bit against the CPU twin."""
import pytest
import torch

from open_transformers_b200.ops import functional as K
from open_transformers_b200.ops.native import cuda_lib

pytestmark = pytest.mark.gpu
PAIR = 512  # otb_gemm_tile's answer for CTA pairs


# 256-row tiles whose second CTA holds few, no or all rows; ragged column tiles; one K step, a ragged one, more than the ring
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
# (the K up to 512 run the same results on single CTAs)
@pytest.mark.parametrize("M,N,K_", [(2304, 4864, 8), (2104, 5008, 72), (2184, 5120, 64), (2056, 9480, 48), (2304, 4872, 456),
                                    (2304, 4864, 520), (2104, 5008, 576), (2056, 9480, 584), (2304, 4872, 1000)])
def test_bf16_pairs(a_mn, b_mn, M, N, K_):
    g = torch.Generator().manual_seed(K_)
    a, b = torch.randn(M, K_, generator=g).bfloat16(), torch.randn(N, K_, generator=g).bfloat16()
    assert (cuda_lib().otb_gemm_tile(M, N, K_, a_mn or b_mn, 0, 0) == PAIR) == (K_ > 512)
    want = K.gemm(a, b, epi=K.EPI_STORE_F32)
    ac, bc = (t.t().contiguous().cuda() if mn else t.cuda() for t, mn in ((a, a_mn), (b, b_mn)))
    kw = dict(a_mn=a_mn, b_mn=b_mn)
    assert torch.equal(K.gemm(ac, bc, epi=K.EPI_STORE_F32, **kw).cpu(), want)
    assert torch.equal(K.gemm(ac, bc, **kw).cpu(), want.bfloat16())
    res = torch.randn(M, N, generator=g).bfloat16()
    assert torch.equal(K.gemm(ac, bc, epi=K.EPI_RESIDUAL, residual=res.cuda(), **kw).cpu(), (want + res.float()).bfloat16())
    big = torch.full((M + 2, N + 16), 7.0, device="cuda")  # a strided result: nothing outside it is touched
    K.gemm(ac, bc, out=big[1:M + 1, 8:N + 8], epi=K.EPI_ACC_F32, **kw)
    assert torch.equal(big[1:M + 1, 8:N + 8].cpu(), want + 7.0)
    big[1:M + 1, 8:N + 8] = 7.0
    assert bool((big == 7.0).all()) and K.kernel_status("cuda") == 0


@pytest.mark.parametrize("M,N,K_", [(2100, 5008, 144), (2304, 4864, 16), (2049, 9480, 1040), (2100, 5008, 1552), (2304, 4872, 1680), (2049, 9480, 1664)])
def test_int8_pairs(M, N, K_):
    assert (cuda_lib().otb_gemm_tile(M, N, K_, 0, 1, 0) == PAIR) == (K_ > 1536)
    g = torch.Generator().manual_seed(N)
    a, b = (torch.randint(-127, 128, (r, K_), dtype=torch.int8, generator=g) for r in (M, N))
    sa, sb = torch.rand(1, generator=g) * 0.01, torch.rand(N, generator=g) * 0.01
    res = torch.randn(M, N, generator=g).bfloat16()
    dev = [t.cuda() for t in (a, b, sa, sb)]
    for dtype in (torch.float32, torch.bfloat16):
        assert torch.equal(K.gemm_i8(*dev, dtype).cpu(), K.gemm_i8(a, b, sa, sb, dtype))
    assert torch.equal(K.gemm_i8(*dev, torch.bfloat16, res.cuda()).cpu(), K.gemm_i8(a, b, sa, sb, torch.bfloat16, res))
    assert K.kernel_status("cuda") == 0


# The shortest pipelines, one tile per pair and launches back to back: a pair has to leave nothing under way behind it (the
# arrivals that release its last stages would land in the shared memory of the pair that follows). K steps of 64 around one and
# a half and two turns of the ring of six, with and without a ragged last one.
@pytest.mark.parametrize("K_", [520, 576, 640, 704, 768, 776])
def test_pairs_that_follow_one_another(K_):
    g = torch.Generator().manual_seed(K_)
    M, N = 2 * 256, 37 * 256  # 74 tiles: one per pair of 148 SMs
    assert cuda_lib().otb_gemm_tile(M, N, K_, 0, 0, 0) == PAIR
    a, b = (torch.randn(r, K_, generator=g).bfloat16() for r in (M, N))
    want = K.gemm(a, b, epi=K.EPI_STORE_F32)
    ac, bc = a.cuda(), b.cuda()
    outs = [torch.empty(M, N, device="cuda") for _ in range(8)]
    for _ in range(25):
        for out in outs:
            K.gemm(ac, bc, epi=K.EPI_STORE_F32, out=out)
    assert all(torch.equal(out.cpu(), want) for out in outs)
    assert K.kernel_status("cuda") == 0


@pytest.mark.parametrize("M,N,pair", [(512, 9472, True), (300, 704, False)])
def test_any_order_of_the_tiles(M, N, pair):
    assert (cuda_lib().otb_gemm_tile(M, N, 520, 0, 0, 0) == PAIR) == pair
    g = torch.Generator().manual_seed(N)
    a, b = (torch.randn(r, 520, generator=g).bfloat16() for r in (M, N))
    want, ac, bc = K.gemm(a, b), a.cuda(), b.cuda()
    try:
        for rotation in (1, 2**31 - 1):  # (the last: the sum of block and rotation needs all 32 bits)
            assert cuda_lib().otb_set_cta_rotation(rotation) == 0
            assert torch.equal(K.gemm(ac, bc).cpu(), want)
    finally:
        assert cuda_lib().otb_set_cta_rotation(0) == 0
    assert K.kernel_status("cuda") == 0
