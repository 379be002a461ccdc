"""Fast forms of kernels at the edges of what chooses them, bit for bit against the CPU twin."""
import ctypes

import pytest
import torch

from open_transformers_b200.ops import functional as K
from open_transformers_b200.ops.native import cuda_lib

pytestmark = pytest.mark.gpu


# every 16-byte piece whole (predicated loads): one size per tile, rows ragged against the tile, K below, at and past a slab
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K_", [(4, 36, 4), (36, 60, 32), (100, 260, 68), (772, 900, 36), (2308, 2312, 20)])
def test_exact_gemm_of_whole_pieces(a_mn, b_mn, M, N, K_):
    g = torch.Generator().manual_seed(M + K_)
    a = torch.randn((K_, M) if a_mn else (M, K_), generator=g)
    b = torch.randn((K_, N) if b_mn else (N, K_), generator=g)
    acc = torch.randn(M, N, generator=g)
    assert torch.equal(K.gemm(a.cuda(), b.cuda(), a_mn=a_mn, b_mn=b_mn).cpu(), K.gemm(a, b, a_mn=a_mn, b_mn=b_mn))
    assert torch.equal(K.gemm(a.cuda(), b.cuda(), a_mn=a_mn, b_mn=b_mn, epi=K.EPI_ACC_F32, out=acc.cuda()).cpu(),
                       K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, epi=K.EPI_ACC_F32, out=acc.clone()))


# values on and one step beside every tie k + 1/2, NaN, both zeros; steps in and out of the range of the fast division
# (2^-80 .. 2^100), a subnormal and an infinite one; lengths with and without a ragged end
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("qmax", [127, 7, 1])
@pytest.mark.parametrize("top", [1.0, 3.1415927, 2.0**-70, 127 * 2.0**-80, 2.0**-90, 2.0**-130, 2.0**100, 2.0**120, float("inf")])
def test_quantiser_near_ties(dtype, qmax, top):
    step = torch.tensor(top, dtype=torch.float32) * torch.tensor(1.0 / qmax, dtype=torch.float32)
    k = torch.arange(-qmax, qmax, dtype=torch.float32) + 0.5
    ties = k * step if top < float("inf") else k
    x = torch.cat([ties, torch.nextafter(ties, ties * 2), torch.nextafter(ties, ties * 0), torch.tensor([0.0, -0.0, 1e-40, float("nan")]),
                   torch.linspace(-1, 1, 1001) * min(top, 3e38)]).clamp(-min(top, 3.3e38), min(top, 3.3e38)).to(dtype)
    x = torch.cat([x, torch.tensor([top, -top]).to(dtype)])
    for n in (x.numel(), x.numel() // 8 * 8):
        part = x[-n:].contiguous()
        q, s = K.quant_act(part.cuda(), qmax)
        want_q, want_s = K.quant_act(part, qmax)
        assert torch.equal(s.cpu(), want_s)
        keep = ~part.isnan() & ~part.isinf()  # (what the quotient NaN becomes is the platform's conversion)
        assert torch.equal(q.cpu()[keep], want_q[keep])


# A NaN becomes -qmax wherever it lies, in a whole group of eight or in the ragged end, with a step in or out of the range of the
# fast division, and leaves its neighbours alone.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("top", [3.0, 2.0**-90, 2.0**120])
def test_quantiser_of_nan(dtype, top):
    x = (torch.linspace(-1, 1, 8 * 300 + 5) * top).to(dtype)
    at = torch.tensor([0, 3, 7, 8, 8 * 150 + 4, 8 * 300 - 1, 8 * 300, 8 * 300 + 4])
    x[at] = float("nan")
    q, s = K.quant_act(x.cuda(), 127)
    want_q, want_s = K.quant_act(x, 127)
    assert torch.equal(s.cpu(), want_s) and (q.cpu()[at] == -127).all()
    rest = ~x.isnan()
    assert torch.equal(q.cpu()[rest], want_q[rest])


# 64-wide tiles where all of them fit the chip at once: one tile, ragged columns and rows, a K of one step and of many, the
# last size of one wave of them (rows of four tiles each, by the device's SM count) and the first past it; more than 32 columns of
# them on 128 KB of A and on less
@pytest.mark.parametrize("M,N,K_,slim", [(1, 8, 8, True), (130, 200, 64, True), (129, 72, 520, True), ("wave", 256, 72, True), ("wave + 1", 256, 72, False),
                                            (32, 2056, 2048, True), (24, 2056, 2048, False)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_slim_gemm_tiles(M, N, K_, slim, a_mn, b_mn):
    if isinstance(M, str):
        M = torch.cuda.get_device_properties(0).multi_processor_count // 4 * 128 + (M == "wave + 1")
    g = torch.Generator().manual_seed(M + K_)
    Mr = (M + 7) // 8 * 8 if a_mn else M  # (a row pitch is a multiple of 16 bytes)
    tile = cuda_lib().otb_gemm_tile(*(ctypes.c_int(v) for v in (Mr, N, K_, a_mn or b_mn, 0, 0)))
    assert (tile == 64) == slim
    a = torch.randn((K_, Mr) if a_mn else (M, K_), generator=g).bfloat16()
    b = torch.randn((K_, N) if b_mn else (N, K_), generator=g).bfloat16()
    for epi in (K.EPI_STORE, K.EPI_STORE_F32, K.EPI_ACC_F32, K.EPI_RESIDUAL):
        kw = {"epi": epi}
        rows = Mr if a_mn else M
        out = torch.randn(rows, N, generator=g) if epi == K.EPI_ACC_F32 else None
        res = torch.randn(rows, N, generator=g).bfloat16() if epi == K.EPI_RESIDUAL else None
        want = K.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=None if out is None else out.clone(), residual=res, **kw)
        got = K.gemm(a.cuda(), b.cuda(), a_mn=a_mn, b_mn=b_mn, out=None if out is None else out.cuda(), residual=None if res is None else res.cuda(), **kw)
        assert torch.equal(got.cpu(), want)
    assert K.kernel_status("cuda") == 0
