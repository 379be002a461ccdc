"""The rule that chooses a product's tile, asked on the host for 148 SMs: where CTA pairs (512) take over from single CTAs, and
where 64-wide tiles, which have to fit the chip in one wave, take over from wider ones."""
import pytest

from open_transformers_b200 import build_native
from open_transformers_b200.ops.native import cuda_lib

PAIR = 512


@pytest.mark.parametrize("M,N,K,mn,i8,pair", [
    (16384, 5632, 512, 0, 0, False), (16384, 5632, 520, 0, 0, True),      # few K steps: the stores are the time
    (16384, 5632, 1536, 0, 1, False), (16384, 5632, 1552, 0, 1, True),    # the same as int8
    (16384, 1408, 256, 0, 0, False), (16384, 1408, 256, 1, 0, False),     # the 256-wide feed-forward sublayer
    (512, 9216, 2048, 0, 0, False), (512, 9472, 2048, 0, 0, True),        # 72 and 74 pair tiles: one wave is 74
    (16384, 128, 2048, 0, 0, False), (16384, 256, 2048, 0, 0, False),     # narrow results: the padding, less than a wave
    (16384, 2048, 7448, 1, 0, True), (16384, 2048, 7456, 1, 0, False),    # 5e11 operations with an MN-major operand
    (16384, 2048, 7456, 0, 0, True), (16384, 128256, 2048, 0, 0, True),   # no such limit without one
])
def test_where_pairs_begin(M, N, K, mn, i8, pair):
    if not (build_native.EXT / "libotb_cuda.so").exists():
        pytest.skip("the CUDA library is not built here")
    tile = cuda_lib().otb_gemm_tile(M, N, K, mn, i8, 148)
    assert (tile == PAIR) == pair and tile in (128, 256, PAIR)


def test_no_pairs_on_one_cta():
    if not (build_native.EXT / "libotb_cuda.so").exists():
        pytest.skip("the CUDA library is not built here")
    assert cuda_lib().otb_gemm_tile(16384, 5632, 2048, 0, 0, 1) in (128, 256)


@pytest.mark.parametrize("mn", [0, 1])
@pytest.mark.parametrize("M,N,K,sms,slim", [
    (1, 8, 8, 148, True), (333, 768, 768, 148, True), (1111, 768, 2048, 148, True),           # 1, 36 and 108 tiles
    (37 * 128, 256, 72, 148, True), (37 * 128 + 1, 256, 72, 148, False),                       # 148 tiles, and one row more
    (128, 148 * 64, 2048, 148, True), (128, 148 * 64 + 8, 2048, 148, False),                   # 148, and eight columns more
    (1, 2048, 8, 148, True), (16, 2048, 768, 148, True), (1, 2056, 2048, 148, False),          # 32 columns of tiles, and 33
    (31, 4096, 2048, 148, False), (32, 4096, 2048, 148, True), (16, 4096, 4096, 148, True),    # 33 and more: from 128 KB of A on
    (16, 4096, 768, 148, False), (85, 5632, 768, 148, False), (86, 5632, 768, 148, True),
    (148 * 128, 64, 64, 148, True), (148 * 128, 72, 64, 148, False),                           # narrow results of many rows
    (128, 64, 64, 1, True), (128, 72, 64, 1, False), (333, 768, 768, 35, False), (333, 768, 768, 36, True),  # a capped grid
])
def test_where_slim_tiles_end(M, N, K, sms, slim, mn):
    if not (build_native.EXT / "libotb_cuda.so").exists():
        pytest.skip("the CUDA library is not built here")
    assert (cuda_lib().otb_gemm_tile(M, N, K, mn, 0, sms) == 64) == slim
    assert cuda_lib().otb_gemm_tile(M, N, K, 0, 1, sms) != 64  # int8 products keep their tiles
