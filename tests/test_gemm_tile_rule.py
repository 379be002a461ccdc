"""The rule that chooses a product's tile, asked on the host for 148 SMs: where CTA pairs (512) take over from single CTAs."""
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
