"""Which exact fp32 products load by predicate: asked of the library's host code, against a fake runtime of 148 SMs. The kernel
that a product with unaligned operands launches is the one with branches."""
from fake_cudart import run_with_fake

CHILD = r"""
import ctypes, sys
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
fake.fake_last.restype = ctypes.c_void_p
I, L, P = ctypes.c_int, ctypes.c_long, ctypes.c_void_p

def kernel(M, N, K, a_mn, b_mn, epi, base):
    assert lib.otb_gemm_f32(P(base), P(base), P(4096), P(4096), I(M), I(N), I(K), L(M if a_mn else K), L(N if b_mn else K), L(N), L(N), I(a_mn),
                            I(b_mn), I(epi), P(0)) == 0
    return fake.fake_last()

STORE, ACC, RES = 1, 2, 3
for M, N, K, a_mn, b_mn, epi, predicated in [
    (256, 704, 2048, 1, 1, STORE, 1), (256, 704, 2048, 1, 1, ACC, 1), (256, 704, 2048, 0, 0, STORE, 0),   # 32-wide tiles
    (2048, 1024, 256, 1, 1, STORE, 1), (1336, 1736, 696, 1, 1, STORE, 1), (1024, 1024, 256, 1, 1, STORE, 1),  # 64-wide: 512, 588, 256 tiles
    (768, 2048, 1000, 1, 1, STORE, 0), (1024, 1408, 256, 1, 1, STORE, 0), (2048, 1408, 256, 1, 1, STORE, 0),  # 384, 352, 704
    (2048, 1792, 256, 1, 1, STORE, 0), (2048, 2304, 256, 1, 1, STORE, 0),                                     # 896, 1152
    (768, 2048, 1000, 1, 1, ACC, 1), (2048, 1408, 256, 1, 1, ACC, 1),
    (768, 2048, 1000, 0, 0, STORE, 1), (2048, 1408, 256, 0, 0, RES, 1), (768, 2048, 1000, 0, 0, ACC, 0), (2048, 1408, 256, 0, 0, ACC, 0),
    (4096, 4096, 512, 1, 1, STORE, 1), (4096, 4096, 512, 1, 1, ACC, 0), (4096, 4096, 512, 0, 0, STORE, 0),    # 128-wide
    (2048, 256, 1408, 0, 1, STORE, 0), (2048, 1408, 256, 1, 0, STORE, 0), (4096, 4096, 512, 0, 1, STORE, 0)]:
    same = kernel(M, N, K, a_mn, b_mn, epi, 4096) == kernel(M, N, K, a_mn, b_mn, epi, 4100)
    assert same != predicated, (M, N, K, a_mn, b_mn, epi)
print("ok")
"""


def test_which_products_load_by_predicate(tmp_path):
    run_with_fake(CHILD, tmp_path)
