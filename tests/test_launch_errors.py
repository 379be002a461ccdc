"""What an entry point returns when a launch is refused, against a fake runtime: an early launch that is refused is tried in the
ordinary way; an error is returned by the call whose launch it was, once, and nothing that depends on that launch follows it. And
which launches are early: products, memory-bound kernels, the attention forward on half the chip, dQ beside dK/dV."""
import pytest
from fake_cudart import run_with_fake

HEAD = r"""
import ctypes, sys
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
N, P = ctypes.c_void_p(0), ctypes.c_void_p(256)
I, L, F = ctypes.c_int, ctypes.c_long, ctypes.c_float
ORDINARY, EARLY = 0, 1

def attn_fwd(D=128, T=128):
    return lib.otb_attn_fwd(P, L(6 * D), P, L(8 * D), P, L(4 * D), P, I(1), I(T), I(4), I(2), I(D), I(0), F(1.0), N, N)

def attn_bwd(D=128, T=128):
    return lib.otb_attn_bwd(P, L(6 * D), P, L(8 * D), P, L(4 * D), P, L(4 * D), P, P, P, L(6 * D), P, L(8 * D), I(1), I(T), I(4), I(2), I(D), I(0),
                            F(1.0), N, N)

def rmsnorm_bwd(rows=64, gain=P):
    return lib.otb_rmsnorm_bwd(P, P, P, P, P, gain, L(rows), I(256), F(1.0), I(1), N)

def head_rmsnorm_bwd(rows=64):
    return lib.otb_head_rmsnorm_bwd(P, L(512), P, L(512), P, P, P, L(512), P, L(rows), I(4), I(128), F(1.0), I(1), N)

def gemm(M=128):
    return lib.otb_gemm_bf16(P, P, P, N, I(M), I(512), I(1024), L(1024), L(1024), L(512), L(0), I(0), I(0), I(0), N, I(0), N)

single = {
    "rmsnorm_fwd": lambda: lib.otb_rmsnorm_fwd(P, P, P, P, L(8), I(256), F(1.0), F(1.0), I(1), N),
    "rmsnorm_fwd_fp32": lambda: lib.otb_rmsnorm_fwd(P, P, P, P, L(8), I(256), F(1.0), F(1.0), I(0), N),
    "rmsnorm_bwd": lambda: rmsnorm_bwd(8, N),
    "head_rmsnorm_fwd": lambda: lib.otb_head_rmsnorm_fwd(P, L(512), P, P, L(512), P, L(8), I(4), I(128), F(1.0), F(1.0), I(1), N),
    "pair_tree_cols": lambda: lib.otb_pair_tree_cols(P, L(8), I(64), N),
    "qknorm_rope_fwd": lambda: lib.otb_qknorm_rope_fwd(P, L(512), P, L(512), P, P, P, L(8), I(4), I(128), I(8), I(1), F(1.0), F(1.0), I(1), N),
    "qknorm_rope_bwd": lambda: lib.otb_qknorm_rope_bwd(P, L(512), P, L(512), P, P, L(512), P, P, L(8), I(4), I(128), I(8), I(1), F(1.0), I(1), N),
    "swiglu_fwd": lambda: lib.otb_swiglu_fwd(P, P, L(8), I(64), I(1), N),
    "swiglu_bwd": lambda: lib.otb_swiglu_bwd(P, P, P, L(8), I(64), I(1), N),
    "ce_zloss": lambda: lib.otb_ce_zloss(P, P, P, P, L(8), I(64), F(1.0), F(1.0), I(1), I(1), N),
    "det_sum": lambda: lib.otb_det_sum(P, L(8), I(0), F(1.0), P, N),
    "embedding_fwd": lambda: lib.otb_embedding_fwd(P, P, P, L(8), I(64), I(1), N),
    "attn_fwd": attn_fwd,
    "attn_fwd_64": lambda: attn_fwd(64),
    "gemm": gemm,
}
"""

# a single launch: refused early only, then both ways; the next call is not charged with it
ONE = HEAD + r"""
for name, call in single.items():
    early = name != "embedding_fwd"
    fake.fake_reset()
    assert call() == 0 and (fake.fake_launched(), fake.fake_launched_early()) == (1, early), name
    fake.fake_reset()
    fake.fake_refuse_launch(EARLY, 0, 1, 801)
    assert call() == 0 and (fake.fake_launched(), fake.fake_launched_early()) == (1, 0), name
    fake.fake_reset()
    fake.fake_refuse_launch(EARLY, 0, 1, 801)
    fake.fake_refuse_launch(ORDINARY, 0, 1, 701)
    assert call() == 701 and fake.fake_launched() == 0, name
    assert fake.fake_pending() == 0, name
    fake.fake_reset()
    assert call() == 0, name
for T, early in ((18 * 256, True), (18 * 256 + 1, False), (64 * 256, False)):  # 4 heads: 72, 76 and 256 pairs of query tiles, 148 SMs
    fake.fake_reset()
    assert attn_fwd(128, T) == attn_fwd(64, T) == 0 and fake.fake_launched_early() == 2 * early, T
for M in (1, 4096, 148 * 128):
    fake.fake_reset()
    assert gemm(M) == 0 and fake.fake_launched_early() == 1, M
fake.fake_reset()
fake.fake_refuse_launch(EARLY, 0, 1, 701)  # a CTA pair's launch has a cluster attribute and no second try
assert gemm(1 << 16) == 701 and fake.fake_pending() == 0
print("ok")
"""

# several launches: whichever is refused, the call returns its code and launches nothing behind it, also where a later early
# launch would be refused and repeated
SEVERAL = HEAD + r"""
for D in (64, 128):
    for T in (128, 100):  # whole and ragged steps
        fake.fake_reset()
        assert attn_bwd(D, T) == 0 and (fake.fake_launched(), fake.fake_launched_early()) == (3, 1)
        fake.fake_reset()
        fake.fake_refuse_launch(EARLY, 0, 1, 801)
        assert attn_bwd(D, T) == 0 and (fake.fake_launched(), fake.fake_launched_early()) == (3, 0)
        for nth in range(3):
            fake.fake_reset()
            fake.fake_refuse_launch(EARLY, 0, 2, 801)
            fake.fake_refuse_launch(ORDINARY, nth, 1, 701)
            assert attn_bwd(D, T) == 701 and fake.fake_launched() == nth and fake.fake_pending() == 0, (D, T, nth)
        fake.fake_reset()
        fake.fake_refuse_launch(EARLY, 0, 1, 801)
        fake.fake_refuse_launch(ORDINARY, 1, 1, 701)  # dK/dV by itself
        assert attn_bwd(D, T) == 701 and fake.fake_launched() == 1 and fake.fake_pending() == 0, (D, T)
for call, rows in ((rmsnorm_bwd, 64), (rmsnorm_bwd, 8 * 1200), (head_rmsnorm_bwd, 64), (head_rmsnorm_bwd, 16 * 1200)):
    fake.fake_reset()
    assert call(rows) == 0
    launches = fake.fake_launched()
    assert fake.fake_launched_early() == launches
    assert launches == (2 if rows == 64 else 3)
    for nth in range(launches):
        fake.fake_reset()
        fake.fake_refuse_launch(EARLY, 0, 8, 801)
        fake.fake_refuse_launch(ORDINARY, nth, 1, 701)
        assert call(rows) == 701 and fake.fake_launched() == nth and fake.fake_pending() == 0, (call.__name__, rows, nth)
print("ok")
"""


# threads by the width of a row: some at every width, no columns at all among them
WIDTHS = HEAD + r"""
for D in (0, 8, 12, 248, 256, 264, 2040, 2048, 2056, 1 << 20):
    for bf16 in (0, 1):
        fake.fake_reset()
        assert lib.otb_embedding_bwd(P, P, P, L(8), P, I(D), I(1), I(bf16), N) == 0 and fake.fake_launched() == 1, D
        assert lib.otb_ce_zloss(P, P, P, P, L(8), I(D // 8 * 8), F(1.0), F(1.0), I(1), I(bf16), N) == 0 and fake.fake_launched() == 2, D
print("ok")
"""


@pytest.mark.parametrize("child", [ONE, SEVERAL, WIDTHS], ids=["one launch", "several launches", "widths"])
def test_refused_launches(child, tmp_path):
    run_with_fake(child, tmp_path)
