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


# the rows that fill up a step after the last query; in the last 16 queries, or whole pieces and a whole half of nothing else
@pytest.mark.parametrize("T", [33, 80, 129, 200, 333])
@pytest.mark.parametrize("H,Hkv,D,window", [(4, 2, 64, 0), (2, 1, 128, 40)])
def test_infinite_key_beside_padding(T, H, Hkv, D, window):
    """The last key holds an infinity that its one query turns into a score of -inf: everything but that query's own gradient stays
    finite. (Scores of the padding against that key are NaN; the exponential's clamp makes 2^-126 of them, which meets rows of zeros.)"""
    B = 2
    g = torch.Generator().manual_seed(T + D)
    qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).to(torch.bfloat16) for n in (H + Hkv, H + 2 * Hkv, H))
    last = qk.view(B, T, H + Hkv, D)[:, T - 1]
    last[:, :H, 5], last[:, H:, 5] = -1.0, float("inf")

    def run(dev):
        a, b, d = qk.to(dev), qkv.to(dev), dO.to(dev)
        O, lse = K.attn_fwd(a, b, B, T, H, Hkv, D, window)
        dqk, dqkv = torch.zeros_like(a), torch.zeros_like(b)
        K.attn_bwd(a, b, O, d, lse, dqk, dqkv, B, T, H, Hkv, D, window)
        return [t.cpu() for t in (O, lse, dqk[:, H * D:], dqkv)]

    for got, ref in zip(run("cuda"), run("cpu")):
        assert ref.isfinite().all() and torch.equal(got, ref)


def test_int8_probabilities_are_rounded_twice():
    """127 p is rounded before it is rounded to an integer: a fused multiply-add differs in a few of the 2.0 M visible probabilities (1.5 M
    with the window)."""
    B, T, H, D = 1, 1000, 4, 128
    g = torch.Generator().manual_seed(1)
    qk, qkv = torch.randn(B * T, 2 * H * D, generator=g).to(torch.bfloat16), torch.randn(B * T, 3 * H * D, generator=g).to(torch.bfloat16)
    for window in (0, 512):
        got = K.attn_fwd(qk.cuda(), qkv.cuda(), B, T, H, H, D, window, int8_pv=True)
        for x, ref in zip(got, K.attn_fwd(qk, qkv, B, T, H, H, D, window, int8_pv=True)):
            assert torch.equal(x.cpu(), ref)


# several items a CTA, each of several query steps a head, the last one ragged (an odd and an even number of halves); with a window whose edge
# falls in the ragged step
@pytest.mark.parametrize("B,T,H,Hkv,D,window", [(30, 333, 4, 2, 64, 0), (26, 450, 4, 4, 64, 200), (28, 297, 4, 2, 128, 0), (33, 261, 6, 3, 128, 140)])
def test_ragged_steps_of_many_items(B, T, H, Hkv, D, window):
    g = torch.Generator().manual_seed(T)
    qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).to(torch.bfloat16) for n in (H + Hkv, H + 2 * Hkv, H))

    def run(dev):
        a, b, d = qk.to(dev), qkv.to(dev), dO.to(dev)
        O, lse = K.attn_fwd(a, b, B, T, H, Hkv, D, window)
        dqk, dqkv = torch.zeros_like(a), torch.zeros_like(b)
        K.attn_bwd(a, b, O, d, lse, dqk, dqkv, B, T, H, Hkv, D, window)
        return [t.cpu() for t in (O, lse, dqk, dqkv)]

    assert -(-T // 128) * Hkv * B > 148
    for got, ref in zip(run("cuda"), run("cpu")):
        assert torch.equal(got, ref)
    assert K.kernel_status("cuda") == 0


def _same(got, ref):
    """Bit for bit, but for what a NaN holds."""
    got, ref = got.cpu(), ref.cpu()
    assert torch.equal(got.isnan(), ref.isnan())
    bits = torch.int16 if ref.element_size() == 2 else torch.int32
    assert torch.equal(got.masked_fill(ref.isnan(), 0).view(bits), ref.masked_fill(ref.isnan(), 0).view(bits))


def _values(T, heads, D, exponent, seed):
    """Values of magnitude 2^exponent .. 2^(exponent + 1)."""
    g = torch.Generator().manual_seed(seed)
    v = torch.ldexp(1.0 + torch.rand(T, heads, D, generator=g), torch.tensor(exponent))
    return (v * (torch.randint(0, 2, v.shape, generator=g) * 2 - 1)).to(torch.bfloat16)


# outputs are divided in two ways, without the divider where all of a warp's are between 2^-60 and 2^80
@pytest.mark.parametrize("D,int8_pv", [(64, False), (128, False), (128, True)])
@pytest.mark.parametrize("exponent", [-118, -110, -62, -61, -60, -59, 0, 78, 79, 80, 81, 118])
def test_outputs_at_the_bounds_of_the_division(D, int8_pv, exponent):
    T, H = 131, 2
    g = torch.Generator().manual_seed(D)
    qk = torch.randn(T, 2 * H * D, generator=g).to(torch.bfloat16)
    qkv = torch.cat([torch.zeros(T, 2 * H, D, dtype=torch.bfloat16), _values(T, H, D, exponent, D)], 1).view(T, -1)
    for got, ref in zip(K.attn_fwd(qk.cuda(), qkv.cuda(), 1, T, H, H, D, 0, int8_pv=int8_pv), K.attn_fwd(qk, qkv, 1, T, H, H, D, 0, int8_pv=int8_pv)):
        assert ref.isfinite().all()
        _same(got, ref)


@pytest.mark.parametrize("D,int8_pv", [(64, False), (128, False), (128, True)])
@pytest.mark.parametrize("what", ["zero columns", "a zero row", "one lane", "infinities", "NaN", "NaN query"])
def test_outputs_that_are_divided(D, int8_pv, what):
    """What takes a warp to the divider: zeros of either sign, one value of one lane, an infinity, a NaN, and a row whose sum is out of
    bounds. (The CPU twin forms products of finite numbers only: its outputs that meet an infinity or a NaN are not compared, those of
    the same warp beside them are.)"""
    T, H, inf = 200, 3, float("inf")
    g = torch.Generator().manual_seed(D + 1)
    qk, qkv = torch.randn(T, 2 * H * D, generator=g).to(torch.bfloat16), torch.randn(T, 3 * H * D, generator=g).to(torch.bfloat16)
    v = qkv.view(T, 3 * H, D)[:, 2 * H:]
    met = torch.zeros(T, H, D, dtype=torch.bool)
    if what == "zero columns":
        v[:, 0, 3], v[:, 0, 40:50], v[:, 2, 17] = 0.0, -0.0, -0.0
    elif what == "a zero row":
        v[0, 1] = -0.0  # the first query's outputs
    elif what == "one lane":
        v[0, 0, 5], v[0, 1, 6], v[0, 2, 7] = 2.0**-61, 2.0**-60, 2.0**81  # the first query's own; the others' are sums with the rest
    elif what == "infinities":  # (of an int8 block: a step of infinity, and sums of zeros times that)
        v[0, 0, 5], v[0, 2, 6] = inf, -inf
        met[:, 0, 5] = met[:, 2, 6] = not int8_pv
    elif what == "NaN":
        v[0, 1, 5] = float("nan")
        met[:, 1, 5] = not int8_pv
    else:
        qk.view(T, 2 * H, D)[[70, 199], 1, 0] = float("nan")
        met[[70, 199], 1] = True
    (O, lse), (O_ref, lse_ref) = (K.attn_fwd(a, b, 1, T, H, H, D, 0, int8_pv=int8_pv) for a, b in ((qk.cuda(), qkv.cuda()), (qk, qkv)))
    O = O.cpu().view(T, H, D)
    _same(O.masked_fill(met, 0), O_ref.view(T, H, D).masked_fill(met, 0))
    lost = met.all(-1).t()
    _same(lse.cpu()[0].masked_fill(lost, 0), lse_ref[0].masked_fill(lost, 0))
    if what == "infinities" and not int8_pv:
        assert (O[:, 0, 5] == inf).all() and (O[:, 2, 6] == -inf).all()
    elif what == "NaN" and not int8_pv:
        assert O[:, 1, 5].isnan().all()
