"""Memory-bound kernels on a GPU at the edges of their tilings: bit for bit against the CPU twin."""
import pytest
import torch

from open_transformers_b200.ops import functional as K

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def _same(dev, host, what):
    assert torch.equal(dev.cpu(), host), what


@pytest.mark.parametrize("dtype", [BF16, F32])
# register widths, and one past the last; bf16 keeps rows up to 768, and 2056 to 4096 of 12288 and more, in registers; where rows
# are read twice, four groups per turn up to 9472 rows (148 SMs) and two above
@pytest.mark.parametrize("rows,D", [(1, 8), (9, 248), (7, 1032), (3, 4096), (5, 4104), (9, 256), (9, 264), (9, 768), (9, 776), (9, 2048), (12288, 2048),
                                    (12288, 2056), (12287, 2056), (12289, 4096), (9472, 1032), (9473, 1032), (9473, 4104)])
def test_rmsnorm_forward_widths(dtype, rows, D):
    g = torch.Generator().manual_seed(D)
    x, w = torch.randn(rows, D, generator=g).to(dtype), torch.randn(D, generator=g).to(dtype)
    for weight in (w, None):
        dev = K.rmsnorm_fwd(x.cuda(), None if weight is None else weight.cuda(), 1e-5)
        for a, b in zip(dev, K.rmsnorm_fwd(x, weight, 1e-5)):
            _same(a, b, "rmsnorm")


# heads that do not fill a warp's group, narrow heads, and ``pad``: a row pitch (or an offset) that forbids the wide loads
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("rows,heads,D,seq,pad", [(1, 1, 4, 1, 0), (37, 5, 128, 10, 0), (50, 3, 64, 50, 0), (33, 6, 20, 11, 1), (16, 4, 128, 16, 2),
                                                  # four heads per warp (4800 heads and more), not all of them there; one head per token
                                                  (961, 5, 128, 31, 0), (1600, 3, 64, 50, 0), (800, 6, 20, 11, 1), (1201, 4, 128, 1201, 2), (5000, 1, 64, 100, 0)])
def test_qknorm_rope_groups(dtype, norm, rows, heads, D, seq, pad):
    g = torch.Generator().manual_seed(rows + D)
    cos, sin = K.rope_tables(seq, D, 10000.0, "cpu")
    wide = torch.randn(rows, heads * D + 8 + pad, generator=g).to(dtype)
    dwide = torch.randn(rows, heads * D + pad, generator=g).to(dtype)

    def run(dev):
        x, dy = wide.to(dev)[:, pad:], dwide.to(dev)[:, pad:]
        out, rstd = K.qknorm_rope_fwd(x, cos.to(dev), sin.to(dev), heads, D, seq, norm, 1e-5)
        din = torch.zeros(rows, heads * D + pad, dtype=dtype, device=dev)[:, pad:]
        K.qknorm_rope_bwd(dy, x, rstd, din, cos.to(dev), sin.to(dev), heads, D, seq, norm)
        return (out, rstd, din) if norm else (out, din)

    for a, b in zip(run("cuda"), run("cpu")):
        _same(a, b, "rope")


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("rows,F", [(1, 8), (3, 264), (2, 3072), (2, 3080), (2, 6152)])  # one group, one sweep, two sweeps of 384 threads
def test_swiglu_widths(dtype, rows, F):
    g = torch.Generator().manual_seed(F)
    gu, dh = torch.randn(rows, 2 * F, generator=g).to(dtype), torch.randn(rows, F, generator=g).to(dtype)
    _same(K.swiglu_fwd(gu.cuda()), K.swiglu_fwd(gu), "forward")
    _same(K.swiglu_bwd(gu.cuda(), dh.cuda()), K.swiglu_bwd(gu, dh), "backward")


# both forms of the kernel at the line between them: 1024 columns, 2048 rows (and the widths above on a CTA per row)
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("rows,F", [(2048, 1016), (2047, 1024), (2048, 1024), (2049, 3072), (2050, 3080), (2048, 6152), (70000, 8)])
def test_swiglu_forms(dtype, rows, F):
    g = torch.Generator().manual_seed(F)
    gu, dh = torch.randn(rows, 2 * F, generator=g).to(dtype), torch.randn(rows, F, generator=g).to(dtype)
    _same(K.swiglu_fwd(gu.cuda()), K.swiglu_fwd(gu), "forward")
    _same(K.swiglu_bwd(gu.cuda(), dh.cuda()), K.swiglu_bwd(gu, dh), "backward")


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("V", [8, 4096, 4104, 16392, 70008, 128256])  # one group, whole sweeps, ragged ones, both unrolls
def test_loss_row_widths(dtype, V):
    g = torch.Generator().manual_seed(V)
    x = (3 * torch.randn(3, V, generator=g)).to(dtype)
    labels = torch.tensor([0, V - 1, -100])
    for grad in (False, True):
        a, b = x.clone().cuda(), x.clone()
        dev, host = K.ce_zloss_(a, labels.cuda(), 1e-4, 0.25, grad), K.ce_zloss_(b, labels, 1e-4, 0.25, grad)
        for p, q in zip((*dev, a), (*host, b)):
            _same(p, q, "loss")


@pytest.mark.parametrize("B,T,H,Hkv,D", [(1, 64, 3, 1, 64), (3, 37, 4, 2, 64), (2, 131, 2, 1, 128)])  # rows that end inside a group of 8
def test_attention_row_groups(B, T, H, Hkv, D):
    g = torch.Generator().manual_seed(T)
    qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).to(BF16) for n in (H + Hkv, H + 2 * Hkv, H))

    def run(dev):
        a, b, d = qk.to(dev), qkv.to(dev), dO.to(dev)
        O, lse = K.attn_fwd(a, b, B, T, H, Hkv, D, 0)
        dqk, dqkv = torch.zeros_like(a), torch.zeros_like(b)
        K.attn_bwd(a, b, O, d, lse, dqk, dqkv, B, T, H, Hkv, D, 0)
        return O, lse, dqk, dqkv

    for p, q in zip(run("cuda"), run("cpu")):
        _same(p, q, "attention")


@pytest.mark.parametrize("dtype", [BF16, F32])
def test_loss_rows_with_far_values(dtype):
    """Rows whose exponents reach the clamp, at its edge, or hold infinities, beside an ordinary one."""
    V = 5000
    x = torch.randn(5, V, generator=torch.Generator().manual_seed(9))
    x[1] *= 100
    x[2, 17] = -87.0 + float(x[2].max())
    x[3, 4321] = -float("inf")
    x[4, 1:] = -float("inf")
    x = x.to(dtype)
    labels = torch.tensor([1, 2, 17, 4, 0])
    a, b = x.clone().cuda(), x.clone()
    dev, host = K.ce_zloss_(a, labels.cuda(), 1e-4, 0.25), K.ce_zloss_(b, labels, 1e-4, 0.25)
    for p, q in zip((*dev, a), (*host, b)):
        _same(p, q, "loss")


# every form of the loss kernel on both sides of each line (bf16: 8192 and 81920 columns, fp32: 24576 and 32768, and four rows per SM)
@pytest.mark.parametrize("dtype,V", [(BF16, 8192), (BF16, 8200), (BF16, 81920), (BF16, 81928), (F32, 24576), (F32, 24584), (F32, 32768), (F32, 32776)])
@pytest.mark.parametrize("rows", [8, 593])
def test_loss_forms_with_far_values(dtype, V, rows):
    """Ordinary rows beside rows whose exponents reach the clamp, at its edge, or hold infinities of either sign or a NaN."""
    x = torch.randn(rows, V, generator=torch.Generator().manual_seed(V))
    x[1] *= 100
    x[2, 17] = -87.0 + float(x[2].max())
    x[3, 4321] = -float("inf")
    x[4, 1:] = -float("inf")
    x[5, V - 1] = float("inf")
    x[6, 100] = float("nan")
    x[7, V - 3] = -87.5 + float(x[7].max())
    x = x.to(dtype)
    labels = torch.randint(0, V, (rows,), generator=torch.Generator().manual_seed(1))
    labels[4] = 0
    a, b = x.clone().cuda(), x.clone()
    dev, host = K.ce_zloss_(a, labels.cuda(), 1e-4, 0.25), K.ce_zloss_(b, labels, 1e-4, 0.25)
    for p, q, what in zip((*dev, a), (*host, b), ("ce", "lse", "gradient")):
        torch.testing.assert_close(p.cpu(), q, rtol=0, atol=0, equal_nan=True, msg=what)
