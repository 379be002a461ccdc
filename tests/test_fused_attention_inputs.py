"""Fused projections and per-head gains of the attention module against the layers they stand for: bit for bit."""
import pytest
import torch

from open_transformers_b200.config.schema import QATConfig
from open_transformers_b200.models.modules import core
from open_transformers_b200.ops import autograd as A
from open_transformers_b200.ops import functional as K


def _run(mod, x, dy, cos, sin, fused):
    for p in mod.parameters():
        p.grad = None
    x = x.clone().requires_grad_()
    untouched = core._untouched
    core._untouched = untouched if fused else (lambda m, c: False)
    try:
        y = mod(x, cos, sin)
    finally:
        core._untouched = untouched
    y.backward(dy)
    return [y.detach(), x.grad] + [p.grad.clone() for _, p in sorted(mod.named_parameters())]


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("method,B,T,H,Hkv,D,gain", [("lsq", 1, 17, 2, 1, 64, True), ("absmax", 2, 40, 3, 3, 64, False), ("lsq", 2, 72, 4, 2, 128, True)])
def test_attention_module(device, dtype, method, B, T, H, Hkv, D, gain):
    g = torch.Generator().manual_seed(T)
    d = 64
    mod = core.GQAQKNorm(d, H, Hkv, D, qk_norm_gain=gain, qat=QATConfig(enabled=True, method=method))
    with torch.no_grad():
        for name, p in mod.named_parameters():
            p.copy_(torch.randn(p.shape, generator=g) * 0.05 + (1.0 if "norm" in name else 0.0))
            if name.endswith("weight_scale"):
                p.copy_(torch.rand(p.shape, generator=g) * 1e-3 + 5e-4)
    mod = mod.to(device)
    cos, sin = K.rope_tables(T, D, 10000.0, device)
    x, dy = (torch.randn(B, T, d, generator=g).to(device, dtype) for _ in range(2))
    for a, b in zip(_run(mod, x, dy, cos, sin, True), _run(mod, x, dy, cos, sin, False)):
        assert torch.equal(a, b)


def test_a_hooked_layer_is_called():
    """A forward hook on a projection or on a gain keeps the layer's own call."""
    mod = core.GQAQKNorm(64, 2, 1, 32, qat=QATConfig(enabled=True, method="absmax"))
    with torch.no_grad():
        for p in mod.parameters():
            p.fill_(0.01)
    cos, sin = K.rope_tables(4, 32, 10000.0, "cpu")
    seen = []
    mod.wk.register_forward_hook(lambda *a: seen.append("wk"))
    mod.k_norm.register_forward_hook(lambda *a: seen.append("k_norm"))
    mod(torch.ones(1, 4, 64), cos, sin)
    assert seen == ["wk", "k_norm"]


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])  # (the gains are fused on a GPU only)
@pytest.mark.parametrize("cls", [core.QuantLinear, core.RMSNorm])
def test_a_forward_replaced_on_the_class_is_called(monkeypatch, device, cls):
    mod = core.GQAQKNorm(64, 2, 1, 64, qat=QATConfig(enabled=True, method="absmax"))
    with torch.no_grad():
        for p in mod.parameters():
            p.fill_(0.01)
    mod = mod.to(device)
    cos, sin = K.rope_tables(4, 64, 10000.0, device)
    seen, own = [], cls.forward
    monkeypatch.setattr(cls, "forward", lambda self, *a, **kw: (seen.append(self), own(self, *a, **kw))[1])
    mod(torch.ones(1, 4, 64, device=device), cos, sin)
    assert seen == ([mod.wq, mod.wk, mod.wv, mod.wo] if cls is core.QuantLinear else [mod.q_norm, mod.k_norm])


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("name", ["q_norm", "k_norm"])
def test_head_norm_without_a_gain(monkeypatch, device, name):
    """A module whose query or key norm was replaced by one without a weight: no gain to fuse."""
    g = torch.Generator().manual_seed(3)
    mod = core.GQAQKNorm(64, 2, 1, 64)
    setattr(mod, name, core.RMSNorm(64, gain=False))
    with torch.no_grad():
        for p in mod.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * 0.05)
    mod = mod.to(device)
    cos, sin = K.rope_tables(9, 64, 10000.0, device)
    x, dy = (torch.randn(2, 9, 64, generator=g).to(device) for _ in range(2))
    want = _run(mod, x, dy, cos, sin, False)
    monkeypatch.setattr(K, "head_norm_supported", lambda x, D: True)  # (so that the CPU run asks the same question)
    for a, b in zip(_run(mod, x, dy, cos, sin, True), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_gradient_of_the_joint_projections_at_any_address(device):
    """A contiguous gradient that starts at an odd element (the layers by themselves get aligned copies of their columns)."""
    g = torch.Generator().manual_seed(5)
    mod = core.GQAQKNorm(64, 2, 1, 64, qat=QATConfig(enabled=True, method="absmax"))
    with torch.no_grad():
        for p in mod.parameters():
            p.copy_(torch.randn(p.shape, generator=g) * 0.05)
    mod = mod.to(device)
    x = torch.randn(2, 9, 64, generator=g).to(device, torch.bfloat16).requires_grad_()
    dy = torch.randn(2 * 9 * 256 + 1, generator=g).to(device, torch.bfloat16)[1:].view(2, 9, 256)
    weights = [m.weight for m in (mod.wq, mod.wk, mod.wv)]
    for a, b in zip(torch.autograd.grad(mod._qkv(x), [x, *weights], dy), torch.autograd.grad(mod._qkv(x), [x, *weights], dy.clone())):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,D,pad", [(1, 1, 8, 0), (5, 3, 64, 8), (33, 5, 128, 16), (130, 2, 120, 0)])
def test_per_head_norm(dtype, tokens, heads, D, pad):
    g = torch.Generator().manual_seed(tokens)
    x, dy = (torch.randn(tokens, heads * D + pad, generator=g).to(dtype) for _ in range(2))
    w = torch.randn(D, generator=g).to(dtype)
    rows = lambda t: t[:, : heads * D].reshape(-1, D).contiguous()  # noqa: E731
    y, rstd = K.rmsnorm_fwd(rows(x), w, 1e-5)
    dx, dg = K.rmsnorm_bwd(rows(dy), rows(x), w, rstd, True)
    xc, dyc = x.cuda()[:, : heads * D], dy.cuda()[:, : heads * D]
    yc, dxc = torch.zeros_like(x).cuda()[:, : heads * D], torch.zeros_like(x).cuda()[:, : heads * D]
    rc = K.head_rmsnorm_fwd(xc, w.cuda(), yc, heads, D, 1e-5)
    dgc = K.head_rmsnorm_bwd(dyc, xc, w.cuda(), rc, dxc, heads, D, True)
    for a, b in ((yc, y), (rc, rstd), (dxc, dx), (dgc, dg)):
        assert torch.equal(a.cpu().reshape(b.shape), b)
