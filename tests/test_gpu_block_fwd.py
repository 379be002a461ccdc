"""A decoder block without gradients runs as one native call: the bits of its modules called one by one, and only where nothing
but their launches is wanted."""
import pytest
import torch

from open_transformers_b200.config import load_config
from open_transformers_b200.models.modules import core
from open_transformers_b200.ops import functional as K
from open_transformers_b200.ops import native
from open_transformers_b200.train.engine import TrainEngine

pytestmark = pytest.mark.gpu


def _engine(recipe, *over):
    return TrainEngine(load_config(recipe, ["run.virtual_dp_size=1", "run.dp_shard_size=1", "run.dp_replicate_size=1", *over]), "cuda:0")


@pytest.fixture
def calls(monkeypatch):
    n = []
    real = K.block_fwd
    monkeypatch.setattr(K, "block_fwd", lambda *a: (n.append(1), real(*a))[1])
    return n


def _one_by_one(model, ids):
    hooks = [b.attn.wo.register_forward_hook(lambda *a: None) for b in model.blocks]
    try:
        return model(ids).logits
    finally:
        for h in hooks:
            h.remove()


# one token; one and several query tiles with a ragged last one; more than one sequence; bf16 (window and full layers) and fp32;
# without QK-norm; 128-wide heads
@pytest.mark.parametrize("recipe,over,B,T", [
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 1, 1),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 3, 129),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 1, 777),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false", "model.modules.attention=gqa_plain_repop"], 2, 200),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false", "model.n_heads=6", "model.n_kv_heads=2",
                          "model.head_dim=128", "model.attn_int8_pv=false"], 1, 300),
    ("tiny_cpu", [], 2, 37)])
def test_same_bits_as_the_modules(calls, recipe, over, B, T):
    model = _engine(recipe, *over).model.eval()
    ids = torch.randint(0, 512, (B, T), generator=torch.Generator().manual_seed(T)).cuda()
    with torch.no_grad():
        want = _one_by_one(model, ids)
        assert not calls
        before = native.launch_count
        got = model(ids).logits
        assert len(calls) == len(model.blocks) and native.launch_count - before == 9 * len(calls) + 3
    assert torch.equal(got, want)
    assert K.kernel_status("cuda") == 0


def test_other_calls_keep_the_modules(calls, monkeypatch):
    model = _engine("tiny_cpu").model.eval()
    ids = torch.randint(0, 512, (1, 16), device="cuda")
    model(ids)  # gradients
    with torch.no_grad():
        want = _one_by_one(model, ids)
        native.start_timing()
        model(ids)
        native.timing_report()
        for cls in (core.Linear, core.RMSNorm, core.SwiGLU, type(model.blocks[0].attn)):
            with monkeypatch.context() as m:
                own = cls.forward
                m.setattr(cls, "forward", lambda self, *a, _own=own, **k: _own(self, *a, **k))
                assert torch.equal(model(ids).logits, want)
        with torch.autograd.forward_ad.dual_level():
            model(ids)
    assert not calls


def _blocks(model, B=1, T=130):
    x = torch.randn(B, T, model.cfg.d_model, generator=torch.Generator().manual_seed(T)).to(model.compute_dtype).cuda()
    cos, sin = model.rope(T)

    def run(x):
        for blk in model.blocks:
            x = blk(x, cos, sin)
        return x

    return x, run


SMALL = ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"]


def _by_modules(model, run, x):
    hooks = [b.attn.wo.register_forward_hook(lambda *a: None) for b in model.blocks]
    try:
        return run(x)
    finally:
        for h in hooks:
            h.remove()


def test_onlookers_keep_the_modules(calls):
    """Function transforms (which the modules' autograd functions refuse), dispatch and function modes see the modules' own calls."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kw=None):
            return f(*args, **(kw or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, f, types, args=(), kw=None):
            return f(*args, **(kw or {}))

    model = _engine("100m_smoke_repop", *SMALL).model.eval()
    x, run = _blocks(model)
    with torch.no_grad():
        want = _by_modules(model, run, x)
        for mode in (Dispatch, Function):
            with mode():
                got = run(x)
            assert torch.equal(got, want)
        for transformed in (lambda: torch.func.vmap(run)(x[None]), lambda: torch.func.jvp(run, (x,), (x,)), lambda: torch.func.vjp(run, x)):
            with pytest.raises(RuntimeError):
                transformed()
        assert not calls
        assert torch.equal(run(x), want) and len(calls) == 2
    with torch.inference_mode():
        assert torch.equal(run(x), want) and len(calls) == 4


def test_weights_are_read_anew(calls):
    """Weights written in place or put in another's place count at the next call; one that is not ready as it lies, or whose rows
    may still be on their way, keeps the modules."""
    model = _engine("100m_smoke_repop", *SMALL).model.eval()
    x, run = _blocks(model)
    with torch.no_grad():
        before = run(x)
        down = model.blocks[1].ffn.w_down
        down._compute_weight.mul_(0.5)
        want = _by_modules(model, run, x)
        assert not torch.equal(want, before) and torch.equal(run(x), want) and len(calls) == 4
        down._compute_weight = down._compute_weight * 2
        assert torch.equal(run(x), before) and len(calls) == 6
        down._compute_weight = down._compute_weight.t().contiguous().t()  # not row-major
        assert down._compute_weight.shape == (768, 2048)
        with pytest.raises(AssertionError):  # as by the modules
            run(x)
        assert len(calls) == 7
        down._compute_weight = down._compute_weight.contiguous()

        class Arrived:
            pending = staticmethod(lambda: False)

        for slot in (down._slot_weight, model.blocks[1].attn._fused_qkv[2], model.blocks[1].norm2._slot_weight):
            slot.gather, n = Arrived(), len(calls)
            assert torch.equal(run(x), before) and len(calls) == n + 1
            slot.gather = None


def test_captured_with_a_second_stream():
    """Chained launches in a graph, behind and in front of a fork: the replayed bits are those of the calls."""
    model = _engine("100m_smoke_repop", *SMALL).model.eval()
    x, run = _blocks(model)
    x2, _ = _blocks(model, T=97)
    cos, sin = model.rope(97)
    side = torch.cuda.Stream()

    def both():
        here = torch.cuda.current_stream()
        a = run(x)
        side.wait_stream(here)
        with torch.cuda.stream(side):
            b = model.blocks[0](x2, cos, sin)
        c = run(a)
        here.wait_stream(side)
        return a, c, model.blocks[1](b, cos, sin)

    with torch.no_grad():
        both()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = both()
        x.mul_(1.5)
        x2.mul_(0.75)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        want = both()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


def test_two_threads_on_one_stream():
    """Attention backward, whose dQ begins beside dK/dV, with chained launches of another thread between its own."""
    import threading

    def work(seed):
        g = torch.Generator().manual_seed(seed)
        B, T, H, Hkv, D = 1, 450 + 64 * seed, 8, 2, 64
        qk, qkv, dO = (torch.randn(B * T, n * D, generator=g).bfloat16().cuda() for n in (H + Hkv, H + 2 * Hkv, H))
        w, gu = torch.randn(H * D, generator=g).bfloat16().cuda(), torch.randn(T, 2 * H * D, generator=g).bfloat16().cuda()

        def once():
            O, lse = K.attn_fwd(qk, qkv, B, T, H, Hkv, D, 0)
            dqk, dqkv = torch.empty_like(qk), torch.zeros_like(qkv)
            K.attn_bwd(qk, qkv, O, dO, lse, dqk, dqkv, B, T, H, Hkv, D, 0)
            y, _ = K.rmsnorm_fwd(dqk[:, : H * D].contiguous(), w, 1e-5)
            return dqk, dqkv, y, K.swiglu_fwd(gu)

        return once

    jobs = [work(s) for s in range(2)]
    want = [[t.clone() for t in job()] for job in jobs]
    torch.cuda.synchronize()
    stream, bad = torch.cuda.current_stream(), []

    def run(i):
        with torch.cuda.stream(stream):
            for _ in range(25):
                out = jobs[i]()
                torch.cuda.synchronize()
                if not all(torch.equal(a, b) for a, b in zip(out, want[i])):
                    bad.append(i)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and K.kernel_status("cuda") == 0
