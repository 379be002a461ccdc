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


# one token; one and several query tiles with a ragged last one; more than one sequence; bf16 (window and full layers) and fp32
@pytest.mark.parametrize("recipe,over,B,T", [
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 1, 1),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 3, 129),
    ("100m_smoke_repop", ["model.n_layers=2", "model.vocab_size=512", "model.qat.enabled=false"], 1, 777),
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
