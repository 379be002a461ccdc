"""The model's train() / eval(): what nn.Module does, submodules with a method of their own included."""
import pytest
from torch import nn

from open_transformers_b200.config import load_config
from open_transformers_b200.models.llama3 import build_model


class Counting(nn.Module):
    def __init__(self):
        super().__init__()
        self.calls = []

    def train(self, mode=True):
        self.calls.append(mode)
        return super().train(mode)


def test_mode_reaches_every_module():
    model = build_model(load_config("tiny_cpu", ["model.n_layers=2", "model.vocab_size=1024"]).model)
    model.extra = Counting()
    model.blocks[1].attn.extra = nn.ModuleList([nn.Identity(), nn.Dropout(0.5)])
    model.blocks[0].eval()
    for mode in (True, False, True):
        assert model.train(mode) is model
        assert all(m.training is mode for m in model.modules())
    assert model.extra.calls == [True, False, True]
    assert model.eval() is model and not any(m.training for m in model.modules())
    mine = []
    model.blocks[0].ffn.train = lambda mode=True: mine.append(mode)
    model.train()
    assert mine == [True] and model.training and not model.blocks[0].ffn.training
    with pytest.raises(ValueError):
        model.train(1)


class Hiding(nn.Module):
    """Keeps a submodule of its own out of what is switched."""

    def __init__(self):
        super().__init__()
        self.shown, self.hidden = nn.Identity(), nn.Identity()

    def children(self):
        return iter([self.shown])


class HidingByName(Hiding):
    children = nn.Module.children

    def named_children(self):
        return iter([("shown", self.shown)])


class Elsewhere(nn.Module):
    """Keeps its mode somewhere else."""

    @property
    def training(self):
        return self.__dict__.get("mode")

    @training.setter
    def training(self, mode):
        self.__dict__["mode"] = mode


class Writing(nn.Module):
    def __init__(self):
        object.__setattr__(self, "written", [])
        super().__init__()

    def __setattr__(self, name, value):
        self.written.append((name, value))
        super().__setattr__(name, value)


def _extended(**modules):
    model = build_model(load_config("tiny_cpu", ["model.n_layers=1", "model.vocab_size=1024"]).model)
    for name, m in modules.items():
        model.blocks[0].add_module(name, m)
    return model


@pytest.mark.parametrize("how", [lambda model: model.eval(), lambda model: nn.Module.train(model, False)])
def test_modules_with_ways_of_their_own(how):
    hiding, by_name, elsewhere, writing, twice = Hiding(), HidingByName(), Elsewhere(), Writing(), Counting()
    model = _extended(hiding=hiding, by_name=by_name, elsewhere=elsewhere, writing=writing, twice=twice, again=twice, none=None)
    by_instance = nn.Sequential(nn.Identity())
    by_instance.children = lambda: iter(())
    model.by_instance = by_instance
    model.train()
    writing.written.clear(), twice.calls.clear()
    assert how(model) is model
    for m in (hiding, by_name):
        assert (m.training, m.shown.training, m.hidden.training) == (False, False, True)
    assert elsewhere.training is False and "training" not in elsewhere.__dict__
    assert writing.written == [("training", False)] and twice.calls == [False]
    assert not by_instance.training and by_instance[0].training


def test_replaced_methods_are_called(monkeypatch):
    model, calls, plain = _extended(), [], nn.Module.train
    monkeypatch.setattr(nn.Module, "train", lambda self, mode=True: calls.append(self) or plain(self, mode))
    model.eval()
    assert set(calls) == set(model.modules())


class Above(nn.Module):
    def train(self, mode=True):
        self.asked = mode
        return super().train(mode)


def test_classes_beside_the_model_are_called():
    model = _extended()
    model.__class__ = type("Beside", (type(model), Above), {})
    assert model.eval() is model and model.asked is False and not any(m.training for m in model.modules())
    model = _extended()
    model.__class__ = type("Keeping", (type(model),), {"children": lambda self: iter(())})
    assert not model.eval().training and model.blocks[0].training
