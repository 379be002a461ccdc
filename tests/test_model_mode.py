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

