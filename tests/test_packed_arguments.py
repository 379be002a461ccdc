"""Arguments of the packed entry points: the numbers that the one-object-per-argument calls take."""
import struct

import numpy as np
import pytest
import torch

from open_transformers_b200.ops import functional as K
from open_transformers_b200.ops import native


@pytest.mark.parametrize("given,want", [((3, 512, 1e-5), (3, 512, 1e-5)), ((True, 512.0, 1), (1, 512, 1.0)), ((np.int32(3), np.float64(512), np.float32(0.5)), (3, 512, 0.5)),
                                        ((torch.tensor(3), torch.tensor(512.0), torch.tensor(0.25)), (3, 512, 0.25))])
def test_numbers_of_any_type(monkeypatch, given, want):
    got = []

    class Library:
        @staticmethod
        def entry_p(words):
            got.append(struct.unpack("=2qd", words))
            return 0

    monkeypatch.setattr(native, "cuda_lib", lambda: Library)
    assert native.packed_entry("entry", "2qd")(*given) == 0
    assert got == [want]


def test_what_is_no_number_is_refused(monkeypatch):
    monkeypatch.setattr(native, "cuda_lib", lambda: type("Library", (), {"entry_p": staticmethod(lambda words: 0)}))
    call = native.packed_entry("entry", "2qd")
    for bad in ((None, 1, 1.0), (1, 1), (1, 1, 1.0, 1), (1, "x", 1.0)):
        with pytest.raises((struct.error, TypeError, ValueError)):
            call(*bad)


@pytest.mark.gpu
def test_a_window_given_as_a_float():
    g = torch.Generator().manual_seed(1)
    qk, qkv = (torch.randn(200, n * 64, generator=g).bfloat16().cuda() for n in (2, 3))
    for a, b in zip(K.attn_fwd(qk, qkv, 1, 200, 1, 1, 64, 32.0), K.attn_fwd(qk, qkv, 1, 200, 1, 1, 64, 32)):
        assert torch.equal(a, b)
