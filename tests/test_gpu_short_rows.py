"""Loss rows that stay in registers and the embedding gradient eight columns at a time: bit for bit against the CPU twins."""
import pytest
import torch

from open_transformers_b200.ops import functional as K

pytestmark = pytest.mark.gpu


# one group, a warp of them and one more, either side of each CTA size and of each number of groups per thread, and of the longest row taken
@pytest.mark.parametrize("V", [8, 256, 264, 512, 1024, 2056, 4096, 4104, 8192, 8200, 12296, 16384, 16392])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_loss_rows(V, dtype):
    rows = 5
    g = torch.Generator().manual_seed(V)
    x = (torch.randn(rows, V, generator=g) * 3).to(dtype)
    x[1, V - 1] = -400.0  # exponent clamped
    x[2, 0], x[3, V // 2] = float("nan"), float("-inf")
    labels = torch.tensor([0, V - 1, -1, V // 2, V - 8])

    def run(dev, grad):
        a = x.to(dev)
        ce, lse = K.ce_zloss_(a, labels.to(dev), 1e-4, 1.0 / rows, grad)
        return [t.cpu().view(torch.int16 if t.element_size() == 2 else torch.int32) for t in (ce, lse, a)]

    for grad in (True, False):
        for got, ref in zip(run("cuda", grad), run("cpu", grad)):
            assert torch.equal(got, ref)
