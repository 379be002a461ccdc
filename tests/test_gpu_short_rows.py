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
    x[2, 0], x[3, V // 2] = float("nan"), float("-inf")  # (the NaN: in a row that is ignored, and cleared)
    labels = torch.tensor([0, V - 1, -1, V // 2, V - 8])

    def run(dev, grad):
        a = x.to(dev)
        ce, lse = K.ce_zloss_(a, labels.to(dev), 1e-4, 1.0 / rows, grad)
        return [t.cpu().view(torch.int16 if t.element_size() == 2 else torch.int32) for t in (ce, lse, a)]

    for grad in (True, False):
        for got, ref in zip(run("cuda", grad), run("cpu", grad)):
            assert torch.equal(got, ref)


@pytest.mark.parametrize("V", [8, 256, 264, 512, 1024, 2056, 4096, 4104, 8192, 8200, 12296, 16384, 16392])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_loss_rows_of_no_numbers(V, dtype):
    """Rows that count: a NaN away from the label and at it, infinities of either sign, nothing but -inf. Bit for bit but for what a
    NaN holds."""
    inf, nan = float("inf"), float("nan")
    g = torch.Generator().manual_seed(V)
    x = torch.randn(7, V, generator=g)
    x[0, V - 1], x[1, 3], x[2, V // 2], x[3, 1], x[4, :], x[5, 5], x[5, 6], x[6, :] = nan, nan, inf, inf, -inf, inf, -inf, inf
    labels = torch.tensor([0, 3, 0, 1, V - 1, 6, 0])

    def run(dev, grad):
        a = x.to(dtype).to(dev)
        ce, lse = K.ce_zloss_(a, labels.to(dev), 1e-4, 1.0 / 7, grad)
        return [t.cpu() for t in (ce, lse, a)]

    for grad in (True, False):
        for got, ref in zip(run("cuda", grad), run("cpu", grad)):
            assert torch.equal(got.isnan(), ref.isnan())
            assert torch.equal(got.masked_fill(ref.isnan(), 0), ref.masked_fill(ref.isnan(), 0))


@pytest.mark.parametrize("D", [8, 12, 248, 256, 264, 2048, 2056, 4096])  # (12: no whole groups of eight)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_gradient(D, dtype):
    g = torch.Generator().manual_seed(D)
    ids = torch.cat([torch.randint(0, 40, (60,), generator=g), torch.full((9,), 7), torch.tensor([49])])  # runs of one to a dozen
    dy, start = torch.randn(len(ids), D, generator=g).to(dtype), torch.randn(50, D, generator=g)
    for accumulate in (True, False):
        out = []
        for dev in ("cuda", "cpu"):
            dW = start.to(dev).clone()
            K.embedding_bwd(dy.to(dev), ids.to(dev), dW, accumulate)
            out.append(dW.cpu())
        assert torch.equal(*out)
    # a gradient that starts between two 16-byte boundaries takes the column-by-column form
    odd = torch.empty(dy.numel() + 1, dtype=dtype, device="cuda")[1:].view_as(dy).copy_(dy)
    dW = start.cuda()
    K.embedding_bwd(odd, ids.cuda(), dW, True)
    ref = start.clone()
    K.embedding_bwd(dy, ids, ref, True)
    assert torch.equal(dW.cpu(), ref)
