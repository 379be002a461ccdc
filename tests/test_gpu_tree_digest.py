"""Tree digests on a GPU at the edges of leaves, levels and lane groups against the host digest."""
import pytest
import torch

from open_transformers_b200.train import state_hash as SH

pytestmark = pytest.mark.gpu
LEAF = 4096
# empty, below / at / above a leaf, ragged and odd tails, a root of whole words and one that is not, two and three levels
SIZES = [0, 1, 8, 120, 127, 128, 4088, 4095, LEAF, LEAF + 1, LEAF + 8, 2 * LEAF + 36, 127 * LEAF, 128 * LEAF, 128 * LEAF + 4, 129 * LEAF, 16400 * LEAF + 20]


def _bytes(n, seed):
    return torch.randint(0, 256, (n,), dtype=torch.uint8, generator=torch.Generator().manual_seed(seed))


def test_batch_of_all_sizes():
    host = [_bytes(n, i) for i, n in enumerate(SIZES)]
    dev = [t.cuda() for t in host]
    want = [SH.tree_digest_bytes(t.numpy().tobytes()) for t in host]
    assert SH.tree_digest_batch(dev) == want
    assert [SH.tree_digest_tensor(t) for t in dev if t.numel()] == [w for t, w in zip(dev, want) if t.numel()]


@pytest.mark.parametrize("count", [1, 15, 17, 70])  # groups of four lanes that do not fill a warp, a CTA or the grid
def test_plan_of_many(count):
    host = [_bytes(4 * (1 + (i * 7919) % 9000), i) for i in range(count)]
    plan = SH.TreeDigestPlan([t.cuda() for t in host])
    plan.launch()
    torch.cuda.synchronize()
    assert plan.digests() == [SH.tree_digest_bytes(t.numpy().tobytes()) for t in host]
