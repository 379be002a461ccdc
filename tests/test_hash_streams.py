"""The engine's prepared hash streams against the records fed one by one."""
import pytest
import torch

from open_transformers_b200.train import state_hash as SH
from open_transformers_b200.train.engine import TrainEngine
from helpers import tiny_cfg


# one shard, and down to four elements of a gain per shard
@pytest.mark.parametrize("shards", [1, 2, 32])
@pytest.mark.parametrize("grads", [True, False])
def test_streams_equal_records(tmp_path, shards, grads):
    cfg = tiny_cfg(str(tmp_path), ["run.virtual_dp_size=%d" % shards, "run.dp_shard_size=%d" % shards])
    eng = TrainEngine(cfg, "cpu")
    for flat in (eng.master, eng.m1, eng.m2, eng.grad_red):
        flat.copy_(torch.randn(flat.shape, generator=torch.Generator().manual_seed(shards)))
    for step in (0, 7):  # the second hash reuses the streams
        eng.opt_step = step
        state = SH.audit_shard_state_digest(eng.named_master(), eng.optimizer_state(), dict(eng.named_grads()) if grads else None, shards, eng.V,
                                            include_grads=grads, tensor_digest="tree")
        want = SH.finalize_state_hash(state, eng.param_groups, None, None)
        assert eng.sharded_state_hash(None, None, include_grads=grads, tensor_digest="tree") == want
