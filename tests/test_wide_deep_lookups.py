"""Which lookups the multi-hot Wide&Deep model makes of an engine with fused bag lookups, on a stand-in for that engine."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200.models import MultiHotWideAndDeep
from kraken_b200.pytorch import native


class FakeEngine:
    def __init__(self, nccl):
        self.nccl, self.calls = nccl, []

    def pull_sparse_table(self, table_id, indices):
        self.calls.append(("rows", table_id))
        return torch.zeros(*indices.shape, {1: 1, 2: 8}[table_id])

    def pull_sparse_pooled(self, table_id, values, offsets, weights=None, mean=False, bag_mean=None, patch_value=0.0,
                           share_with=None):
        self.calls.append(("pooled", table_id, patch_value, mean, share_with))
        return torch.zeros(offsets.numel() - 1, {1: 1, 2: 8}[table_id]), None


class Doubled(kk.JaggedEmbedding):
    def forward(self, input):
        return super().forward(input) * 2


def replaced(model):
    model.wide = Doubled(1)
    model.wide.embedding.sparse_table.set_table_id(1)


def hooked(model):
    model.wide.register_forward_hook(lambda m, i, o: None)


def hooked_before(model):
    model.wide.register_forward_pre_hook(lambda m, i: None)


def patched(model):
    model.wide._patch_value = 2.0
    model.wide._mode = "mean"


def overridden(model):
    forward = model.wide.forward
    model.wide.forward = lambda bags: forward(bags)


@pytest.mark.parametrize("change,wide,share", [
    (None, ("pooled", 1, 0.0, False, None), 1), (patched, ("pooled", 1, 2.0, True, None), 1),
    (hooked, ("pooled", 1, 0.0, False, None), None), (hooked_before, ("pooled", 1, 0.0, False, None), None),
    (replaced, ("pooled", 1, 0.0, False, None), None), (overridden, ("pooled", 1, 0.0, False, None), None),
    ("nccl", ("rows", 1), None)])
def test_the_wide_part_is_the_module_wide(monkeypatch, change, wide, share):
    """Both tables share a dedup only where the wide lookup is known to be of the same ids; with collectives in the place of
    the fused exchange the wide table goes through those."""
    eng = FakeEngine(nccl=change == "nccl")
    monkeypatch.setattr(native, "_engine", eng)
    monkeypatch.setattr(native, "_as_registered", lambda table_id, rows: rows)
    model = MultiHotWideAndDeep(num_fields=2, num_dense=3, dim=8, hidden=(8,))
    model.wide.embedding.sparse_table.set_table_id(1)
    model.deep.sparse_table.set_table_id(2)
    if callable(change):
        change(model)
    called = []
    handle = None
    if change is None:
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: called.append(m))
    bags = kk.JaggedTensor(torch.tensor([3, 4, 3, 9]), torch.tensor([0, 1, 2, 3, 4]))
    model(torch.zeros(2, 3), bags)
    if handle is not None:
        handle.remove()
        assert model.wide in called and eng.calls[-1][-1] is None  # a hook on every module is a hook on this one
        eng.calls.clear()
        model(torch.zeros(2, 3), bags)
    assert eng.calls == [wide, ("pooled", 2, 0.0, False, share)]
