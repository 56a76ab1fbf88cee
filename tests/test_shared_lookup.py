"""When a channel's lookup uses another channel's dedup, on stand-ins for the kernels."""
from types import SimpleNamespace

import pytest
import torch

from kraken_b200.parallel import sparse_shard
from kraken_b200.parallel.sparse_shard import Dedup, SparseChannel


class Kernels:
    KrakenError = RuntimeError

    def __init__(self):
        self.called, self.args = [], {}

    def __getattr__(self, name):
        def call(*args, **kwargs):
            self.called.append(name)
            self.args[name] = args
        return call


def channel(world, cap_u, cap_s, salt=0):
    ch = object.__new__(SparseChannel)
    own = Dedup(cap_u, *(torch.zeros(1) for _ in range(6)))
    ch.__dict__.update(world=world, owner_world=world, cap=1000, cap_u=cap_u, cap_s=cap_s, salt=salt, spin=1, serial=0,
                       launches=0, hbits=4, lbits=4, ctrl=torch.zeros(8), cnt=None, slot_of=None, lset=None, pos=None,
                       win=None, slot_cache=None, lay=None, arena=SimpleNamespace(heap=None), _hkeys=torch.zeros(1),
                       table=SimpleNamespace(name="t", host=lambda: None, dim=4, device="cpu", optim=None,
                                             generation=1), _own=own,
                       dedup=own, _wait=int(world > 1), ugrad=torch.zeros(cap_u, 4), multi=None, _bag_of=None)
    return ch


# (ranks, bounds on the unique ids of the channel that has looked up and of the one that follows, bound per owner, shared)
@pytest.mark.parametrize("world,first,second,per_owner,shared", [
    (1, 500, 500, 500, True), (4, 500, 500, 300, True), (4, 500, 600, 300, True), (1, 500, 500, 300, True),
    (4, 501, 500, 500, False), (1, 501, 500, 500, False)])
def test_bounds_that_let_a_dedup_be_shared(monkeypatch, world, first, second, per_owner, shared):
    a, b = channel(world, first, per_owner), channel(world, second, per_owner)
    kernels = Kernels()
    monkeypatch.setattr(sparse_shard, "C", kernels)
    ids = torch.arange(10)
    a._lookup_phase(ids, True)
    kernels.called.clear()
    b._lookup_phase(ids, True, share_from=a)
    ran = "local_lookup" in kernels.called or "dedup_bucketize" in kernels.called
    assert ran == (not shared) and b.dedup is (a.dedup if shared else b._own) and b.lookups == (0 if shared else 1)


def test_another_owner_salt_needs_a_dedup_of_its_own(monkeypatch):
    monkeypatch.setattr(sparse_shard, "C", Kernels())
    a, b = channel(4, 500, 500, salt=1), channel(4, 500, 500, salt=2)
    b._lookup_phase(torch.arange(10), True, share_from=a)
    assert b.dedup is b._own


def given(kernels, name, tensor):
    return any(a is tensor for a in kernels.args[name])


# Pooled lookups of one id list for two tables, then their pushes, in both orders: every kernel gets the buffers of the one
# dedup; once those have been written again, the push of the table that shared them resolves its ids.
@pytest.mark.parametrize("world", [1, 4])
@pytest.mark.parametrize("sharer_first", [False, True])
def test_pooled_lookups_and_pushes_of_a_shared_dedup(monkeypatch, world, sharer_first):
    a, b = channel(world, 500, 500), channel(world, 500, 500)
    kernels = Kernels()
    monkeypatch.setattr(sparse_shard, "C", kernels)
    ids, off, lr = torch.arange(10), torch.tensor([0, 4, 10]), torch.ones(1)
    combine, scatter = ("local_combine", "local_push") if world == 1 else ("pull_combine", "push_scatter")
    _, ta = a.pull(ids, bag_offsets=off)
    _, tb = b.pull(ids, bag_offsets=off, share_from=a)
    assert given(kernels, combine, a.inv) and kernels.called.count("local_lookup") + kernels.called.count("dedup_bucketize") == 1
    kernels.called.clear()
    for ch, ticket in ((b, tb), (a, ta)) if sharer_first else ((a, ta), (b, tb)):
        ch.push(torch.zeros(2, 4), lr, ticket=ticket)
        assert given(kernels, scatter, a.inv) and given(kernels, "local_push" if world == 1 else "push_dispatch", a.off)
    assert "local_lookup" not in kernels.called and "dedup_bucketize" not in kernels.called
    a.pull(ids, bag_offsets=off)
    _, tb = b.pull(ids, bag_offsets=off, share_from=a)
    a.pull(ids + 5, bag_offsets=off)
    kernels.called.clear()
    b.push(torch.zeros(2, 4), lr, ticket=tb, ids=ids, bag_offsets=off)
    assert ("local_lookup" if world == 1 else "dedup_bucketize") in kernels.called and given(kernels, scatter, b._own.inv)


# A shard that was reallocated between a pull and its push: the slots are resolved again, by this rank alone.
@pytest.mark.parametrize("world", [1, 4])
@pytest.mark.parametrize("accumulated", [False, True])
def test_push_after_the_shard_was_reallocated(monkeypatch, world, accumulated):
    ch = channel(world, 500, 500)
    kernels = Kernels()
    monkeypatch.setattr(sparse_shard, "C", kernels)
    probe = "local_probe" if world == 1 else "pull_probe"
    for moved in (False, True):
        _, ticket = ch.pull(torch.arange(10))
        if moved:
            ch.table.generation += 1
        kernels.called.clear()
        if accumulated:
            ch.push_accumulated(torch.ones(1), ticket)
        else:
            ch.push(torch.zeros(10, 4), torch.ones(1), ticket=ticket)
        assert (probe in kernels.called) == moved and "dedup_bucketize" not in kernels.called
        if moved:
            assert kernels.called[0] == probe and kernels.args[probe][5] is False
