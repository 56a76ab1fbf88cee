"""Growth decisions on sampled row counters (B200 only)."""
import pytest
import torch

import kraken_b200.pytorch as kk

pytestmark = pytest.mark.gpu
DEV = "cuda"


# Tables that fill up call by call, alone and in a combined call, with and without housekeeping between the calls: the
# bound never falls below the rows there are, no lookup finds a full table, and no row is lost by growing.
@pytest.mark.parametrize("combined", [False, True])
@pytest.mark.parametrize("end_step", [False, True])
def test_tables_grow_before_they_are_full(combined, end_step):
    kk.initialize("gpu", table_capacity=1 << 10)
    eng = kk.native.engine()
    kk.init_model("m", kk.OptimType.kSGD, {})
    kk.update_lr(1.0)
    tids = [kk.register_sparse_table(f"t{k}", 4, torch.float32, kk.InitializerType.kConstant, {"value": "1"})
            for k in range(3)]
    n = 500
    for step in range(12):
        ids = [torch.arange(n, device=DEV) + step * n // (k + 1) for k in range(3)]
        g = [torch.ones(n, 4, device=DEV) for _ in tids]
        if combined:
            kk.combine_pull_sparse_table(tids, ids)
            kk.combine_push_sparse_table(tids, ids, g)
        else:
            for t, i, x in zip(tids, ids, g):
                kk.pull_sparse_table(t, i)
                kk.push_sparse_table(t, i, x)
        if end_step:
            eng.end_step()
        for k, t in enumerate(tids):
            table = eng.sparse[t]
            rows = table.num_rows()
            assert rows == n + step * n // (k + 1) and table.rows_bound() >= rows and rows < 0.9 * table.capacity
    eng.check()
    for k, t in enumerate(tids):
        last = 11 * n // (k + 1)
        ids = torch.arange(n + last, device=DEV)
        times = torch.zeros(n + last, device=DEV)
        for step in range(12):
            times[step * n // (k + 1):step * n // (k + 1) + n] += 1
        rows, found = eng.sparse[t].lookup(ids)
        assert bool(found.bool().all()) and torch.equal(rows, (1 - times)[:, None].expand(-1, 4))


def test_a_combined_lookup_is_not_bounded_by_the_tables_own_buffers():
    kk.initialize("gpu", table_capacity=1 << 10)
    eng = kk.native.engine()
    kk.init_model("m", kk.OptimType.kSGD, {})
    tids = [kk.register_sparse_table(f"t{k}", 4, torch.float32, kk.InitializerType.kConstant, {"value": "1"})
            for k in range(2)]
    for t in tids:
        kk.pull_sparse_table(t, torch.arange(10, device=DEV))  # buffers for 1024 ids
    ids = [torch.arange(5000, device=DEV)] * 2
    rows = kk.combine_pull_sparse_table(tids, ids)
    eng.check()
    for t, r in zip(tids, rows):
        assert torch.equal(r, torch.ones(5000, 4, device=DEV))
        assert eng.sparse[t].num_rows() == 5000 <= eng.sparse[t].rows_bound() and eng.sparse[t].capacity > 5000 / 0.6


def test_imported_rows_count_while_a_sample_is_in_flight():
    kk.initialize("gpu", table_capacity=1 << 12)
    eng = kk.native.engine()
    kk.init_model("m", kk.OptimType.kSGD, {})
    t = kk.register_sparse_table("t", 4, torch.float32, kk.InitializerType.kConstant, {"value": "1"})
    eng.counters.start()                      # taken before the rows arrive
    eng.sparse[t].import_rows(torch.arange(2000, device=DEV), torch.zeros(2000, 4, device=DEV))
    assert eng.counters.poll(wait=True) and eng.sparse[t].rows_bound() >= 2000
    eng.counters.start()
    assert eng.counters.poll(wait=True) and eng.sparse[t].rows_bound() == 2000


def test_replays_count_the_rows_they_may_create():
    """Replays create rows that no eager call announced; a sample of the counters may be many replays old when the host runs
    ahead, so it is held back here.  The eager lookup behind them then grows the table in time."""
    from kraken_b200.utils.graph import GraphedStep
    kk.initialize("gpu", table_capacity=1 << 12, max_ids_per_call=1024)
    eng = kk.native.engine()
    emb = kk.Embedding(4, initializer=kk.ConstantInitializer(1.0), name="t")
    kk.Optimizer("m", emb.named_parameters(), 0.5, kk.SGD())
    ids = torch.arange(400, device=DEV)
    step = GraphedStep(lambda x: emb(x).sum().detach(), (ids,), warmup=1)
    t = emb.sparse_table.table_id()
    table = eng.sparse[t]
    eng.counters.poll(wait=True)
    eng.counters.start()
    eng.counters.poll = lambda wait=False: False          # "not landed yet"
    for k in range(1, 5):
        step(ids + 400 * k)
        assert table.rows_bound() >= 400 * (k + 1)
    del eng.counters.poll
    kk.pull_sparse_table(t, torch.arange(10_000, 11_000, device=DEV))
    assert table.num_rows() == 400 * 5 + 1000 and table.num_rows() <= 0.6 * table.capacity and step.recaptures == 0
    assert float(step(ids)) == 1600.0 and step.recaptures == 1
    eng.check()


def test_a_refused_lookup_leaves_no_sample_for_a_captured_one():
    """The sample's copy and event belong to the call that decided on them: in a graph they would be replayed, and the event
    could not be asked for any more."""
    kk.initialize("gpu", table_capacity=1 << 10)
    eng = kk.native.engine()
    kk.init_model("m", kk.OptimType.kSGD, {})
    t = kk.register_sparse_table("t", 4, torch.float32, kk.InitializerType.kConstant, {"value": "1"})
    ids = torch.arange(500, device=DEV)
    kk.pull_sparse_table(t, ids)
    eng.counters.poll(wait=True)
    with pytest.raises(kk.KrakenError, match="exceed the channel capacity"):
        kk.pull_sparse_table(t, torch.arange(5000, device=DEV))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rows = kk.pull_sparse_table(t, ids)
    graph.replay()
    assert torch.equal(rows, torch.ones(500, 4, device=DEV))
    for _ in range(3):
        eng.end_step()
        torch.cuda.synchronize()
    assert eng.sparse[t].sampled_rows == 500


def test_an_engine_that_is_let_go_is_freed_at_once():
    """Tables and exchange buffers are gigabytes: nothing may keep them until the garbage collector looks for cycles."""
    import gc
    import weakref
    kk.initialize("gpu", table_capacity=1 << 12)
    eng = kk.native.engine()
    kk.init_model("m", kk.OptimType.kSGD, {})
    a, b = (kk.register_sparse_table(n, 8, torch.float32, kk.InitializerType.kConstant, {"value": "1"}) for n in "ab")
    ids, off = torch.arange(64, device=DEV), torch.arange(0, 65, 2, device=DEV)
    eng.pull_sparse_pooled(a, ids, off)
    eng.pull_sparse_pooled(b, ids, off, share_with=a)
    kk.combine_pull_sparse_table([a, b], [ids, ids])
    eng.end_step()
    gone = [weakref.ref(x) for x in (eng.channels[a], eng.channels[b], eng.sparse[a])]
    gc.collect()
    gc.disable()
    try:
        kk.stop()
        del eng
        assert [r() is None for r in gone] == [True] * 3
    finally:
        gc.enable()
