"""A slot's value, optimizer state and step counter side by side: the pitch rule, and that nothing overlaps."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200.parallel.sparse_shard import record_pitch


@pytest.mark.parametrize("counts", [False, True])
@pytest.mark.parametrize("slabs", [0, 1, 2, 3])
def test_a_record_holds_its_parts_and_pads_little(slabs, counts):
    for dim in range(1, 300):
        used = dim * (1 + slabs)
        pitch = record_pitch(dim, used, counts)
        assert pitch >= used
        if slabs == 0 and not counts:
            assert pitch == dim
        if dim % 4 == 0:
            assert pitch % 4 == 0      # every part of every record starts on 16 bytes
        assert pitch <= 8 or 4 * pitch <= 5 * (used + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("optim,conf", [(kk.OptimType.kSGD, {}), (kk.OptimType.kSGD, {"momentum": "0.9"}),
                                        (kk.OptimType.kAdagrad, {"initial_accumulator_value": "0.1"}),
                                        (kk.OptimType.kAdam, {}), (kk.OptimType.kAdam, {"amsgrad": "true"}),
                                        (kk.OptimType.kRMSprop, {"momentum": "0.5", "centered": "true"})])
@pytest.mark.parametrize("dim", [1, 2, 3, 4, 5, 8, 10, 16, 17, 20, 64])
def test_parts_of_a_record_keep_apart(optim, conf, dim):
    """Every column of an imported table comes back bit for bit, also after the table has been rebuilt larger."""
    kk.initialize("gpu", table_capacity=1 << 8)
    kk.init_model("m", optim, conf)
    t = kk.register_sparse_table("e", dim, torch.float32, kk.InitializerType.kConstant, {"value": "0"})
    eng = kk.native.engine()
    table = eng.sparse[t]
    torch.manual_seed(dim)
    n = 100
    ids = torch.randperm(100_000)[:n].cuda()
    states = {int(st): torch.randn(n, dim).cuda()
              for st, on in zip(table.optim_info["slab_state_types"], table.optim_info["slabs"]) if on}
    cols = {"ids": ids, "vals": torch.randn(n, dim).cuda(), "states": states,
            "states_i": {0: torch.randint(1, 1000, (n,)).cuda()} if table.steps is not None else {}}
    eng.import_sparse(t, cols)
    for _ in range(2):
        out = eng.export_sparse(t)
        a, b = out["ids"].argsort(), ids.argsort()
        assert torch.equal(out["ids"][a], ids[b]) and torch.equal(out["vals"][a], cols["vals"][b])
        assert out["states"].keys() == states.keys() and out["states_i"].keys() == cols["states_i"].keys()
        for st in states:
            assert torch.equal(out["states"][st][a], states[st][b])
        for st in cols["states_i"]:
            assert torch.equal(out["states_i"][st][a], cols["states_i"][st][b])
        assert table.reserve(1000) or table.capacity > 1000
    # a slot that holds no row yet: value 0, state as the optimizer starts it
    free = table.keys == -1
    fill = table.optim_info["initial_accumulator_value"] if table.optim_info["type"] == 0 else 0.0
    assert bool((table.val[free] == 0).all())
    for k, s in enumerate(table.slabs):
        assert s is None or bool((s[free] == (fill if k == 0 else 0.0)).all())
    assert table.steps is None or bool((table.steps[free] == 0).all())


# Pitches that are no multiple of the four floats of a thread's store, records larger than one; totals with a rest.
@pytest.mark.gpu
@pytest.mark.parametrize("rows,pitch,at,dim", [(1, 1, 0, 1), (3, 1, 0, 0), (5, 3, 1, 2), (7, 5, 2, 1), (333, 30, 10, 10),
                                               (1000, 128, 64, 64), (300_001, 7, 3, 3)])
def test_records_are_filled_by_column(rows, pitch, at, dim):
    from kraken_b200._native import C
    records = torch.full((rows, pitch), 7.0, device="cuda")
    C.fill_records(records, at, dim, 0.1)
    want = torch.zeros(rows, pitch, device="cuda")
    want[:, at:at + dim] = 0.1
    assert torch.equal(records, want)
    with pytest.raises(RuntimeError):
        C.fill_records(records, at, pitch - at + 1, 0.1)


@pytest.mark.gpu
def test_a_reshard_resets_records_in_one_pass(monkeypatch):
    """Every part of a slot lies in one record, so what a reshard clears is cleared once and not by columns; rows that stay
    keep their columns, free slots start as the optimizer starts them."""
    kk.initialize("gpu", table_capacity=1 << 8)
    kk.init_model("m", kk.OptimType.kAdagrad, {"initial_accumulator_value": "0.1"})
    t = kk.register_sparse_table("e", 5, torch.float32, kk.InitializerType.kConstant, {"value": "0"})
    eng = kk.native.engine()
    table = eng.sparse[t]
    torch.manual_seed(1)
    ids = torch.randperm(1000)[:60].cuda()
    state = int(table.optim_info["slab_state_types"][0])
    cols = {"ids": ids, "vals": torch.randn(60, 5).cuda(), "states": {state: torch.rand(60, 5).cuda()}, "states_i": {}}
    eng.import_sparse(t, cols)
    resets = []
    whole = table._reset_records
    monkeypatch.setattr(table, "_reset_records", lambda: (resets.append(1), whole()))
    eng.owner_world = 2   # as if another rank had held rows: all come back to this one
    assert eng.reshard(1) == 0 and resets == [1]
    out = eng.export_sparse(t)
    a, b = out["ids"].argsort(), ids.argsort()
    assert torch.equal(out["ids"][a], ids[b]) and torch.equal(out["vals"][a], cols["vals"][b])
    assert torch.equal(out["states"][state][a], cols["states"][state][b])
    free = table.keys == -1
    assert bool((table.val[free] == 0).all()) and bool((table.slabs[0][free] == 0.1).all())


# Row widths around the groups of lanes that move a row, rows around a warp's and a block's; some slots of a warp hold a row.
@pytest.mark.gpu
@pytest.mark.parametrize("dim", [7, 8, 9, 15, 16, 31, 32, 33])
@pytest.mark.parametrize("rows", [1, 31, 33, 257])
def test_rows_are_moved_whole(dim, rows):
    kk.initialize("gpu", table_capacity=1 << 10)
    kk.init_model("m", kk.OptimType.kAdam, {"amsgrad": "true"})
    t = kk.register_sparse_table("e", dim, torch.float32, kk.InitializerType.kConstant, {"value": "0"})
    eng = kk.native.engine()
    table = eng.sparse[t]
    torch.manual_seed(dim + rows)
    ids = torch.randperm(100_000)[:rows].cuda()
    states = {int(st): torch.randn(rows, dim).cuda() for st in table.optim_info["slab_state_types"]}
    cols = {"ids": ids, "vals": torch.randn(rows, dim).cuda(), "states": states,
            "states_i": {0: torch.randint(1, 1000, (rows,)).cuda()}}
    eng.import_sparse(t, cols)
    out, want = eng.export_sparse(t), ids.argsort()
    got = out["ids"].argsort()
    assert torch.equal(out["vals"][got], cols["vals"][want]) and torch.equal(out["states_i"][0][got], cols["states_i"][0][want])
    assert all(torch.equal(out["states"][st][got], states[st][want]) for st in states)
    half = table.export(filter_mode=3, min_steps=500)   # some rows of a warp only
    kept = cols["states_i"][0][want] >= 500
    got = half["ids"].argsort()
    assert torch.equal(half["ids"][got], ids[want][kept]) and torch.equal(half["vals"][got], cols["vals"][want][kept])
