"""The one-GPU kernels of the sparse path (csrc/cuda/sparse_local.cu) against the CPU shard (B200 only)."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"

OPTIMS = [(kk.OptimType.kSGD, {}), (kk.OptimType.kSGD, {"momentum": "0.9"}),
          (kk.OptimType.kAdagrad, {"initial_accumulator_value": "0.1"}), (kk.OptimType.kAdam, {}),
          (kk.OptimType.kAdam, {"amsgrad": "true"}), (kk.OptimType.kRMSprop, {"momentum": "0.5", "centered": "true"})]


def make(dim, optim, conf, capacity=1 << 12, **options):
    kk.initialize("gpu", seed=11, table_capacity=capacity, **options)
    kk.init_model("m", optim, conf)
    kk.update_lr(0.05)
    t = kk.register_sparse_table("e", dim, torch.float32, kk.InitializerType.kNormal, {"stddev": "0.5"})
    shard = C.CpuShard(11)
    shard.init_model("m", optim, conf)
    shard.create_sparse_table(t, "e", dim, kk.InitializerType.kNormal, {"stddev": "0.5"})
    return t, shard


# Row widths on both sides of the vector width, of a power of two and of a block's threads; id counts around
# a block's rows (256 / chunks) and with one id only.
@pytest.mark.parametrize("optim,conf", OPTIMS)
@pytest.mark.parametrize("dim,ids", [(1, 255), (1, 257), (3, 85), (10, 26), (16, 65), (20, 52), (64, 1), (100, 11),
                                     (1028, 5), (1030, 3)])
def test_push_updates_rows_as_the_cpu_shard(optim, conf, dim, ids):
    t, shard = make(dim, optim, conf)
    torch.manual_seed(dim + ids)
    for step in range(3):
        batch = torch.randint(0, ids, (2 * ids + 1,)) if step else torch.arange(ids)
        rows = kk.pull_sparse_table(t, batch.to(DEV))
        uniq, inv = C.cpu_dedup(batch)
        # pull: a copy of the rows; after k updates the rows carry their rounding, see below
        assert torch.allclose(rows.cpu(), shard.pull_sparse(t, uniq)[inv], atol=2e-4)
        g = torch.randn(batch.numel(), dim)
        kk.push_sparse_table(t, batch.to(DEV), g.to(DEV))
        assert shard.push_sparse(t, uniq, C.cpu_segment_sum(g, inv, uniq.numel()), 0.05) == 0
    kk.native.engine().check()
    every = torch.arange(ids)
    # three updates of at most lr = 0.05 each, their gradient sums added in another order: 1e-5 relative per sum,
    # amplified where Adam and RMSprop divide two small numbers
    assert torch.allclose(kk.pull_sparse_table(t, every.to(DEV)).cpu(), shard.pull_sparse(t, every), atol=2e-4)
    ch = kk.native.engine().channels[t]
    assert float(ch.ugrad.abs().max()) == 0.0  # zero again for the next step


# Gradients that are a part of a flat tensor: contiguous, but on any 4-byte boundary.
@pytest.mark.parametrize("dim", [4, 6, 64])
@pytest.mark.parametrize("at", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("combined", [False, True])
def test_push_of_gradients_that_start_anywhere(dim, at, combined):
    kk.initialize("gpu", table_capacity=1 << 10)
    kk.init_model("m", kk.OptimType.kSGD, {})
    kk.update_lr(1.0)
    tids = [kk.register_sparse_table(f"e{k}", dim, torch.float32, kk.InitializerType.kConstant, {"value": "1"})
            for k in range(2)]
    ids = torch.arange(50, device=DEV)
    g = torch.randn(at + 50 * dim, device=DEV)[at:].view(50, dim)
    assert g.is_contiguous()
    if combined:
        kk.combine_pull_sparse_table(tids, [ids, ids])
        eng = kk.native.engine()
        ch, = eng.group_channels.values()
        both = torch.randn(at + 100 * dim, device=DEV)[at:].view(100, dim)
        ch.push(both, eng.lr_dev, ticket=eng.group_tickets.pop(tuple(tids))[0])
        wants = both.split(50)
    else:
        for t in tids:
            kk.pull_sparse_table(t, ids)
            kk.push_sparse_table(t, ids, g)
        wants = (g, g)
    kk.native.engine().check()
    for t, want in zip(tids, wants):
        assert torch.equal(kk.pull_sparse_table(t, ids), 1 - want)


def test_push_drops_the_gradient_of_an_unknown_id():
    t, _ = make(8, kk.OptimType.kSGD, {})
    known = torch.arange(4, device=DEV)
    before = kk.pull_sparse_table(t, known).clone()
    kk.push_sparse_table(t, torch.tensor([2, 900, 3], device=DEV), torch.ones(3, 8, device=DEV))
    with pytest.raises(kk.KrakenError):
        kk.native.engine().check()
    after = kk.pull_sparse_table(t, known)
    assert torch.allclose(after, before - 0.05 * torch.tensor([0, 0, 1.0, 1.0], device=DEV)[:, None])
    assert float(kk.native.engine().channels[t].ugrad.abs().max()) == 0.0


# Id counts around the threads of a block (256), around the grid that fills the chip, from which on a launch is not made
# early (592 blocks: 151297 ids), far above it, and with heavy repetition; rows that exist, rows that are created, and both.
@pytest.mark.parametrize("n,space", [(1, 1), (255, 300), (256, 256), (257, 40), (5003, 4000), (151_296, 100_000),
                                     (151_297, 100_000), (606207, 500_000), (606208, 500_000), (700_001, 9)])
def test_lookup_numbers_every_id_once_and_finds_its_row(n, space):
    t, shard = make(4, kk.OptimType.kSGD, {}, capacity=1 << 21, max_ids_per_call=800_000)
    torch.manual_seed(n)
    for _ in range(2):
        ids = torch.randint(0, space, (n,)) * 7919 - 3
        rows = kk.pull_sparse_table(t, ids.to(DEV))
        ch = kk.native.engine().channels[t]
        uniq, inv = ch.uniq[:int(ch.off[1])].cpu(), ch.inv[:n].cpu().long()
        assert torch.equal(uniq[inv], ids) and torch.equal(uniq.sort().values, torch.unique(ids))
        want, at = C.cpu_dedup(ids)
        assert torch.allclose(rows.cpu(), shard.pull_sparse(t, want)[at], atol=1e-5)  # Box-Muller in float32, rows of ~0.5
        assert int(ch.cnt[0]) == 0 and bool((ch.lset == -1).all())
    kk.native.engine().check()
    assert kk.native.engine().sparse[t].num_rows() <= space


@pytest.mark.parametrize("dim", [1, 3, 20, 64, 1028])
@pytest.mark.parametrize("mean", [False, True])
def test_bags_are_pooled_from_the_table(dim, mean):
    t, shard = make(dim, kk.OptimType.kSGD, {})
    torch.manual_seed(dim)
    lens = torch.tensor([0, 1, 3, 4, 5, 0, 8, 9, 17] * 30)
    off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)])
    ids = torch.randint(0, 90, (int(off[-1]),))
    w = torch.rand(ids.numel())
    out, ticket = kk.native.engine().pull_sparse_pooled(t, ids.to(DEV), off.to(DEV), weights=w.to(DEV), mean=mean,
                                                        patch_value=0.5)
    uniq, inv = C.cpu_dedup(ids)
    rows = shard.pull_sparse(t, uniq)[inv] * w[:, None]
    want = torch.zeros(lens.numel(), dim).index_add_(0, torch.repeat_interleave(torch.arange(lens.numel()), lens), rows)
    if mean:
        want = want / lens.clamp(min=1)[:, None]
    want[lens == 0] = 0.5
    assert torch.allclose(out.cpu(), want, atol=1e-4)  # up to 17 rows of ~0.5 in float32
    kk.native.engine().check()


def test_ids_beyond_the_unique_limit_are_reported():
    t, _ = make(4, kk.OptimType.kSGD, {}, max_ids_per_call=4096, max_unique_per_call=100)
    kk.pull_sparse_table(t, torch.arange(101, device=DEV))
    with pytest.raises(kk.KrakenError):
        kk.native.engine().check()
    assert torch.isfinite(kk.pull_sparse_table(t, torch.arange(100, device=DEV))).all()
    kk.native.engine().check()


# More unique ids than the bound for one owner, which a job of one GPU can set too: reported, and no consumer is handed
# slots that do not cover them all.
def test_ids_beyond_the_limit_per_owner_are_reported():
    kk.initialize("gpu", table_capacity=1 << 12, max_ids_per_call=4096, max_unique_per_call=1000, max_per_owner_per_call=100)
    kk.init_model("m", kk.OptimType.kSGD, {})
    a, b = (kk.register_sparse_table(n, d, torch.float32, kk.InitializerType.kConstant, {"value": "3"})
            for n, d in (("a", 16), ("b", 1)))
    eng = kk.native.engine()
    for n in (100, 101, 900):
        ids = torch.arange(n, device=DEV)
        for t, share, d in ((a, None, 16), (b, a, 1)):
            rows, inv, ticket = eng.pull_sparse_unique(t, ids, share_with=share, in_place=True)
            assert ticket.slots is None or ticket.slots.numel() >= n
            got = rows[inv[:n].long()]
            assert got.shape == (n, d) and int((got == 3).all(1).sum()) == min(n, 100)  # the others read as zeros
            if n > 100:
                with pytest.raises(kk.KrakenError):
                    eng.channels[t].check()
            eng.push_sparse_accumulated(t, ticket)
        eng.check()


# The first occurrence of an id is updated from the caller's gradients, the others from their sum; widths on both sides
# of the line below which every gradient is summed (8), with bags (weights, mean, empty ones) and without, and further
# pushes of the same shape in which other ids are the ones that repeat.
@pytest.mark.parametrize("dim", [7, 8, 10, 20, 64, 1028])
@pytest.mark.parametrize("bags", [None, "sum", "mean"])
def test_push_of_ids_that_occur_once_and_of_ids_that_repeat(dim, bags):
    t, shard = make(dim, kk.OptimType.kAdagrad, {"initial_accumulator_value": "0.1"}, max_ids_per_call=4096)
    torch.manual_seed(dim)
    eng = kk.native.engine()
    for step in range(3):
        once = torch.randperm(600)[:300] + 1000 * (step % 2)
        ids = torch.cat([once, torch.randint(0, 600, (200,)) + 1000, torch.full((40,), 7)])
        ids = ids[torch.randperm(ids.numel())]
        n = ids.numel()
        uniq, inv = C.cpu_dedup(ids)
        if bags is None:
            kk.pull_sparse_table(t, ids.to(DEV))
            g = torch.randn(n, dim)
            kk.push_sparse_table(t, ids.to(DEV), g.to(DEV))
        else:
            lens = torch.tensor([0, 1, 5, 4, 8, 0, 9] * 20)
            off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)])
            assert int(off[-1]) == n
            w = torch.rand(n)
            _, ticket = eng.pull_sparse_pooled(t, ids.to(DEV), off.to(DEV), weights=w.to(DEV), mean=bags == "mean")
            gb = torch.randn(lens.numel(), dim)
            eng.push_sparse_pooled(t, ticket, gb.to(DEV), ids.to(DEV))
            g = (gb / lens.clamp(min=1)[:, None] if bags == "mean" else gb).repeat_interleave(lens, 0) * w[:, None]
        shard.pull_sparse(t, uniq)
        assert shard.push_sparse(t, uniq, C.cpu_segment_sum(g, inv, uniq.numel()), 0.05) == 0
    eng.check()
    every = torch.arange(1600)
    every = every[(every < 600) | (every >= 1000)]
    # three Adagrad updates of at most 0.05 / sqrt(0.1) * |g|, their sums of up to 41 terms in another order
    assert torch.allclose(kk.pull_sparse_table(t, every.to(DEV)).cpu(), shard.pull_sparse(t, every), atol=2e-4)
    assert float(eng.channels[t].ugrad.abs().max()) == 0.0


# Row counts around the launch lines of the update: a row of 64 floats has 16 threads, so a block takes 8 rows; launches of
# fewer than 1184 blocks are made early, and beyond 11840 blocks (94720 rows) a block takes further rows.  The same for the
# segment sum with 16 rows a block: 592 and 2368 blocks (9472 and 37888 rows).
@pytest.mark.parametrize("rows", [9464, 9465, 9473, 37889, 94720, 94721, 200_003])
@pytest.mark.parametrize("bags", [False, True])
def test_push_around_the_launch_lines(rows, bags):
    n = rows + rows // 3
    t, shard = make(64, kk.OptimType.kAdam, {"eps": "0.01"}, capacity=1 << 19, max_ids_per_call=n)
    torch.manual_seed(rows)
    eng = kk.native.engine()
    ids = torch.cat([torch.arange(rows), torch.randint(0, rows, (n - rows,))])[torch.randperm(n)]
    uniq, inv = C.cpu_dedup(ids)
    shard.pull_sparse(t, uniq)
    for _ in range(2):
        if bags:
            off = torch.cat([torch.arange(0, n, 3), torch.tensor([n])])
            _, ticket = eng.pull_sparse_pooled(t, ids.to(DEV), off.to(DEV))
            gb = torch.randn(off.numel() - 1, 64)
            eng.push_sparse_pooled(t, ticket, gb.to(DEV), ids.to(DEV))
            g = gb.repeat_interleave(off[1:] - off[:-1], 0)
        else:
            kk.pull_sparse_table(t, ids.to(DEV))
            g = torch.randn(n, 64)
            kk.push_sparse_table(t, ids.to(DEV), g.to(DEV))
        assert shard.push_sparse(t, uniq, C.cpu_segment_sum(g, inv, uniq.numel()), 0.05) == 0
    eng.check()
    got, found = eng.sparse[t].lookup(uniq.to(DEV))
    assert bool(found.bool().all())
    want = shard.pull_sparse(t, uniq)
    # rows of ~0.5 from a float32 Box-Muller: 1e-5; sums of up to ~6 values of ~1 in another order: 1e-6 each, of which an
    # update passes on at most 0.05 / eps = 5 times that where a sum is near zero, and far less elsewhere
    assert torch.allclose(got.cpu(), want, atol=2e-5)


# Offsets that leave ids out in front of the first bag, behind the last, or altogether, after pushes of more bags: such an
# occurrence has no gradient, whichever occurrence of its id the lookup found first.  Momentum moves every row that was
# looked up, with a gradient of zero too.
@pytest.mark.parametrize("dim", [7, 10, 64])
@pytest.mark.parametrize("mode", ["sum", "mean", "weights"])
def test_ids_outside_every_bag_have_no_gradient(dim, mode):
    t, shard = make(dim, kk.OptimType.kSGD, {"momentum": "0.9"}, max_ids_per_call=4096)
    torch.manual_seed(dim)
    eng = kk.native.engine()
    for head, lens, tail in [(0, [3, 2, 4] * 40, 0), (7, [2, 0, 3] * 5, 0), (0, [1, 4], 200), (300, [5], 300), (40, [], 0),
                             (5, [0, 0], 5), (0, [3, 1] * 30, 60)]:
        inside = sum(lens)
        lens = torch.tensor(lens, dtype=torch.int64)
        off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)]) + head
        ids = torch.randint(0, 300, (head + inside + tail,))
        w = torch.rand(ids.numel()) if mode == "weights" else None
        _, ticket = eng.pull_sparse_pooled(t, ids.to(DEV), off.to(DEV), weights=w.to(DEV) if w is not None else None,
                                           mean=mode == "mean")
        gb = torch.randn(lens.numel(), dim)
        eng.push_sparse_pooled(t, ticket, gb.to(DEV), ids.to(DEV))
        g = torch.zeros(ids.numel(), dim)
        per_bag = gb / lens.clamp(min=1)[:, None] if mode == "mean" else gb
        g[head:head + inside] = per_bag.repeat_interleave(lens, 0)
        if w is not None:
            g *= w[:, None]
        uniq, inv = C.cpu_dedup(ids)
        shard.pull_sparse(t, uniq)
        assert shard.push_sparse(t, uniq, C.cpu_segment_sum(g, inv, uniq.numel()), 0.05) == 0
    eng.check()
    every = torch.arange(300)
    # seven updates of 0.05 times sums of ~10 values of ~1, added in another order
    assert torch.allclose(kk.pull_sparse_table(t, every.to(DEV)).cpu(), shard.pull_sparse(t, every), atol=2e-4)


# The step of dense tables on one GPU with DCT, residual and threshold carried over steps and refreshed every second:
# tables around the size below which one travels whole (256) and around a block's elements (4096).
@pytest.mark.parametrize("optim,conf", OPTIMS)
def test_dct_step_matches_the_cpu_compressor(optim, conf):
    kk.initialize("gpu", emitter_type=kk.EmitterType.kDCT, life_span=2, eta=0.75)
    kk.init_model("m", optim, conf)
    kk.update_lr(0.05)
    torch.manual_seed(3)
    sizes = [1, 255, 256, 257, 4095, 4097, 9000]
    ids = [kk.register_dense_table(f"w{n}", torch.randn(n)) for n in sizes]
    shard = C.CpuShard(0)
    shard.init_model("m", optim, conf)
    states = {i: C.DctState() for i in ids}
    for i, n, v in zip(ids, sizes, kk.combine_pull_dense_table(ids)):
        shard.create_dense_table(i, f"w{n}", v.cpu().clone())
    for step in range(5):
        for i, n in zip(ids, sizes):
            g = torch.randn(n)
            kk.push_dense_table(i, g.to(DEV))
            packed = C.cpu_dct_compress(g, 2, 0.75, states[i])
            if packed is not None:
                shard.push_dense_coo(i, packed[0], packed[1], 0.05)
            else:
                shard.push_dense(i, g, 0.05)
        for i, v in zip(ids, kk.combine_pull_dense_table(ids)):
            # the same float32 formulas element by element, compiled by two compilers
            assert torch.allclose(v.cpu(), shard.pull_dense(i).view(-1), atol=1e-5), (step, i)
    kk.native.engine().check()


def test_dct_that_keeps_nothing_is_refused_at_every_step():
    kk.initialize("gpu", emitter_type=kk.EmitterType.kDCT, life_span=4, eta=0.999)
    kk.init_model("m", kk.OptimType.kSGD, {})
    kk.update_lr(0.5)
    t = kk.register_dense_table("w", torch.ones(300))
    kk.push_dense_table(t, torch.ones(300, device=DEV))
    for _ in range(3):
        with pytest.raises(kk.KrakenError, match="keeps no element"):
            kk.pull_dense_table(t)
    bucket = kk.native.engine().bucket
    assert torch.equal(bucket.param_view(t, (300,)), torch.ones(300, device=DEV))
    assert torch.equal(bucket.grad_view(t, (300,)), torch.ones(300, device=DEV))


# Two tables that share one dedup, with another lookup of the first between pull and push of the second: the second's
# ticket is out of date then and its ids are resolved again.
# A third case has the second table's buffers smaller than the first's: it runs its own dedup.
@pytest.mark.parametrize("between", [False, True, "smaller"])
def test_tables_that_share_a_dedup(between):
    kk.initialize("gpu", table_capacity=1 << 12, **({} if between == "smaller" else {"max_ids_per_call": 4096}))
    kk.init_model("m", kk.OptimType.kSGD, {})
    kk.update_lr(1.0)
    a, b = (kk.register_sparse_table(n, d, torch.float32, kk.InitializerType.kConstant, {"value": "3"})
            for n, d in (("a", 16), ("b", 1)))
    eng = kk.native.engine()
    if between == "smaller":
        kk.pull_sparse_table(a, torch.arange(2000, device=DEV))
        kk.pull_sparse_table(b, torch.arange(600, device=DEV))
        assert eng.channels[a].cap_u > eng.channels[b].cap_u
    ids = torch.randint(0, 50, (200,), device=DEV)
    off = torch.arange(0, 201, 4, device=DEV)
    pa, ta = eng.pull_sparse_pooled(a, ids, off)
    pb, tb = eng.pull_sparse_pooled(b, ids, off, share_with=a)
    assert torch.equal(pa, torch.full((50, 16), 12.0, device=DEV)) and torch.equal(pb, torch.full((50, 1), 12.0, device=DEV))
    if between is True:
        kk.pull_sparse_table(a, torch.arange(100, 400, device=DEV))
    eng.push_sparse_pooled(b, tb, torch.ones(50, 1, device=DEV), ids)
    eng.push_sparse_pooled(a, ta, torch.ones(50, 16, device=DEV), ids)
    eng.check()
    every = torch.arange(50, device=DEV)
    count = torch.bincount(ids, minlength=50).float()[:, None]
    for t, d in ((a, 16), (b, 1)):
        rows, found = eng.sparse[t].lookup(every)
        assert torch.equal(rows[found.bool()], (3 - count).expand(-1, d)[found.bool()])


def test_a_shared_dedup_outlives_the_channel_that_ran_it():
    from kraken_b200.parallel.sparse_shard import GpuSparseTable, SparseChannel
    dev = torch.device("cuda", torch.cuda.current_device())
    lr = torch.ones(1, device=dev)
    tables = [GpuSparseTable(k, f"t{k}", 8, kk.InitializerType.kConstant, {"value": "3"}, kk.OptimType.kSGD, {}, 0, 1 << 10, 1,
                             dev) for k in range(2)]
    first, second = (SparseChannel(t, 0, 1, 256) for t in tables)
    ids = torch.tensor([5, 6, 5, 7], device=dev)
    first.pull(ids)
    _, ticket = second.pull(ids, share_from=first)
    del first
    second.push(torch.ones(4, 8, device=dev), lr, ticket=ticket)
    _, ticket = second.pull(ids, share_from=second)
    second.push(torch.ones(4, 8, device=dev), lr, ticket=ticket)
    rows, found = tables[1].lookup(torch.tensor([5, 6, 7], device=dev))
    assert bool(found.bool().all()) and torch.equal(rows[:, 0].cpu(), torch.tensor([-1.0, 1.0, 1.0]))
    second.check()
