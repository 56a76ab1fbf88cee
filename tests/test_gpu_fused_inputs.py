"""Lookups that write the MLP's input themselves, against the modules called one by one (B200 only)."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200.models import MultiHotWideAndDeep, WideAndDeep

pytestmark = pytest.mark.gpu
DEV = "cuda"
FIELDS, BATCH, SPACE = 5, 37, 150


def multihot(dim):
    return MultiHotWideAndDeep(num_fields=FIELDS, num_dense=3, dim=dim, hidden=(32, 16), mean_fields=(1, 4))


def wide_deep(dim):
    return WideAndDeep(num_fields=FIELDS, num_dense=3, dim=dim, hidden=(32, 16))


def batch(kind, seed):
    g = torch.Generator().manual_seed(seed)
    dense = torch.randn(BATCH, 3, generator=g).to(DEV)
    if kind is wide_deep:
        return dense, torch.randint(0, SPACE, (BATCH, FIELDS), generator=g).to(DEV)
    lens = torch.randint(0, 6, (BATCH * FIELDS,), generator=g)
    off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)])
    ids = torch.randint(0, SPACE, (int(off[-1]),), generator=g)
    return dense, kk.JaggedTensor(ids.to(DEV), off.to(DEV))


def train(kind, dim, optim, general, steps=3, order=None, freeze=()):
    kk.initialize("gpu", table_capacity=1 << 12, max_ids_per_call=4096, seed=5)
    torch.manual_seed(2)
    model = kind(dim).to(DEV)
    opt = kk.Optimizer("m", model.named_parameters(), 0.05, optim)
    if general:  # a hook, even one that does nothing, wants what the module by itself takes in
        model.mlp.register_forward_pre_hook(lambda m, i: None)
    tables = [getattr(model.wide, "embedding", model.wide).sparse_table, model.deep.sparse_table]
    for k in freeze:
        tables[k].requires_grad_(False)
    outs = []
    for step in range(steps):
        if order == "two forwards":   # the first one's lookup is no longer the latest when its backward runs
            a, b = model(*batch(kind, 2 * step)), model(*batch(kind, 2 * step + 1))
            out = torch.cat([a, b])
        else:
            out = model(*batch(kind, step))
            if order == "scoring between":
                with torch.no_grad():
                    model(*batch(kind, 100 + step))
        (out * torch.linspace(-1, 1, out.numel(), device=DEV)).sum().backward()
        opt.step()
        outs.append(out.detach().clone())
    eng = kk.native.engine()
    eng.check()
    every = torch.arange(SPACE, device=DEV)
    rows = [eng.sparse[t.table_id()].lookup(every)[0].clone() for t in tables]
    weights = [p.detach().clone() for p in model.mlp.parameters()]
    shared = eng.channels[tables[0].table_id()].dedup is eng.channels[tables[1].table_id()].dedup
    kk.stop()
    return outs, rows, weights, shared


def same(a, b):
    """The same products rounded at the same places; float32 sums in another order (a few dozen terms: 1e-5), and now and
    then one of them on the other side of a bfloat16 rounding (2^-8 of one term) in a later step."""
    for x, y in zip(a, b):
        assert float((x - y).norm()) <= 2e-3 * float(y.norm()) + 1e-6


@pytest.mark.parametrize("kind,dims", [(multihot, (4, 8, 12, 16, 64, 6)), (wide_deep, (4, 8, 16, 64, 12, 6))])
@pytest.mark.parametrize("optim", [kk.SGD(), kk.Adagrad(initial_accumulator_value=0.1)], ids=["sgd", "adagrad"])
def test_trains_as_the_modules_by_themselves(kind, dims, optim):
    for dim in dims:  # among them widths that only the general path takes
        fused, general = (train(kind, dim, optim, g) for g in (False, True))
        assert torch.allclose(fused[0][0], general[0][0], rtol=1e-4, atol=1e-5)   # one step: nothing to amplify
        for a, b in zip(fused[:3], general[:3]):
            same(a, b)
        if dim in (8, 16, 64):
            assert fused[3]   # one dedup for both tables


@pytest.mark.parametrize("kind", [multihot, wide_deep])
@pytest.mark.parametrize("order", ["two forwards", "scoring between"])
def test_backward_of_a_lookup_that_is_not_the_latest(kind, order):
    fused, general = (train(kind, 8, kk.SGD(), g, order=order) for g in (False, True))
    for a, b in zip(fused[:3], general[:3]):
        same(a, b)


@pytest.mark.parametrize("freeze", [(0,), (1,), (0, 1)])
def test_a_frozen_table_keeps_its_rows(freeze):
    fused, general = (train(wide_deep, 8, kk.SGD(), g, freeze=freeze) for g in (False, True))
    for a, b in zip(fused[:3], general[:3]):
        same(a, b)


def test_more_ids_than_are_read_in_place():
    """Above half a million ids the rows of both tables are gathered first."""
    n, space = (1 << 19) // FIELDS + 2, 20_000
    assert n * FIELDS > 1 << 19
    g = torch.Generator().manual_seed(1)
    dense, ids = torch.randn(n, 3, generator=g).to(DEV), torch.randint(0, space, (n, FIELDS), generator=g).to(DEV)
    results = []
    for general in (False, True):
        kk.initialize("gpu", table_capacity=1 << 16, max_ids_per_call=n * FIELDS, seed=5)
        torch.manual_seed(2)
        model = wide_deep(8).to(DEV)
        opt = kk.Optimizer("m", model.named_parameters(), 0.05, kk.SGD())
        if general:
            model.mlp.register_forward_pre_hook(lambda m, i: None)
        out = model(dense, ids)
        (out * torch.linspace(-1, 1, n, device=DEV)).sum().backward()
        opt.step()
        eng = kk.native.engine()
        eng.check()
        every = torch.arange(space, device=DEV)
        rows = [eng.sparse[t.table_id()].lookup(every)[0].clone() for t in (model.wide.sparse_table, model.deep.sparse_table)]
        results.append((out.detach().clone(), *rows, *[p.detach().clone() for p in model.mlp.parameters()]))
        kk.stop()
    assert torch.allclose(results[0][0], results[1][0], rtol=1e-4, atol=1e-5)
    same(results[0][1:], results[1][1:])
