"""The multi-hot Wide&Deep model on the GPU engine: its two tables share a lookup where they can (B200 only)."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200.models import MultiHotWideAndDeep

pytestmark = pytest.mark.gpu
DEV = "cuda"
FIELDS, BATCH = 6, 32


def make(**options):
    kk.initialize("gpu", table_capacity=1 << 12, max_ids_per_call=4096, seed=5, **options)
    torch.manual_seed(2)
    model = MultiHotWideAndDeep(num_fields=FIELDS, num_dense=3, dim=8, hidden=(32,), mean_fields=(1, 4)).to(DEV)
    opt = kk.Optimizer("m", model.named_parameters(), 0.1, kk.SGD())
    return model, opt


def batch(seed):
    g = torch.Generator().manual_seed(seed)
    lens = torch.randint(0, 5, (BATCH * FIELDS,), generator=g)
    off = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)])
    ids = torch.randint(0, 200, (int(off[-1]),), generator=g)
    dense = torch.randn(BATCH, 3, generator=g)
    return dense.to(DEV), kk.JaggedTensor(ids.to(DEV), off.to(DEV))


def rows(table):
    ids = torch.arange(200, device=DEV)
    return kk.native.engine().sparse[table.table_id()].lookup(ids)[0].clone()


@pytest.mark.parametrize("frozen", ["wide", "deep", "both", "none"])
def test_a_frozen_table_is_not_trained(frozen):
    model, opt = make()
    tables = {"wide": model.wide.embedding.sparse_table, "deep": model.deep.sparse_table}
    for seed in range(2):
        opt.zero_grad()
        model(*batch(seed)).sum().backward()
        opt.step()
    for name, t in tables.items():
        t.requires_grad_(frozen not in (name, "both"))
    before = {name: rows(t) for name, t in tables.items()}
    opt.zero_grad()
    model(*batch(0)).sum().backward()
    opt.step()
    for name, t in tables.items():
        assert torch.equal(rows(t), before[name]) == (frozen in (name, "both")), name
    kk.native.engine().check()


# The same steps with the shared lookup and, because of a hook that does nothing, with one lookup per table.
def test_shared_and_separate_lookups_train_alike():
    results = []
    for hook in (False, True):
        model, opt = make()
        if hook:
            model.wide.register_forward_hook(lambda m, i, o: None)
        outs = []
        for seed in range(3):
            opt.zero_grad()
            out = model(*batch(seed))
            out.sum().backward()
            opt.step()
            outs.append(out.detach().clone())
        eng = kk.native.engine()
        eng.check()
        wide, deep = (eng.channels[t.table_id()] for t in (model.wide.embedding.sparse_table, model.deep.sparse_table))
        assert wide.lookups == 3 and deep.lookups == (3 if hook else 0)
        results.append((torch.stack(outs), rows(model.wide.embedding.sparse_table), rows(model.deep.sparse_table)))
        kk.stop()
    for a, b in zip(*results):
        # sums of a few dozen float32 values in another order, through a bf16 layer: one rounding of 2^-8 may differ
        assert torch.allclose(a, b, rtol=2e-2, atol=2e-2 * float(b.abs().max()))
