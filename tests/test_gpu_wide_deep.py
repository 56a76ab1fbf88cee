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
