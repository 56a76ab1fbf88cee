"""The learning rate that the kernels read follows the schedule, whatever was captured or enqueued before (B200 only)."""
import pytest
import torch

import kraken_b200.pytorch as kk
from kraken_b200.pytorch.lr import StepLR
from kraken_b200.utils.graph import GraphedStep

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 0.5 is a float32, 0.05 is not: a rate that is kept as one need not compare equal to the other.
@pytest.mark.parametrize("rate", [0.5, 0.05])
@pytest.mark.parametrize("replayed", [None, 0, 1])
def test_a_rate_that_changed_during_a_capture_reaches_what_follows(rate, replayed):
    """Two warm-up steps, then two captures, of which the first crosses a boundary of the schedule; nothing of it is
    replayed before the steps that follow, or one of the two graphs is."""
    kk.initialize("gpu", table_capacity=1 << 10, seed=2)
    emb = kk.Embedding(4, initializer=kk.ConstantInitializer(0.0), name="e")
    opt = kk.Optimizer("m", emb.named_parameters(), StepLR(rate, step_size=3, gamma=0.25), kk.SGD())
    eng = kk.native.engine()

    def train(ids):
        loss = emb(ids).sum()   # gradient 1 for every occurrence
        loss.backward()
        opt.step()
        return loss.detach()

    ids = torch.arange(8, device=DEV)
    step = GraphedStep(train, (ids,), warmup=2, slots=2, optimizer=opt)
    if replayed is None:
        train(ids)
    else:
        step.replay(replayed)
    assert eng.lr == pytest.approx(rate * 0.25) and float(eng.lr_dev) == pytest.approx(eng.lr)
    table = eng.sparse[emb.sparse_table.table_id()]
    before = table.lookup(ids)[0].clone()
    train(ids)
    assert torch.allclose(before - table.lookup(ids)[0], torch.full_like(before, rate * 0.25), rtol=1e-4)


def test_a_step_has_its_own_rate_when_the_host_runs_ahead():
    kk.initialize("gpu", table_capacity=1 << 10, seed=2)
    eng = kk.native.engine()
    kk.update_lr(1.0)
    seen = []
    torch.cuda._sleep(200_000_000)   # a tenth of a second in which the host enqueues everything below
    for k in range(20):
        kk.update_lr(0.1 * 0.9 ** k)
        seen.append(eng.lr_dev.clone())   # what a kernel enqueued here reads
    assert [float(s) for s in seen] == pytest.approx([0.1 * 0.9 ** k for k in range(20)])
