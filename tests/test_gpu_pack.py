"""The kernels between the sparse exchange and the MLP, forward and backward, against float64 (B200 only)."""
import pytest
import torch

from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 500

# Fields around a lane's one and two of a sample's 16 or 32 lanes and around a batch of rows; every row width.
SIZES = [(3, 1, 4), (70, 15, 4), (33, 33, 4), (5, 17, 8), (40, 26, 16), (1, 27, 16), (9, 29, 16), (64, 65, 16), (7, 31, 32),
         (19, 33, 64), (3, 65, 128), (20011, 26, 16)]


def problem(B, F, D, folded, slots):
    torch.manual_seed(B + F + D)
    RD = D + 4 if folded else D
    inv = (U * torch.rand(B, F, device=DEV) ** 4).int().clamp_(max=U - 1)  # skewed
    inv1 = torch.randint(0, U, (B, F), device=DEV, dtype=torch.int32)
    rows, first = torch.randn(U, RD, device=DEV), torch.randn(U, 1, device=DEV)
    at, at1 = inv.long(), inv1.long()
    slots2 = slots1 = None
    if slots:
        slots2, slots1 = (torch.randperm(U, device=DEV).int() for _ in range(2))
        at, at1 = slots2.long()[at], slots1.long()[at1]
    w = rows[at, D] if folded else first[at1, 0]
    return inv, inv1, rows, first, slots2, slots1, rows[at, :D].double(), w.double()


@pytest.mark.parametrize("B,F,D", SIZES)
@pytest.mark.parametrize("folded,fm,slots", [(True, True, False), (False, True, True), (False, False, True), (True, True, True)])
def test_forward(B, F, D, folded, fm, slots):
    inv, inv1, rows, first, slots2, slots1, e, w = problem(B, F, D, folded, slots)
    nd = 13
    ldx = (F * D + nd + 15) // 16 * 16
    dense = torch.randn(B, nd, device=DEV)
    x = torch.full((B, ldx), 7.0, device=DEV, dtype=torch.bfloat16)
    logit, ssum = torch.empty(B, device=DEV), torch.empty(B, D, device=DEV)
    C.deepfm_pack_forward(rows, inv, None if folded else first, None if folded else inv1, dense, B, F, D, x, logit, slots2,
                          None if folded else slots1, ssum if fm else None, fm)
    want = torch.zeros(B, ldx, device=DEV, dtype=torch.float64)
    want[:, : F * D], want[:, F * D: F * D + nd] = e.view(B, F * D), dense.double()
    assert torch.equal(x, want.float().to(torch.bfloat16))  # rounded once
    value, size = w.sum(1), w.abs().sum(1)
    if fm:
        s, q, sabs = e.sum(1), (e * e).sum(1), e.abs().sum(1)
        # a float32 sum of F terms is off by F x 2^-24 of the sum of magnitudes at most
        assert bool(((ssum.double() - s).abs() <= F * 2 ** -24 * sabs).all())
        value, size = value + 0.5 * (s * s - q).sum(1), size + (sabs * sabs).sum(1) + q.sum(1)
    assert bool(((logit.double() - value).abs() <= (F + D + 8) * 2 ** -24 * size).all())


@pytest.mark.parametrize("B,F,D", SIZES)
@pytest.mark.parametrize("folded,fm,with_dx,slots", [(True, True, True, False), (False, True, False, True),
                                                     (False, False, True, True), (True, True, True, True)])
def test_backward(B, F, D, folded, fm, with_dx, slots):
    inv, inv1, rows, _, slots2, _, e, _ = problem(B, F, D, folded, slots)
    dlogit = torch.randn(B, device=DEV)
    dx = torch.randn(B, F * D + 4, device=DEV).to(torch.bfloat16) if with_dx else None
    ssum = torch.randn(B, D, device=DEV) if fm else None
    grad2, grad1 = torch.zeros(U, rows.size(1), device=DEV), None if folded else torch.zeros(U, 1, device=DEV)
    C.deepfm_pack_backward(rows, inv, None if folded else inv1, dx, dlogit, B, F, D, grad2, grad1, slots2, ssum)
    n, at = B * F, inv.long().view(-1)
    terms = torch.zeros(B, F, D, device=DEV, dtype=torch.float64)
    size = terms.clone()
    if with_dx:
        g = dx[:, : F * D].double().view(B, F, D)
        terms, size = terms + g, size + g.abs()
    if fm:
        g, s = dlogit.double().view(B, 1, 1), ssum.double().unsqueeze(1)
        terms, size = terms + g * (s - e), size + 2 * g.abs() * (s.abs() + e.abs())

    def close(got, at, terms, size):
        """float32 sums of ``counts`` terms in any order: their rounding errors, at most 2^-24 of the sum of magnitudes
        each, add up like a random walk; a term has three of its own."""
        zeros = torch.zeros(U, terms.size(1), device=DEV, dtype=torch.float64)
        counts = torch.bincount(at, minlength=U).double().unsqueeze(1)
        bound = 2 ** -23 * (2 * counts.sqrt() + 4) * zeros.index_add(0, at, size)
        assert bool(((got.double() - zeros.index_add(0, at, terms)).abs() <= bound).all())

    close(grad2[:, :D], at, terms.view(n, D), size.view(n, D))
    first = dlogit.double().view(B, 1).expand(B, F).reshape(n, 1)
    close(grad2[:, D: D + 1] if folded else grad1, at if folded else inv1.long().view(-1), first, first.abs())
    if folded:
        assert bool((grad2[:, D + 1:] == 0).all())


# What Wide&Deep (fm False) and two-table DeepFM take with more ids than are read in place: gathered rows of two tables; and
# rows that lie further apart than they are wide, the first-order ones as well.
@pytest.mark.parametrize("B,F,D", [(33, 33, 4), (40, 26, 16), (9, 29, 16), (7, 31, 32), (19, 33, 64), (3, 65, 128)])
@pytest.mark.parametrize("fm", [False, True])
@pytest.mark.parametrize("slots,pitch", [(False, 0), (False, 8), (True, 12)])
def test_two_tables(B, F, D, fm, slots, pitch):
    inv, inv1, rows, first, slots2, slots1, e, w = problem(B, F, D, False, slots)
    if pitch:
        wide, narrow = torch.full((U, D + pitch), float("nan"), device=DEV), torch.full((U, pitch), float("nan"), device=DEV)
        wide[:, :D], narrow[:, :1] = rows, first
        rows, first = wide[:, :D], narrow[:, :1]
    ldx = (F * D + 13 + 7) // 8 * 8
    dense = torch.randn(B, 13, device=DEV)
    x = torch.full((B, ldx), 7.0, device=DEV, dtype=torch.bfloat16)
    logit, ssum = torch.empty(B, device=DEV), torch.empty(B, D, device=DEV)
    C.deepfm_pack_forward(rows, inv, first, inv1, dense, B, F, D, x, logit, slots2, slots1, ssum if fm else None, fm)
    want = torch.zeros(B, ldx, device=DEV, dtype=torch.float64)
    want[:, : F * D], want[:, F * D: F * D + 13] = e.view(B, F * D), dense.double()
    assert torch.equal(x, want.float().to(torch.bfloat16))
    value, size = w.sum(1), w.abs().sum(1)
    if fm:
        s, q, sabs = e.sum(1), (e * e).sum(1), e.abs().sum(1)
        value, size = value + 0.5 * (s * s - q).sum(1), size + (sabs * sabs).sum(1) + q.sum(1)
    assert bool(((logit.double() - value).abs() <= (F + D + 8) * 2 ** -24 * size).all())   # as above

    dx, dlogit = torch.randn(B, F * D + 4, device=DEV).to(torch.bfloat16), torch.randn(B, device=DEV)
    grad2, grad1 = torch.zeros(U, D, device=DEV), torch.zeros(U, 1, device=DEV)
    C.deepfm_pack_backward(rows, inv, inv1, dx, dlogit, B, F, D, grad2, grad1, slots2, ssum if fm else None)
    terms = dx[:, : F * D].double().view(B, F, D)
    size = terms.abs()
    if fm:
        g, s = dlogit.double().view(B, 1, 1), ssum.double().unsqueeze(1)
        terms, size = terms + g * (s - e), size + 2 * g.abs() * (s.abs() + e.abs())
    once = dlogit.double().view(B, 1, 1).expand(B, F, 1)
    for got, at, terms, size in ((grad2, inv, terms, size), (grad1, inv1, once, once.abs())):
        at, zeros = at.long().view(-1), torch.zeros(U, terms.size(2), device=DEV, dtype=torch.float64)
        counts = torch.bincount(at, minlength=U).double().unsqueeze(1)
        bound = 2 ** -23 * (2 * counts.sqrt() + 4) * zeros.index_add(0, at, size.reshape(B * F, -1))   # as above
        assert bool(((got.double() - zeros.index_add(0, at, terms.reshape(B * F, -1))).abs() <= bound).all())
