"""Head kernels of the MLP - a single output and a few outputs - against float64 (B200 only)."""
import pytest
import torch

from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"


def close(got, want, terms):
    """float32 sums of ``terms`` products in any order: each rounding is at most 2^-24 of the sum of magnitudes, of which
    ``want``'s second part is the bound."""
    value, magnitude = want
    assert bool(((got.double() - value).abs() <= 2 ** -23 * (terms ** 0.5 + 4) * magnitude + 1e-30).all())


# Rows around a block's eight warps, a row each; columns around the 64 that a warp takes at a time.
@pytest.mark.parametrize("M", [1, 3, 4, 5, 33, 1000])
@pytest.mark.parametrize("K", [8, 248, 256, 264, 400])
def test_single_output_forward(M, K):
    torch.manual_seed(M + K)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w, b, add = torch.randn(K, device=DEV), torch.randn(1, device=DEV), torch.randn(M, device=DEV)
    y = torch.empty(M, device=DEV)
    C.rowdot_forward(x, w, b, y, add)
    p = x.double() * w.double()
    close(y, (p.sum(1) + b.double() + add.double(), p.abs().sum(1) + b.double().abs() + add.double().abs()), K + 2)


# Classes on both sides of every compile-time bound, rows around a block's four (forward) and 32 (backward), columns around
# a thread's and a block's.
@pytest.mark.parametrize("classes", [1, 4, 5, 8, 10, 12, 13, 16])
@pytest.mark.parametrize("M,K", [(1, 8), (3, 504), (4, 512), (33, 520), (31, 2056), (200, 4096)])
@pytest.mark.parametrize("relu", [False, True])
def test_few_outputs(classes, M, K, relu):
    torch.manual_seed(classes + M + K)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w, b = torch.randn(classes, K, device=DEV), torch.randn(classes, device=DEV)
    g = torch.randn(M, classes, device=DEV)
    assert C.head_supported(x, w, torch.empty_like(w))
    y = torch.empty(M, classes, device=DEV)
    C.head_forward(x, w, b, y)
    xd, wd, gd = x.double(), w.double(), g.double()
    close(y, (xd @ wd.t() + b.double(), xd.abs() @ wd.abs().t() + b.double().abs()), K + 1)
    dw, db = torch.ones_like(w), torch.ones_like(b)
    dx = torch.empty_like(x)
    C.head_backward(x, w, g, relu, dx, dw, db)
    close(dw, (1 + gd.t() @ xd, 1 + gd.abs().t() @ xd.abs()), M + 1)
    close(db, (1 + gd.sum(0), 1 + gd.abs().sum(0)), M + 1)
    want = gd @ wd
    if relu:
        want = want * (xd > 0)
        assert bool((dx[x <= 0] == 0).all())
    # one rounding to bfloat16's 8 significant bits, on top of the sum of up to 16 products
    assert bool(((dx.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -20 * (gd.abs() @ wd.abs())).all())
    kept = dw.clone()
    C.head_backward(x, w, g, relu, None, dw, db)   # no input gradient wanted; the others are added to
    close(dw, (kept.double() + gd.t() @ xd, kept.double().abs() + gd.abs().t() @ xd.abs()), M + 1)


def test_operands_the_kernels_do_not_take():
    x = torch.zeros(4, 16, dtype=torch.bfloat16, device=DEV)
    w = torch.zeros(10, 16, device=DEV)
    assert C.head_supported(x, w)
    assert not C.head_supported(x, torch.zeros(17, 16, device=DEV))                # more classes than the sums have registers
    assert not C.head_supported(x[:, 1:9], torch.zeros(10, 8, device=DEV))         # rows off a 16-byte boundary
    assert not C.head_supported(x, torch.zeros(161, device=DEV)[1:].view(10, 16))  # weights off a 16-byte boundary
    assert not C.head_supported(x, w, torch.zeros(16, 10, device=DEV).t())         # gradient buffer with another stride


def test_more_rows_than_a_grid_is_high():
    """65535 blocks of rows and one more, in the direction of a grid that ends there."""
    M, K, classes = 65535 * 32 + 7, 8, 3
    torch.manual_seed(0)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w, b, g = torch.randn(classes, K, device=DEV), torch.randn(classes, device=DEV), torch.randn(M, classes, device=DEV)
    y, dx, dw, db = torch.empty(M, classes, device=DEV), torch.empty_like(x), torch.zeros_like(w), torch.zeros_like(b)
    C.head_forward(x, w, b, y)
    C.head_backward(x, w, g, False, dx, dw, db)
    xd, wd, gd = x.double(), w.double(), g.double()
    close(y, (xd @ wd.t() + b.double(), xd.abs() @ wd.abs().t() + b.double().abs()), K + 1)
    close(dw, (gd.t() @ xd, gd.abs().t() @ xd.abs()), M)
    close(db, (gd.sum(0), gd.abs().sum(0)), M)
    want = gd @ wd
    assert bool(((dx.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -20 * (gd.abs() @ wd.abs())).all())


# Blocks of one and of several row ranges, with a remainder; one range alone.
@pytest.mark.parametrize("M,K,classes", [(20, 256, 10), (1000, 4096, 10), (40_003, 256, 3), (777, 520, 16)])
def test_backward_repeats_bit_for_bit(M, K, classes):
    torch.manual_seed(M)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w, g = torch.randn(classes, K, device=DEV), torch.randn(M, classes, device=DEV)
    outs = []
    for _ in range(10):
        dx, dw, db = torch.empty_like(x), torch.ones_like(w), torch.ones(classes, device=DEV)
        C.head_backward(x, w, g, True, dx, dw, db)
        outs.append((dx, dw, db))
    for o in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(o, outs[0]))
