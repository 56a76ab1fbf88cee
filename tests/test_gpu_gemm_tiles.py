"""Tiles, rings and epilogues of the tcgen05 GEMMs against float64, at the edges of each variant (B200 only)."""
import pytest
import torch

from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"

# Rows, columns and contraction around 256 and 128 (rows of a pair and of a CTA), 32 (columns of an output box), 64 (a k-block),
# fewer k-blocks than stages and more, grids of less and more than one wave.
SHAPES = [(1, 8, 8), (63, 64, 72), (128, 128, 64), (129, 136, 56), (257, 264, 520), (255, 1032, 200), (1000, 208, 72),
          (1024, 4096, 784), (300, 4096, 1032), (5000, 400, 432), (19000, 400, 432), (20001, 72, 264)]


def rnd(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


def check(got, want, magnitude, terms, rounding):
    """Sums of ``terms`` float32 products in any order, and one rounding of the result."""
    bound = (terms ** 0.5 + 8) * 2 ** -23 * magnitude + rounding * want.abs() + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("relu", [False, True])
def test_forward(M, N, K, relu):
    torch.manual_seed(M + N + K)
    x, w, b = rnd(M, K), rnd(N, K, scale=0.1), torch.randn(N, device=DEV)
    y = torch.full((M + 1, (N + 7) // 8 * 8 + 8), 7.0, device=DEV, dtype=torch.bfloat16)   # what is around the output stays
    mask = torch.zeros(((N + 15) // 16, (M + 63) // 64 * 64), device=DEV, dtype=torch.int16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    C.linear_forward(x, w, b, relu, y[:M, :N], status, mask if relu else None)
    want = x.double() @ w.double().t() + b.double()
    check(y[:M, :N], want.relu() if relu else want, x.double().abs() @ w.double().abs().t() + b.double().abs(), K + 1, 2 ** -8)
    assert bool((y[M:] == 7).all()) and bool((y[:, N:] == 7).all())
    if relu:
        bits = (mask[:, :M].t().to(torch.int32) & 0xFFFF).unsqueeze(-1) >> torch.arange(16, device=DEV)
        bits = (bits & 1).reshape(M, -1).bool()
        # (a positive result can round to the smallest bfloat16 only from far below it: no case here)
        assert torch.equal(bits[:, :N], y[:M, :N].float() > 0) and not bool(bits[:, N:].any())
    assert status.item() == 0


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("masked", ["no", "bits", "activations"])
def test_input_gradient(M, N, K, masked):
    torch.manual_seed(M + N + K)
    dy, w, h = rnd(M, N), rnd(N, K, scale=0.1), rnd(M, K).relu()
    dx = torch.full((M + 1, K + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    mask = None
    if masked == "bits":
        on = torch.nn.functional.pad(h > 0, (0, -K % 16)).view(M, -1, 16).to(torch.int32)
        words = (on << torch.arange(16, device=DEV, dtype=torch.int32)).sum(-1)
        mask = torch.zeros(((K + 15) // 16, (M + 63) // 64 * 64), device=DEV, dtype=torch.int16)
        mask[:, :M] = torch.where(words >= 32768, words - 65536, words).to(torch.int16).t()
    C.linear_dgrad(dy, w.t().contiguous(), h if masked == "activations" else None, dx[:M, :K], status, mask)
    want = dy.double() @ w.double()
    if masked != "no":
        want = want * (h > 0)
    check(dx[:M, :K], want, dy.double().abs() @ w.double().abs(), N, 2 ** -8)
    assert bool((dx[M:] == 7).all()) and bool((dx[:, K:] == 7).all())
    assert status.item() == 0


# variant 4: on pairs of CTAs whatever the size; 0: by the rule, among them sizes on both sides of it
@pytest.mark.parametrize("M,N,K", SHAPES + [(20000, 400, 432), (4096, 640, 1032), (33000, 264, 264), (520, 4096, 4096)])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("variant", [0, 4])
def test_weight_gradient(M, N, K, bias, variant):
    torch.manual_seed(M + N + K)
    dy, x = rnd(M, N, scale=0.1), rnd(M, K)
    dw = torch.ones(N + 1, K + 4, device=DEV)
    db = torch.ones(N + 1, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    C.gemm_set_tuning(variant, 0)
    try:
        for _ in range(2):  # it adds
            C.linear_wgrad(dy, x, dw[:N, :K], status, db[:N] if bias else None)
    finally:
        C.gemm_set_tuning(0, 0)
    d, xd = dy.double(), x.double()
    # a sum of up to M products and of the splits' partial sums, twice
    check(dw[:N, :K], 1 + 2 * (d.t() @ xd), 1 + 2 * (d.abs().t() @ xd.abs()), M + 200, 0)
    check(db[:N], 1 + 2 * d.sum(0) if bias else torch.ones(N, device=DEV).double(), 1 + 2 * d.abs().sum(0), M + 200, 0)
    assert bool((dw[N:] == 1).all()) and bool((dw[:, K:] == 1).all()) and db[N].item() == 1
    assert status.item() == 0


@pytest.mark.parametrize("M", [1, 70, 4096, 40001])   # one tile per CTA, and the persistent kernel
def test_columns_without_a_gradient_are_cleared(M):
    torch.manual_seed(M)
    dy, w = rnd(M, 400), rnd(400, 416, scale=0.1)
    dx = torch.full((M + 1, 440), 7.0, device=DEV, dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    C.linear_dgrad(dy, w.t().contiguous(), None, dx[:M, :416], status, None, 16)
    check(dx[:M, :416], dy.double() @ w.double(), dy.double().abs() @ w.double().abs(), 400, 2 ** -8)
    assert bool((dx[:M, 416:432] == 0).all()) and bool((dx[:M, 432:] == 7).all()) and bool((dx[M] == 7).all())
    assert status.item() == 0
