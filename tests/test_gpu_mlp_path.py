"""Weight casts and fused gradients of the MLP path (csrc/cuda/model_kernels.cu, mlp_gemm.cu) (B200 only)."""
import pytest
import torch

from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"


# Matrix edges around the 64 x 64 tiles, more layers than one launch takes (8), widths and addresses that only the
# general kernel can read; the copies are roundings of the same floats, so they are equal bit for bit.
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("shapes", [[(8, 8)], [(64, 64), (72, 56), (400, 432)], [(128, 8), (8, 200)] * 5, [(10, 24), (16, 12)],
                                    [(4096, 784)]])
def test_cast_weights(shapes, transpose):
    torch.manual_seed(0)
    ws = [torch.randn(s, device=DEV) for s in shapes]
    if len(shapes) == 1:  # an address that is not on 16 bytes
        n, k = shapes[0]
        ws.append(torch.randn(n * k + 1, device=DEV)[1:].view(n, k))
    w16s, wt16s, buf = C.cast_weights(ws, transpose)
    assert len(w16s) == len(ws) and len(wt16s) == (len(ws) if transpose else 0) and buf is not None
    for k, w in enumerate(ws):
        assert torch.equal(w16s[k], w.to(torch.bfloat16))
        if transpose:
            assert torch.equal(wt16s[k], w.t().to(torch.bfloat16))


def test_scoring_between_training_steps_leaves_the_gradients_right():
    from kraken_b200.models import MLP
    torch.manual_seed(1)
    model = MLP(64, [128, 64, 1]).to(DEV)
    x = torch.randn(300, 64, device=DEV)
    model(x).sum().backward()
    want = [p.grad.clone() for p in model.parameters()]
    for p in model.parameters():
        p.grad = None
    with torch.no_grad():
        prepared = model.prepare()   # no transposes
        model(x, prepared=prepared)
    model(x, prepared=prepared).sum().backward()
    for p, w in zip(model.parameters(), want):
        # split sums added in another order
        assert torch.allclose(p.grad, w, rtol=1e-4, atol=1e-4 * float(w.abs().max()))


# Batches around the 64 rows of a stage and the stages of the ring, widths around the 128 columns of a tile and with
# several column tiles of dW; the bias gradient is added to what is there and is float32 sums of bf16 values.
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (63, 128, 64), (64, 136, 256), (65, 400, 432), (257, 120, 520), (1000, 256, 64),
                                   (40001, 400, 432)])
def test_wgrad_sums_the_bias_gradient(m, n, k):
    torch.manual_seed(m)
    dy = torch.randn(m, n, device=DEV).to(torch.bfloat16)
    x = torch.randn(m, k, device=DEV).to(torch.bfloat16)
    dw, db = torch.zeros(n, k, device=DEV), torch.full((n,), 3.0, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    C.linear_wgrad(dy, x, dw, status, db)
    want = dy.double().sum(0) + 3.0
    # float32 sums of m values of magnitude 1: at most m roundings of 2^-24 of the running sum's size, ~sqrt(m)
    assert float((db.double() - want).abs().max()) <= 1e-6 * (10 + m ** 0.5) * max(1.0, m ** 0.5 / 8)
    ref = torch.zeros_like(dw)
    C.linear_wgrad(dy, x, ref, status)
    assert torch.allclose(dw, ref, rtol=1e-4, atol=1e-4 * float(ref.abs().max()))
    assert int(status) == 0


# The bias gradient beside a kernel that floods the SMs' memory units with reductions, as the sparse backward does: reads
# of a stage that are held up must still be done before the stage is refilled.
def test_bias_gradient_is_right_beside_heavy_memory_traffic():
    torch.manual_seed(5)
    m, n, k = 65536, 400, 432
    dy = torch.randn(m, n, device=DEV).to(torch.bfloat16)
    x = torch.randn(m, k, device=DEV).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = dy.double().sum(0)
    rows = torch.randint(0, 400_000, (1_700_000,), device=DEV)
    grads, table = torch.randn(1_700_000, 16, device=DEV), torch.zeros(400_000, 16, device=DEV)
    dbs = [torch.zeros(n, device=DEV) for _ in range(20)]
    dw = torch.zeros(n, k, device=DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for db in dbs:
        with torch.cuda.stream(side):
            C.linear_wgrad(dy, x, dw, status, db)
        table.index_add_(0, rows, grads)
    torch.cuda.synchronize()
    for db in dbs:
        # 65536 float32 additions of values of magnitude 1 in blocks: sums of ~256, roundings of 2^-24 of them
        assert float((db.double() - want).abs().max()) < 2e-3


def test_inputs_of_unjoined_weight_gradients_are_not_given_away():
    """With the join deferred the weight gradients may still wait on their stream when the backward pass has returned: the
    memory of the activations they read must not go to the next allocation of the main stream."""
    from kraken_b200.models import MLP
    from kraken_b200.ops import mlp as fused
    torch.manual_seed(1)
    model = MLP(64, [128, 64, 1]).to(DEV)
    for p in model.parameters():
        p.grad = torch.zeros_like(p)
    rows = 1 << 16
    model(torch.randn(rows, 64, device=DEV).to(torch.bfloat16)).sum().backward()
    torch.cuda.synchronize()
    fused.set_deferred_join(True)
    try:
        x = torch.randn(rows, 64, device=DEV).to(torch.bfloat16)
        want = x.data_ptr()
        side = fused._side_stream(x.device)
        with torch.cuda.stream(side):
            torch.cuda._sleep(400_000_000)  # about 0.2 s
        model(x).sum().backward()
        del x
        held = [torch.empty(rows, 64, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
        assert not side.query() and want not in [h.data_ptr() for h in held]
        torch.cuda.current_stream().wait_stream(fused.take_pending_side_stream(held[0].device))
    finally:
        fused.set_deferred_join(False)
    torch.cuda.synchronize()


def test_weights_of_a_single_layer_can_be_prepared():
    """There is no hidden layer whose weights could be cast ahead: nothing is prepared, and nothing refused."""
    from kraken_b200.ops import mlp as fused
    torch.manual_seed(0)
    x, w, b = torch.randn(33, 64, device=DEV), torch.randn(10, 64, device=DEV), torch.randn(10, device=DEV)
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            prepared = fused.prepare_weights([w])
            assert list(prepared.w16s) == [] and list(prepared.wt16s) == []
            assert torch.equal(fused.fused_mlp(x, [w], [b], prepared=prepared), fused.fused_mlp(x, [w], [b]))


@pytest.mark.parametrize("M,sizes", [(200, (64, 48, 16)), (4096, (400, 400, 8)), (65536, (256, 128, 24)), (1024, (2048, 8))])
def test_biases_that_are_not_stored_back_to_back(M, sizes):
    """Each is copied in front of the kernel that adds it, and that kernel waits for the copy; through every plan of the
    forward pass, the head among the layers."""
    from kraken_b200.ops import mlp as fused
    torch.manual_seed(M)
    K = 432
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    ws = [torch.randn(n, k, device=DEV) / k ** 0.5 for n, k in zip(sizes, (K,) + sizes[:-1])]
    for _ in range(5):
        bs = [torch.randn(n, 3, device=DEV)[:, 1] for n in sizes]
        with torch.no_grad():
            want = fused.fused_mlp(x, ws, [b.clone(memory_format=torch.contiguous_format) for b in bs])
            assert torch.equal(fused.fused_mlp(x, ws, bs), want)
    ws, bs = [w.requires_grad_() for w in ws], [b.requires_grad_() for b in bs]
    fused.fused_mlp(x, ws, bs).sum().backward()
    fused.check_gemm_status(x.device)
    assert all(b.grad is not None and bool(b.grad.isfinite().all()) for b in bs)
