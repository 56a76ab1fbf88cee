"""Several buffers copied in one launch (B200 only)."""
import pytest
import torch

from kraken_b200._native import C

pytestmark = pytest.mark.gpu
DEV = "cuda"


# Sizes around a 16-byte piece, a block and the grid; buffers on any byte; more of them than one launch takes.
@pytest.mark.parametrize("sizes", [[1, 15], [16, 17, 31], [4095, 4096, 4097], [0, 5, 0], [1 << 20, 3, (1 << 22) + 1],
                                   list(range(1, 20)), [7]])
@pytest.mark.parametrize("at", [0, 1, 8])
def test_bytes(sizes, at):
    g = torch.Generator(device=DEV).manual_seed(len(sizes) + at)
    src = [torch.randint(0, 256, (n + at,), dtype=torch.uint8, device=DEV, generator=g)[at:] for n in sizes]
    room = [torch.zeros(n + 32, dtype=torch.uint8, device=DEV) for n in sizes]
    C.copy_batch([r[16:16 + n] for r, n in zip(room, sizes)], src)
    for r, s, n in zip(room, src, sizes):
        assert torch.equal(r[16:16 + n], s) and not bool(r[:16].any()) and not bool(r[16 + n:].any())


def test_what_is_not_a_plain_copy_is_copied_as_torch_does():
    src = [torch.arange(12, device=DEV).view(3, 4).t(), torch.arange(5), torch.ones(3, device=DEV, dtype=torch.float64),
           torch.full((1,), 2.0, device=DEV), torch.arange(6.0, device=DEV)]
    dst = [torch.zeros(4, 3, dtype=torch.int64, device=DEV), torch.zeros(5, dtype=torch.int64, device=DEV),
           torch.zeros(3, device=DEV), torch.zeros(4, device=DEV), torch.zeros(6, device=DEV)]
    C.copy_batch(dst, src)
    for d, s in zip(dst, src):
        assert torch.equal(d, torch.zeros_like(d).copy_(s))
    with pytest.raises(RuntimeError):
        C.copy_batch(dst, src[:-1])


def test_buffers_that_overlap_are_copied_in_the_order_they_are_named():
    """A step whose inputs are its own earlier inputs: what the first copies wrote is what the later ones read."""
    n = 1 << 22
    def buffers():
        return [torch.full((n,), float(k), device=DEV) for k in range(4)]
    pairs = [lambda a, b, c, d: ([b, c, d], [a, b, c]),             # every one gets the first one's values
             lambda a, b, c, d: ([d, c, b], [c, b, a]),             # shifted by one
             lambda a, b, c, d: ([a, b], [b, a]),
             lambda a, b, c, d: ([a, b, a], [b, c, d]),             # written twice
             lambda a, b, c, d: ([a[n // 2:], b[:n // 2 + 5]], [c[n // 2:], a[n // 2 - 5:]]),
             lambda a, b, c, d: ([a[1:n // 2], c], [b[1:n // 2], a]),
             lambda a, b, c, d: ([a, b, c], [a, b, d])]             # onto itself
    for make in pairs:
        for _ in range(5):
            got, want = buffers(), buffers()
            C.copy_batch(*make(*got))
            for t, s in zip(*make(*want)):
                t.copy_(s)
            assert all(torch.equal(x, y) for x, y in zip(got, want))
    a = torch.arange(64.0, device=DEV)
    for t, s in ((a[:48], a[16:]), (a[16:], a[:48])):
        with pytest.raises(RuntimeError):   # as copy_ itself: a part of what is read is written
            C.copy_batch([t, torch.empty(3, device=DEV)], [s, torch.ones(3, device=DEV)])


@pytest.mark.parametrize("at", [1, 2, 3])
def test_floats_off_a_16_byte_boundary_are_not_copied_by_bytes(at):
    """A batch sliced out of a larger tensor starts on any float.  By single bytes it took eight times as long as one on
    16 bytes, 400 us for 49; a factor of four is left to whatever else the machine does."""
    n = 1 << 24
    src, dst = torch.randn(n + 4, device=DEV), [torch.empty(n, device=DEV) for _ in range(2)]

    def took(s):
        best = float("inf")
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            C.copy_batch(dst, [s, s])
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert took(src[at:at + n]) <= 4 * took(src[:n])
    C.copy_batch(dst, [src[at:at + n], src[:n]])
    assert torch.equal(dst[0], src[at:at + n]) and torch.equal(dst[1], src[:n])


# Pieces of 4, 8 and 16 bytes side by side in one launch, whole and with a rest; nothing around the buffers is written.
@pytest.mark.parametrize("n", [1, 2, 3, 5, 255, 1025, 70001])
def test_buffers_on_any_word(n):
    src = torch.randint(0, 256, (7, 4 * n + 64), dtype=torch.uint8, device=DEV)
    parts = [(0, 0, 4 * n), (4, 0, 4 * n), (8, 8, 4 * n + 3), (4, 12, 4 * n + 1), (0, 16, 4 * n), (12, 4, 4 * n), (8, 0, 4 * n + 2)]
    room = torch.zeros_like(src)
    want = room.clone()
    for k, (a, b, m) in enumerate(parts):
        want[k, b:b + m] = src[k, a:a + m]
    C.copy_batch([room[k, b:b + m] for k, (_, b, m) in enumerate(parts)], [src[k, a:a + m] for k, (a, _, m) in enumerate(parts)])
    assert torch.equal(room, want)
