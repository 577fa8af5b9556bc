"""Products at the ends of the lazy value ranges: every length around the
one-row / four-step border and the two-stream schedule, inputs of the largest
and smallest residues and of unreduced words, outputs aliasing operands."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_helpers import dev

pytestmark = pytest.mark.gpu
P = O.P


def operand(kind, n, seed):
    if kind == "top":
        return np.full(n, P - 1, np.uint64)
    if kind == "wrap":                       # unreduced: 2^64 - 1 - small
        return np.uint64(2**64 - 1) - np.arange(n, dtype=np.uint64) % np.uint64(7)
    if kind == "step":                       # 0 and p - 1 in blocks, half-p edges
        v = np.where(np.arange(n) & 8, P - 1, 0).astype(np.uint64)
        v[::5] = P // 2
        v[::7] = P // 2 + 1
        return v
    return np.random.default_rng(seed).integers(0, 2**64 - 1, n, dtype=np.uint64)


@pytest.mark.parametrize("lg,batch", [(1, 5), (2, 3), (3, 3), (4, 9), (5, 17), (6, 65), (8, 7),
                                      (11, 3), (12, 3), (13, 1), (13, 33), (14, 3), (15, 2),
                                      (17, 2)])
@pytest.mark.parametrize("lhs,rhs", [("top", "top"), ("wrap", "step"), ("step", "any"),
                                     ("any", "wrap")])
def test_product_ranges(pcg, lg, batch, lhs, rhs):
    n = batch << lg
    a, b = operand(lhs, n, 1000 + lg), operand(rhs, n, 2000 + lg)
    want = O.poly_mul(a, b, 1 << lg)
    d_a, d_b, d_c = dev(pcg, a), dev(pcg, b), dev(pcg, np.zeros(n, np.uint64))
    pcg.poly_mul_device(d_c.ptr, d_a.ptr, d_b.ptr, batch, 1 << lg)
    assert (d_c.download(np.uint64, n) == want).all()
    pcg.poly_mul_device(d_a.ptr, d_a.ptr, d_b.ptr, batch, 1 << lg)      # c = a
    assert (d_a.download(np.uint64, n) == want).all()
    d_a = dev(pcg, a)
    pcg.poly_mul_device(d_b.ptr, d_a.ptr, d_b.ptr, batch, 1 << lg)      # c = b
    assert (d_b.download(np.uint64, n) == want).all()


def test_square_in_place(pcg):
    """a, b and c the same buffer, in both plan forms."""
    for lg in (7, 13):
        a = operand("any", 1 << lg, lg)
        d = dev(pcg, a)
        pcg.poly_mul_device(d.ptr, d.ptr, d.ptr, 1, 1 << lg)
        assert (d.download(np.uint64, 1 << lg) == O.poly_mul(a, a, 1 << lg)).all()


# One row (2^1 .. 2^9, ragged rows per CTA), the shortest and longest four-step
# rows, odd and even logN; words at the extremes of 64 bits.
@pytest.mark.parametrize("logN", [1, 3, 4, 5, 9, 10, 11, 13, 16, 19, 22, 24])
def test_ole_check_counts_slots(pcg, logN):
    """0 for a product; N / 2 with X^(N/2) - I added (I^2 = -1: it vanishes in
    every other slot); N with a constant added."""
    N = 1 << logN
    rng = np.random.default_rng(logN)
    x0 = rng.integers(0, 2**64 - 1, N, dtype=np.uint64, endpoint=True)
    x1 = rng.integers(0, 2**64 - 1, N, dtype=np.uint64, endpoint=True)
    z1 = rng.integers(0, P, N, dtype=np.uint64)
    x0[0] = x1[-1] = np.uint64(2**64 - 1)
    d0, d1, dz1 = (pcg.to_device(a) for a in (x0, x1, z1))
    prod, bad = pcg.DeviceBuffer(8 * N), pcg.DeviceBuffer(8)
    pcg.poly_mul_device(prod.ptr, d0.ptr, d1.ptr, 1, N)
    pcg.synchronize()
    z0 = (prod.download(np.uint64, N) + np.uint64(P) - z1) % np.uint64(P)
    I = pow(3, (P - 1) // 4, P)
    half, full = z0.copy(), z0.copy()
    half[N // 2] = (int(half[N // 2]) + 1) % P
    half[0] = (int(half[0]) - I) % P
    full[0] = (int(full[0]) + 7) % P
    for z, want in ((z0, 0), (half, N // 2), (full, N)):
        dz = pcg.to_device(z)
        pcg.verify_ole_device(N, d0.ptr, dz.ptr, d1.ptr, dz1.ptr, bad.ptr)
        pcg.synchronize()
        assert int(bad.download(np.uint64, 1)[0]) == want


# Batches on both sides of the column tile widths' steps (16, 8, 4 columns).
@pytest.mark.parametrize("batch,logN", [(9, 13), (10, 13), (64, 13), (296, 13), (3, 14), (37, 14),
                                        (5, 16), (2, 18), (1, 19), (2, 19)])
def test_column_tile_widths(pcg, batch, logN):
    N = 1 << logN
    rng = np.random.default_rng(batch * 100 + logN)
    a, b = (rng.integers(0, P, batch * N, dtype=np.uint64) for _ in range(2))
    da, db = pcg.to_device(a), pcg.to_device(b)
    c, one = pcg.DeviceBuffer(8 * batch * N), pcg.DeviceBuffer(8 * batch * N)
    pcg.poly_mul_device(c.ptr, da.ptr, db.ptr, batch, N)
    for k in range(batch):
        o = 8 * k * N
        pcg.poly_mul_device(one.ptr + o, da.ptr + o, db.ptr + o, 1, N)
    pcg.synchronize()
    got = c.download(np.uint64, batch * N)
    assert (got == one.download(np.uint64, batch * N)).all()
    assert (got[-N:] == O.poly_mul(a[-N:], b[-N:], N)).all()
