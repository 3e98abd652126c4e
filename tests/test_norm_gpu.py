"""Scaled norm and BiCGSTAB's fused updates at the edges of their tiles.

A partial of the norm is a power-of-two exponent and a sum of squares, so its
edges are the ends of the exponent range, subnormals, infinities and NaN, and
counts around a thread's 8 elements, a CTA's 2048 and the grid's cap.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Sums of squares of at most 100 additions in a row (8 a pass and thread, two
# warp trees, a strided share of 592 partials): 100 * 2^-53 on the sum, half
# of it on the root, and one rounding each of the square, root and product.
RELATIVE = 60 * 2.0 ** -53


def reference(a):
    top = float(np.abs(a).max(initial=0.0))
    if top == 0.0:
        return 0.0
    scale = 2.0 ** max(math.frexp(top)[1] - 1, -1000)
    return math.sqrt(math.fsum((a / scale) ** 2)) * scale


def vector(native, ctx, a):
    v = native.Vector(ctx, a.size, 0, 1)
    v.upload(a)
    return v


@pytest.mark.parametrize("n", [1, 7, 8, 255, 256, 257, 2047, 2048, 2049, 12288, 100003, 1212416, 1212417])
@pytest.mark.parametrize("exponent", [-1000, -300, 0, 300, 1000])
def test_norm_sizes_and_exponents(native, ctx, n, exponent):
    a = np.ldexp(np.random.default_rng(n).uniform(-1.0, 1.0, n), exponent)
    want = reference(a)
    assert abs(native.norm(vector(native, ctx, a)) - want) <= RELATIVE * want


@pytest.mark.parametrize("n", [1, 300, 5000])
def test_norm_range_ends(native, ctx, n):
    rng = np.random.default_rng(n)
    a = np.ldexp(rng.uniform(-1.0, 1.0, n), rng.integers(-500, 500, n))
    want = reference(a)
    assert abs(native.norm(vector(native, ctx, a)) - want) <= RELATIVE * want
    tiny = np.full(n, 5e-324)
    assert native.norm(vector(native, ctx, tiny)) == pytest.approx(math.sqrt(n) * 5e-324, abs=5e-324)
    big = np.zeros(n)
    big[n // 2] = np.finfo(np.float64).max
    assert native.norm(vector(native, ctx, big)) == np.finfo(np.float64).max
    big[n - 1] = -np.inf
    assert native.norm(vector(native, ctx, big)) == np.inf
    big[0] = np.nan
    assert np.isnan(native.norm(vector(native, ctx, big)))


@pytest.mark.parametrize("n", [1, 9, 255, 2049, 30011])
def test_bicgstab_fused_updates(native, ctx, n):
    """Diagonally dominant tridiagonal system: the true residual reaches the
    tolerance asked for, and the reported norms are those of the result."""
    rows, cols, values = [0], [], []
    for i in range(n):
        for j in (i - 1, i, i + 1):
            if 0 <= j < n:
                cols.append(j)
                values.append(4.0 if i == j else -1.0 - 0.1 * (j > i))
        rows.append(len(cols))
    rows, cols, values = np.array(rows), np.array(cols), np.array(values)
    b = np.random.default_rng(n).normal(size=n)
    matrix = native.Matrix(ctx, "bsr", n, 0, 1, rows, cols, values)
    pc = native.Preconditioner(matrix, native.PC_JACOBI, 0)
    vb, vx = vector(native, ctx, b), vector(native, ctx, np.zeros(n))
    r = native.solve(native.BICGSTAB, matrix, pc, vb, vx, native.default_options(relative_tolerance=1e-10),
                     native.Workspace(ctx))
    x = vx.download()
    ax = np.add.reduceat(values * x[cols], rows[:-1])
    true = np.linalg.norm(b - ax)
    assert r.status == 0
    assert true <= 1.01e-10 * np.linalg.norm(b)
    assert abs(r.true_residual_norm - true) <= 1e-13 * np.linalg.norm(b)
