"""ILU and SSOR applies with one CTA per component (the default while the
levels are narrow), bit for bit against the oracle, which they equal term by
term; FP32 and stored-precision factors against the level-scheduled sweep
(OWTK_LOCAL_SWEEP=0), the same arithmetic.  Sizes at the edges of tasks (32
rows), steps (1, 2 and 4 tasks) and the result ring, rows longer than a task
holds in registers, dependencies beyond the ring, non-finite inputs."""
import numpy as np
import pytest

import cases
from conftest import assert_bitwise

pytestmark = pytest.mark.gpu


def _lattice(problems, nx, ny, bs, seed, order="natural"):
    rng = np.random.default_rng(seed)
    xy, edges = problems.lattice(nx, ny, 0.2, rng)
    s = problems.component_diagonal_system(xy, edges, bs, rng, order=order)
    return s.owned, s.rowptr, s.cols, s.vals


def _rows_system(n, bs, seed, neighbours):
    """Diagonally dominant rows: row r couples to the columns neighbours(r, rng) < r, symmetrically."""
    rng = np.random.default_rng(seed)
    pairs = {(r, int(c)) for r in range(n) for c in neighbours(r, rng) if 0 <= c < r}
    rows = np.array([p for a, b in pairs for p in (a, b)] + list(range(n)))
    cols = np.array([p for a, b in pairs for p in (b, a)] + list(range(n)))
    o = np.lexsort((cols, rows))
    rows, cols = rows[o], cols[o]
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    v = -rng.uniform(0.05, 1.0, size=(cols.size, bs))
    off = np.zeros((n, bs))
    np.add.at(off, rows[rows != cols], np.abs(v[rows != cols]))
    v[rows == cols] = 1.1 * off[rows[rows == cols]] + 0.5
    return n, rp, cols, v.reshape(-1)


def _check_ilu(native, ctx, restatement, n, bs, rp, ci, v, seed=0, x=None):
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
    p = native.Preconditioner(m, native.PC_ILU, 0)
    x = np.random.default_rng(seed).uniform(-1, 1, n * bs) if x is None else x
    xv, y = native.Vector(ctx, n, 0, bs).upload(x), native.Vector(ctx, n, 0, bs)
    want = restatement.ilu(n, bs, rp, ci, v, 0).apply(x)
    p.apply(xv, y)
    assert_bitwise(y.download(), want, "ILU(0)")
    p.apply(xv, xv)
    assert_bitwise(xv.download(), want, "ILU(0) in place")


# Levels of a lattice in natural order hold up to min(nx, ny) rows: one task,
# two, four, and more than a step of four.
@pytest.mark.parametrize("nx,ny,bs", [(1, 1, 3), (2, 1, 1), (31, 40, 2), (32, 33, 1), (33, 70, 3), (64, 65, 1),
                                      (65, 66, 4), (128, 130, 3), (129, 140, 1), (260, 150, 2), (3, 500, 33)])
def test_ilu_widths(native, ctx, restatement, problems, nx, ny, bs):
    if nx * ny < 4:
        n, rp, ci, v = _rows_system(nx * ny, bs, 1, lambda r, g: [r - 1])
    else:
        n, rp, ci, v = _lattice(problems, nx, ny, bs, nx + ny)
    _check_ilu(native, ctx, restatement, n, bs, rp, ci, v)


@pytest.mark.parametrize("far", [2, 40])
def test_ilu_dependencies_beyond_the_ring(native, ctx, restatement, far):
    # A chain of levels of 40 rows; every 300th row couples to rows near the
    # start, more than the ring's 12,000 rows back.  40 of them exceed what a
    # task stages and what its registers hold.
    def neighbours(r, rng):
        near = [r - 40, r - 41]
        return near + (rng.integers(0, 200, size=far).tolist() if r > 16000 and r % 300 == 0 else [])
    _check_ilu(native, ctx, restatement, *(lambda t: (t[0], 2, t[1], t[2], t[3]))(_rows_system(20000, 2, 5, neighbours)))


@pytest.mark.parametrize("width", [7, 8, 9, 17])
def test_ilu_long_rows(native, ctx, restatement, width):
    # One row in 150 is `width` entries long (eight fit in registers).
    n, rp, ci, v = _rows_system(3000, 1, width, lambda r, g: list(range(r - 30, r - 30 - (width if r % 150 == 0 else 2), -1)))
    _check_ilu(native, ctx, restatement, n, 1, rp, ci, v)


def test_ilu_non_finite(native, ctx, restatement, problems):
    n, rp, ci, v = _lattice(problems, 40, 40, 2, 3)
    x = np.random.default_rng(1).uniform(-1, 1, n * 2)
    x[37], x[1000], x[2000], x[5] = np.inf, -np.inf, -0.0, np.nan
    m = native.Matrix(ctx, "bsr", n, 0, 2, rp, ci, v)
    p = native.Preconditioner(m, native.PC_ILU, 0)
    y = native.Vector(ctx, n, 0, 2)
    p.apply(native.Vector(ctx, n, 0, 2).upload(x), y)
    want, got = restatement.ilu(n, 2, rp, ci, v, 0).apply(x), y.download()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert_bitwise(got[ok], want[ok], "ILU(0), non-finite input")


def test_ilu_update_values(native, ctx, restatement, problems):
    n, rp, ci, v = _lattice(problems, 70, 50, 3, 8, "rcm")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v)
    p = native.Preconditioner(m, native.PC_ILU, 0)
    v2 = v * np.random.default_rng(9).uniform(0.9, 1.1, v.size)
    m.update_values(v2)
    p.update_values()
    x = np.random.default_rng(2).uniform(-1, 1, n * 3)
    y = native.Vector(ctx, n, 0, 3)
    p.apply(native.Vector(ctx, n, 0, 3).upload(x), y)
    assert_bitwise(y.download(), restatement.ilu(n, 3, rp, ci, v2, 0).apply(x), "after update_values")


@pytest.mark.parametrize("omega", [1.0, 1.3])
@pytest.mark.parametrize("order,nx,ny", [("natural", 90, 40), ("hilbert", 50, 40), ("rcm", 150, 140)])
def test_ssor(native, ctx, restatement, problems, omega, order, nx, ny):
    bs = 2
    n, rp, ci, v = _lattice(problems, nx, ny, bs, nx, order)
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
    p = native.Preconditioner(m, native.PC_SSOR, omega)
    x = np.random.default_rng(4).uniform(-1, 1, n * bs)
    y = native.Vector(ctx, n, 0, bs)
    p.apply(native.Vector(ctx, n, 0, bs).upload(x), y)
    assert_bitwise(y.download(), restatement.ssor_apply(n, bs, rp, ci, v, omega, x)[1], "SSOR")
    # Off-diagonal values written since the preconditioner was made are seen.
    v2 = v.reshape(-1, bs).copy()
    v2[ci != np.repeat(np.arange(n), np.diff(rp))] *= 0.75
    m.update_values(v2.reshape(-1))
    p.apply(native.Vector(ctx, n, 0, bs).upload(x), y)
    assert_bitwise(y.download(), restatement.ssor_apply(n, bs, rp, ci, v2.reshape(-1), omega, x)[1],
                   "SSOR, new values")


def test_ssor_unsorted_ghosts(native, ctx, restatement):
    c = cases.unsorted_case(700, 3, 12, ghosts=20, duplicates=True)
    n, bs = c["owned"], c["bs"]
    m = native.Matrix(ctx, "bsr", n, 20, bs, c["rowptr"], c["cols"], c["vals"])
    p = native.Preconditioner(m, native.PC_SSOR, 1.1)
    xv, y = native.Vector(ctx, n, 20, bs).upload(c["x"]), native.Vector(ctx, n, 20, bs)
    p.apply(xv, y)
    assert_bitwise(y.download()[: n * bs],
                   restatement.ssor_apply(n, bs, c["rowptr"], c["cols"], c["vals"], 1.1, c["x"])[1][: n * bs], "SSOR")


@pytest.mark.parametrize("kind", ["ilu", "ssor", "stored_f32", "stored_bf16"])
def test_fp32_equals_level_scheduled(native, ctx, problems, monkeypatch, kind):
    n, rp, ci, v = _lattice(problems, 130, 90, 3, 21, "rcm")
    stored = kind.startswith("stored")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v, dtype=np.float64 if stored else np.float32)

    def make():
        if stored:
            return native.Preconditioner(m, native.PC_ILU, 0, storage=native.BF16 if "bf16" in kind else native.F32)
        return native.Preconditioner(m, native.PC_SSOR if kind == "ssor" else native.PC_ILU, 1.0 if kind == "ssor" else 0)

    local = make()
    monkeypatch.setenv("OWTK_LOCAL_SWEEP", "0")
    levels = make()
    monkeypatch.delenv("OWTK_LOCAL_SWEEP")
    x = np.random.default_rng(3).uniform(-1, 1, n * 3).astype(np.float32)
    xv = native.Vector(ctx, n, 0, 3, dtype=np.float32).upload(x)
    y1, y2 = (native.Vector(ctx, n, 0, 3, dtype=np.float32) for _ in range(2))
    local.apply(xv, y1)
    levels.apply(xv, y2)
    assert_bitwise(y1.download(), y2.download(), kind)


@pytest.mark.parametrize("bs,lower", [(1, 3), (2, 8), (3, 9), (5, 5), (33, 4)])
def test_factors(native, ctx, restatement, bs, lower):
    # The data-synchronised factorisation takes rows of up to 16 entries and 8
    # lower ones; both sides of that line, odd and large block sizes.
    n, rp, ci, v = _rows_system(900, bs, lower, lambda r, g: [r - 1, r - 2, *range(r - 20, r - 20 - (lower - 2), -1)])
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
    p = native.Preconditioner(m, native.PC_ILU, 0)
    _, _, vals, inv = p.ilu_factors()
    want = restatement.ilu(n, bs, rp, ci, v, 0).factors()
    assert_bitwise(vals, want[2], "factors")
    assert_bitwise(inv, want[3], "inverse diagonal")


def test_factor_zero_pivot(native, ctx, problems):
    n, rp, ci, v = _lattice(problems, 30, 20, 2, 6)
    rows = np.repeat(np.arange(n), np.diff(rp))
    v = v.reshape(-1, 2).copy()
    v[(ci == rows) & (rows == 0)] = 0.0
    m = native.Matrix(ctx, "bsr", n, 0, 2, rp, ci, v.reshape(-1))
    with pytest.raises(native.OwtkError) as err:
        native.Preconditioner(m, native.PC_ILU, 0)
    assert err.value.kind == "zero_pivot"


def _dense(problems, nx, ny, bs, seed, order):
    rng = np.random.default_rng(seed)
    xy, edges = problems.lattice(nx, ny, 0.2, rng)
    return problems.dense_block_system(xy, edges, bs, rng, order=order)


@pytest.mark.parametrize("nx,ny,bs,order", [(5, 3, 3, "natural"), (40, 41, 3, "natural"), (33, 60, 2, "rcm"),
                                            (20, 90, 4, "natural"), (64, 31, 1, "natural"), (120, 110, 3, "rcm")])
def test_block_ilu(native, ctx, restatement, problems, nx, ny, bs, order):
    s = _dense(problems, nx, ny, bs, nx, order)
    n = s.owned
    m = native.Matrix(ctx, "dense", n, 0, bs, s.rowptr, s.cols, s.vals)
    p = native.Preconditioner(m, native.PC_BLOCK_ILU, 0)
    want = restatement.block_ilu(n, bs, s.rowptr, s.cols, s.vals).apply(s.rhs)
    x = native.Vector(ctx, n, 0, bs).upload(s.rhs)
    p.apply(x, x)
    assert_bitwise(x.download(), want, "block ILU(0) in place")


@pytest.mark.parametrize("storage", ["F32", "BF16"])
@pytest.mark.parametrize("nx,ny,bs,order", [(41, 40, 3, "natural"), (60, 33, 2, "rcm"), (30, 50, 4, "rcm"),
                                            (31, 64, 1, "natural"), (150, 140, 3, "rcm")])
def test_block_stored_equals_level_scheduled(native, ctx, problems, monkeypatch, storage, nx, ny, bs, order):
    s = _dense(problems, nx, ny, bs, nx + 1, order)
    n = s.owned
    m = native.Matrix(ctx, "dense", n, 0, bs, s.rowptr, s.cols, s.vals)
    local = native.Preconditioner(m, native.PC_BLOCK_ILU, 0, storage=getattr(native, storage))
    monkeypatch.setenv("OWTK_LOCAL_SWEEP", "0")
    levels = native.Preconditioner(m, native.PC_BLOCK_ILU, 0, storage=getattr(native, storage))
    monkeypatch.delenv("OWTK_LOCAL_SWEEP")
    x = native.Vector(ctx, n, 0, bs, dtype=np.float32).upload(s.rhs.astype(np.float32))
    y1, y2 = (native.Vector(ctx, n, 0, bs, dtype=np.float32) for _ in range(2))
    local.apply(x, y1)
    levels.apply(x, y2)
    assert_bitwise(y1.download(), y2.download(), storage)


def test_block_ilu_dependencies_beyond_the_ring(native, ctx, restatement):
    # Levels of 40 rows; every 200th row couples to a row near the start, more
    # than the ring's rows (3,600 of FP64 3 x 3 blocks) back.
    n, rp, ci, _ = _rows_system(8000, 1, 9, lambda r, g: [r - 40, r - 41] + ([int(g.integers(0, 100))]
                                                                           if r > 6000 and r % 200 == 0 else []))
    rng = np.random.default_rng(2)
    v = rng.uniform(-0.3, 0.3, size=(ci.size, 3, 3))
    v[ci == np.repeat(np.arange(n), np.diff(rp))] += 6.0 * np.eye(3)
    m = native.Matrix(ctx, "dense", n, 0, 3, rp, ci, v.reshape(-1))
    p = native.Preconditioner(m, native.PC_BLOCK_ILU, 0)
    x = rng.uniform(-1, 1, n * 3)
    y = native.Vector(ctx, n, 0, 3)
    p.apply(native.Vector(ctx, n, 0, 3).upload(x), y)
    assert_bitwise(y.download(), restatement.block_ilu(n, 3, rp, ci, v.reshape(-1)).apply(x), "block ILU(0)")
