"""Level-scheduled applies (OWTK_LOCAL_SWEEP=0, and what wide levels take): ILU
on packed factor segments and in place, SSOR, split SSOR and dense-block ILU, bit
for bit against the oracle; FP32 and whole solves packed against in place; the
cluster and lockstep schedules against the level-scheduled one.  Every test first
asks that the schedule it is about is in use."""
import numpy as np
import pytest

import cases
from conftest import assert_bitwise
from test_local_sweep_gpu import _dense, _lattice

pytestmark = pytest.mark.gpu


@pytest.fixture
def by_level(monkeypatch):
    monkeypatch.setenv("OWTK_LOCAL_SWEEP", "0")
    monkeypatch.setenv("OWTK_CHAIN_SWEEP", "0")
    return monkeypatch


def _checked(p):
    assert p.local_schedule().warps == 0 and p.chain_windows() == 0
    assert p.sweep_schedule()[0] == 0 and p.lockstep_schedule()[0] == 0
    return p


def _ilu(native, m, monkeypatch, fill=0, packed=True):
    monkeypatch.setenv("OWTK_PACKED_SWEEP", "1" if packed else "0")
    return _checked(native.Preconditioner(m, native.PC_ILU, fill))


def _apply(native, ctx, p, n, bs, x, in_place=False):
    xv = native.Vector(ctx, n, 0, bs, dtype=x.dtype).upload(x)
    y = xv if in_place else native.Vector(ctx, n, 0, bs, dtype=x.dtype)
    p.apply(xv, y)
    return y.download()


@pytest.mark.parametrize("nx,ny,bs,order,fill", [(120, 120, 3, "rcm", 0), (110, 90, 1, "rcm", 0),
                                                 (90, 70, 4, "natural", 0), (100, 100, 2, "rcm", 1),
                                                 (70, 60, 3, "rcm", 2), (60, 61, 5, "natural", 1),
                                                 (50, 40, 2, "hilbert", 0), (12, 40, 32, "natural", 0),
                                                 (20, 20, 33, "natural", 0)])
def test_ilu(native, ctx, restatement, problems, by_level, nx, ny, bs, order, fill):
    n, rp, ci, v = _lattice(problems, nx, ny, bs, nx + bs, order)
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
    x = np.random.default_rng(nx).uniform(-1, 1, n * bs)
    want = restatement.ilu(n, bs, rp, ci, v, fill).apply(x)
    for packed in (True, False):
        p = _ilu(native, m, by_level, fill, packed)
        assert_bitwise(_apply(native, ctx, p, n, bs, x), want, f"packed {packed}")
        assert_bitwise(_apply(native, ctx, p, n, bs, x, in_place=True), want, f"packed {packed}, in place")


def test_ilu_after_numeric_update(native, ctx, restatement, problems, by_level):
    n, rp, ci, v = _lattice(problems, 100, 90, 3, 4, "rcm")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v)
    p = _ilu(native, m, by_level)
    v2 = v * np.random.default_rng(9).uniform(0.9, 1.1, v.size)
    m.update_values(v2)
    p.update_values()
    x = np.random.default_rng(8).uniform(-1, 1, n * 3)
    assert_bitwise(_apply(native, ctx, p, n, 3, x), restatement.ilu(n, 3, rp, ci, v2, 0).apply(x), "updated")


def test_ilu_fp32_and_solve_packed_equal_in_place(native, ctx, problems, by_level):
    n, rp, ci, v = _lattice(problems, 110, 110, 3, 12, "rcm")
    x = np.random.default_rng(13).uniform(-1, 1, n * 3)
    m32 = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v, dtype=np.float32)
    a, b = (_apply(native, ctx, _ilu(native, m32, by_level, 0, k), n, 3, x.astype(np.float32)) for k in (True, False))
    assert_bitwise(a, b, "FP32")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v)
    rhs = native.Vector(ctx, n, 0, 3).upload(x)
    got = []
    for packed in (True, False):
        s = native.Vector(ctx, n, 0, 3)
        r = native.solve(native.FGMRES, m, _ilu(native, m, by_level, 0, packed), rhs, s)
        assert r.status == 0
        got.append((r.iterations, s.download()))
    assert got[0][0] == got[1][0]
    assert_bitwise(got[0][1], got[1][1], "solution")


@pytest.mark.parametrize("omega", [1.0, 1.3])
@pytest.mark.parametrize("nx,ny,bs,order", [(90, 40, 2, "natural"), (150, 140, 3, "rcm"), (50, 40, 1, "hilbert"),
                                            (12, 40, 33, "natural")])
def test_ssor(native, ctx, restatement, problems, by_level, omega, nx, ny, bs, order):
    n, rp, ci, v = _lattice(problems, nx, ny, bs, nx, order)
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
    p = _checked(native.Preconditioner(m, native.PC_SSOR, omega))
    x = np.random.default_rng(4).uniform(-1, 1, n * bs)
    want = restatement.ssor_apply(n, bs, rp, ci, v, omega, x)[1]
    assert_bitwise(_apply(native, ctx, p, n, bs, x), want, "SSOR")
    assert_bitwise(_apply(native, ctx, p, n, bs, x, in_place=True), want, "SSOR in place")


@pytest.mark.parametrize("omega", [1.0, 1.4])
def test_split_ssor(native, ctx, restatement, problems, by_level, omega):
    n, rp, ci, v = _lattice(problems, 80, 90, 3, 31, "rcm")
    orp, oci, diag, off = cases.split_of(dict(owned=n, bs=3, rowptr=rp, cols=ci, vals=v))
    d, o = (native.Vector(ctx, a.size, 0, 1).upload(a.reshape(-1)) for a in (diag, off))
    m = native.Matrix(ctx, "split", n, 0, 3, orp, oci, diag_ptr=d.data_ptr, off_ptr=o.data_ptr)
    p = _checked(native.Preconditioner(m, native.PC_SPLIT_SSOR, omega))
    x = np.random.default_rng(6).uniform(-1, 1, n * 3)
    want = restatement.split_ssor_apply(n, 3, orp, oci, diag, off, omega, x)
    assert_bitwise(_apply(native, ctx, p, n, 3, x), want, "split SSOR")


@pytest.mark.parametrize("nx,ny,bs,order", [(64, 31, 1, "natural"), (33, 60, 2, "rcm"), (120, 110, 3, "rcm"),
                                            (40, 90, 4, "natural")])
def test_block_ilu(native, ctx, restatement, problems, by_level, nx, ny, bs, order):
    s = _dense(problems, nx, ny, bs, nx, order)
    n = s.owned
    m = native.Matrix(ctx, "dense", n, 0, bs, s.rowptr, s.cols, s.vals)
    p = _checked(native.Preconditioner(m, native.PC_BLOCK_ILU, 0))
    want = restatement.block_ilu(n, bs, s.rowptr, s.cols, s.vals).apply(s.rhs)
    assert_bitwise(_apply(native, ctx, p, n, bs, s.rhs), want, "block ILU(0)")
    assert_bitwise(_apply(native, ctx, p, n, bs, s.rhs, in_place=True), want, "block ILU(0) in place")


@pytest.mark.parametrize("env,query", [("OWTK_CLUSTER_SWEEP", "sweep_schedule"), ("OWTK_LOCKSTEP_SWEEP", "lockstep_schedule")])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_cluster_schedules_equal_level_scheduled(native, ctx, problems, by_level, env, query, dtype):
    n, rp, ci, v = _lattice(problems, 110, 100, 3, 44, "rcm")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v, dtype=dtype)
    levels = _ilu(native, m, by_level)
    by_level.setenv(env, "1")
    cluster = native.Preconditioner(m, native.PC_ILU, 0)
    assert getattr(cluster, query)()[0] > 0 and cluster.local_schedule().warps == 0
    x = np.random.default_rng(7).uniform(-1, 1, n * 3).astype(dtype)
    assert_bitwise(_apply(native, ctx, cluster, n, 3, x), _apply(native, ctx, levels, n, 3, x), env)


# Tasks (two components of a row) a level on both sides of 4,500 for each lower
# entry of the mean row (0.83, 2.5 and 1.67 of them here).
@pytest.mark.parametrize("width,lower,bs,by_value", [(400, 1, 16, True), (600, 1, 16, False), (1100, 3, 20, True),
                                                     (1500, 3, 20, False), (150, 1, 64, False), (300, 2, 33, True)])
def test_factors_by_value_or_flag(native, ctx, restatement, width, lower, bs, by_value):
    depth = 6
    n = width * depth
    r = np.arange(n)
    e = []
    for d in range(lower):
        some = r[(r >= width) & (r % width + d < width)]
        e.append(np.stack([some, some - width + d], 1))
    e = np.concatenate(e)
    rows, cols = np.concatenate([r, e[:, 0], e[:, 1]]), np.concatenate([r, e[:, 1], e[:, 0]])
    o = np.lexsort((cols, rows))
    rows, cols = rows[o], cols[o]
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    v = -np.random.default_rng(width).uniform(0.05, 1.0, size=(cols.size, bs))
    v[rows == cols] = 2.5 * lower
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, cols, v.reshape(-1))
    p = native.Preconditioner(m, native.PC_ILU, 0)
    assert p.factor_by_value() == by_value
    _, _, values, inverse = p.ilu_factors()
    want = restatement.ilu(n, bs, rp, cols, v.reshape(-1), 0).factors()
    assert_bitwise(values, want[2], "factors")
    assert_bitwise(inverse, want[3], "inverse diagonal")
