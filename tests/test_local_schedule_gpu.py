"""Applies with one CTA per component, on patterns whose schedule is known: each
test first asks that the schedule it is about is the one in use (steps of one,
two and four tasks, values beyond the ring, tasks of the slower form), then
compares with the oracle bit for bit, or in FP32 and with stored factors with
the level-scheduled sweep, asked for and checked to be in use."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_local_sweep_gpu import _dense, _lattice, _rows_system

pytestmark = pytest.mark.gpu


def _levels(width, depth, bs, seed, far=0, back=0):
    """Rows of a level couple to three neighbours in the one before; every
    293rd row from `back` levels on to `far` rows of the first levels as well."""
    rng = np.random.default_rng(seed)

    def neighbours(r, _):
        p = r % width
        near = [r - width + d for d in (-1, 0, 1) if 0 <= p + d < width]
        return near + (rng.integers(0, 8 * width, size=far).tolist() if r >= width * back and r % 293 == 0 else [])
    return _rows_system(width * depth, bs, seed, neighbours)


def _preconditioner(native, ctx, kind, n, bs, rp, ci, v, dtype=np.float64):
    m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v, dtype=dtype)
    return m, native.Preconditioner(m, native.PC_SSOR if kind == "ssor" else native.PC_ILU, 1.2 if kind == "ssor" else 0)


def _want(restatement, kind, n, bs, rp, ci, v, x):
    if kind == "ssor":
        return restatement.ssor_apply(n, bs, rp, ci, v, 1.2, x)[1]
    return restatement.ilu(n, bs, rp, ci, v, 0).apply(x)


def _apply(native, ctx, p, n, bs, x):
    y = native.Vector(ctx, n, 0, bs, dtype=x.dtype)
    p.apply(native.Vector(ctx, n, 0, bs, dtype=x.dtype).upload(x), y)
    return y.download()


# Widths at the edges of tasks and of steps of 1, 2 and 4 of them.
@pytest.mark.parametrize("kind", ["ilu", "ssor"])
@pytest.mark.parametrize("width,warps", [(31, 1), (32, 1), (33, 2), (64, 2), (97, 4), (128, 4), (129, 2), (256, 4),
                                         (257, 4), (480, 4)])
@pytest.mark.parametrize("bs", [1, 3])
def test_steps(native, ctx, restatement, kind, width, warps, bs):
    n, rp, ci, v = _levels(width, 40, bs, width)
    _, p = _preconditioner(native, ctx, kind, n, bs, rp, ci, v)
    s = p.local_schedule()
    if kind == "ssor" and width == 129:
        warps = 4   # three steps of two tasks 410 ns, two of four 369
    assert s.warps == warps and s.far_values == s.slow_tasks == 0
    x = np.random.default_rng(2).uniform(-1, 1, n * bs)
    assert_bitwise(_apply(native, ctx, p, n, bs, x), _want(restatement, kind, n, bs, rp, ci, v, x), kind)


# 11,934 rows fit the ring with steps of two or four tasks, 20,400 with one.
@pytest.mark.parametrize("kind", ["ilu", "ssor"])
@pytest.mark.parametrize("width,depth", [(32, 900), (60, 400), (128, 180)])
@pytest.mark.parametrize("far,slow", [(2, False), (40, True)])
def test_beyond_the_ring(native, ctx, restatement, kind, width, depth, far, slow):
    n, rp, ci, v = _levels(width, depth, 2, far, far, depth * 4 // 5)
    _, p = _preconditioner(native, ctx, kind, n, 2, rp, ci, v)
    s = p.local_schedule()
    assert s.warps > 0 and s.far_values > 0 and (s.slow_tasks > 0) == slow
    x = np.random.default_rng(3).uniform(-1, 1, n * 2)
    assert_bitwise(_apply(native, ctx, p, n, 2, x), _want(restatement, kind, n, 2, rp, ci, v, x), kind)


# The tables of a direction are filled by up to four threads, from 512 tasks on.
@pytest.mark.parametrize("kind", ["ilu", "ssor"])
@pytest.mark.parametrize("width,depth,far", [(24, 600, 0), (60, 1200, 2), (60, 1200, 40)])
def test_tables_filled_in_ranges(native, ctx, restatement, kind, width, depth, far):
    n, rp, ci, v = _levels(width, depth, 1, far, far, depth // 3)
    _, p = _preconditioner(native, ctx, kind, n, 1, rp, ci, v)
    s = p.local_schedule()
    assert s.warps > 0 and (s.far_values > 0) == (far > 0) and (s.slow_tasks > 0) == (far > 8)
    x = np.random.default_rng(5).uniform(-1, 1, n)
    assert_bitwise(_apply(native, ctx, p, n, 1, x), _want(restatement, kind, n, 1, rp, ci, v, x), kind)


@pytest.mark.parametrize("kind", ["ilu", "ssor"])
@pytest.mark.parametrize("width,slow", [(8, False), (9, True), (17, True)])
def test_long_rows(native, ctx, restatement, kind, width, slow):
    n, rp, ci, v = _rows_system(3000, 1, width, lambda r, g: list(range(r - 30, r - 30 - (width if r % 150 == 0 else 2), -1)))
    _, p = _preconditioner(native, ctx, kind, n, 1, rp, ci, v)
    s = p.local_schedule()
    assert s.warps > 0 and (s.slow_tasks > 0) == slow
    x = np.random.default_rng(4).uniform(-1, 1, n)
    assert_bitwise(_apply(native, ctx, p, n, 1, x), _want(restatement, kind, n, 1, rp, ci, v, x), kind)


def _both(native, ctx, monkeypatch, make):
    local = make()
    monkeypatch.setenv("OWTK_LOCAL_SWEEP", "0")
    levels = make()
    monkeypatch.delenv("OWTK_LOCAL_SWEEP")
    assert local.local_schedule().warps > 0 and levels.local_schedule().warps == 0
    return local, levels


@pytest.mark.parametrize("kind", ["ilu", "ssor", "stored_f32", "stored_bf16"])
@pytest.mark.parametrize("width,depth,far", [(20, 40, 0), (50, 40, 0), (110, 420, 3), (300, 40, 0)])
def test_fp32_equals_level_scheduled(native, ctx, monkeypatch, kind, width, depth, far):
    n, rp, ci, v = _levels(width, depth, 3, width, far, depth * 4 // 5)
    stored = kind.startswith("stored")
    m = native.Matrix(ctx, "bsr", n, 0, 3, rp, ci, v, dtype=np.float64 if stored else np.float32)

    def make():
        if stored:
            return native.Preconditioner(m, native.PC_ILU, 0, storage=native.BF16 if "bf16" in kind else native.F32)
        return native.Preconditioner(m, native.PC_SSOR if kind == "ssor" else native.PC_ILU, 1.2 if kind == "ssor" else 0)
    local, levels = _both(native, ctx, monkeypatch, make)
    assert (local.local_schedule().far_values > 0) == (far > 0)
    x = np.random.default_rng(5).uniform(-1, 1, n * 3).astype(np.float32)
    assert_bitwise(_apply(native, ctx, local, n, 3, x), _apply(native, ctx, levels, n, 3, x), kind)


@pytest.mark.parametrize("nx,ny,bs,order", [(40, 41, 1, "natural"), (33, 60, 2, "rcm"), (30, 90, 3, "natural"),
                                            (20, 90, 4, "natural")])
def test_block_ilu(native, ctx, restatement, problems, nx, ny, bs, order):
    s = _dense(problems, nx, ny, bs, nx, order)
    n = s.owned
    m = native.Matrix(ctx, "dense", n, 0, bs, s.rowptr, s.cols, s.vals)
    p = native.Preconditioner(m, native.PC_BLOCK_ILU, 0)
    assert p.local_schedule().warps == 1
    want = restatement.block_ilu(n, bs, s.rowptr, s.cols, s.vals).apply(s.rhs)
    assert_bitwise(_apply(native, ctx, p, n, bs, s.rhs), want, "block ILU(0)")


# 2,181 rows of FP64 3 x 3 blocks fit the ring, more of the other kinds: the
# rows that reach back start after four fifths of 300 levels of 40.
@pytest.mark.parametrize("storage", ["F64", "F32", "BF16"])
def test_block_ilu_beyond_the_ring(native, ctx, restatement, monkeypatch, storage):
    n, rp, ci, _ = _levels(40, 300, 1, 6, 1, 240)
    rng = np.random.default_rng(2)
    v = rng.uniform(-0.3, 0.3, size=(ci.size, 3, 3))
    v[ci == np.repeat(np.arange(n), np.diff(rp))] += 6.0 * np.eye(3)
    m = native.Matrix(ctx, "dense", n, 0, 3, rp, ci, v.reshape(-1))
    x = rng.uniform(-1, 1, n * 3)
    local, levels = _both(native, ctx, monkeypatch,
                          lambda: native.Preconditioner(m, native.PC_BLOCK_ILU, 0, storage=getattr(native, storage)))
    s = local.local_schedule()
    assert s.far_values > 0 and s.far_steps < 2 ** 31 - 1
    if storage != "F64":
        x = x.astype(np.float32)
    got = _apply(native, ctx, local, n, 3, x)
    assert_bitwise(got, _apply(native, ctx, levels, n, 3, x), storage)
    if storage == "F64":
        assert_bitwise(got, restatement.block_ilu(n, 3, rp, ci, v.reshape(-1)).apply(x), "block ILU(0)")


@pytest.mark.parametrize("storage", ["F32", "BF16"])
@pytest.mark.parametrize("nx,ny,bs,order", [(41, 40, 3, "natural"), (60, 33, 2, "rcm"), (30, 50, 4, "rcm"),
                                            (31, 64, 1, "natural")])
def test_block_stored_equals_level_scheduled(native, ctx, problems, monkeypatch, storage, nx, ny, bs, order):
    s = _dense(problems, nx, ny, bs, nx + 1, order)
    n = s.owned
    m = native.Matrix(ctx, "dense", n, 0, bs, s.rowptr, s.cols, s.vals)
    local, levels = _both(native, ctx, monkeypatch,
                          lambda: native.Preconditioner(m, native.PC_BLOCK_ILU, 0, storage=getattr(native, storage)))
    x = s.rhs.astype(np.float32)
    assert_bitwise(_apply(native, ctx, local, n, bs, x), _apply(native, ctx, levels, n, bs, x), storage)


def test_plan_is_the_schedule_in_use(native, ctx, problems):
    n, rp, ci, v = _lattice(problems, 128, 130, 3, 258, "rcm")
    for kind in ("ilu", "ssor"):
        plan = native.local_schedule_plan(n, 3, rp, ci, ssor=kind == "ssor")
        _, p = _preconditioner(native, ctx, kind, n, 3, rp, ci, v)
        s = p.local_schedule()
        assert all(getattr(s, k) == getattr(plan, k) for k, _ in s._fields_), kind
