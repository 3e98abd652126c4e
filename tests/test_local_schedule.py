"""The plan of the one-CTA-per-component sweeps, on the CPU: what may not be
planned, and which schedule is taken.

A team copies its next tasks' operands some steps ahead, dependencies beyond
the shared-memory ring among them, so such a dependency has to lie further back
than the copies reach; a plan in which one does not is refused (the applies then
take the level-scheduled sweep)."""
import numpy as np
import pytest

WIDTH = 40                    # rows a level: steps of two tasks
# Two tasks in flight for each of twelve teams, one round of the teams until a
# result is in global memory, and the wait itself.
NEEDED = (2 + 1) * 12 + 1
NO_FAR = 2 ** 31 - 1


def levels(depth, far_levels=0):
    """Row p of a level couples to rows p and p - 1 of the level before; every
    300th row to the one `far_levels` further up as well; symmetric."""
    n = WIDTH * depth
    r = np.arange(n)
    pairs = [np.stack([r[WIDTH:], r[WIDTH:] - WIDTH], 1)]
    inner = r[(r >= WIDTH) & (r % WIDTH > 0)]
    pairs.append(np.stack([inner, inner - WIDTH - 1], 1))
    if far_levels:
        some = r[(r >= WIDTH * far_levels) & (r % 300 == 0)]
        pairs.append(np.stack([some, some - WIDTH * far_levels], 1))
    e = np.concatenate(pairs)
    rows, cols = np.concatenate([r, e[:, 0], e[:, 1]]), np.concatenate([r, e[:, 1], e[:, 0]])
    o = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return n, rp, cols[o]


def test_plan_without_far_values(native):
    n, rp, ci = levels(200)
    s = native.local_schedule_plan(n, 3, rp, ci)
    assert (s.warps, s.lower_steps, s.upper_steps) == (2, 200, 200)
    assert (s.far_values, s.slow_tasks, s.far_steps) == (0, 0, NO_FAR)


@pytest.mark.parametrize("back,taken", [(NEEDED - 1, False), (NEEDED, True), (60, True)])
def test_far_values_lie_behind_the_copies(native, back, taken):
    n, rp, ci = levels(200, back)
    s = native.local_schedule_plan(n, 3, rp, ci, ring_rows=1000)   # 1,000 rows: 23 levels back at most
    assert (s.warps > 0) == taken
    if taken:
        assert s.far_values > 0 and s.far_steps == back
    whole = native.local_schedule_plan(n, 3, rp, ci)               # the ring of the applies holds them all
    assert whole.warps == 2 and whole.far_values == 0


def couples(width, depth, count):
    """Levels of `width` rows; a row couples to `count` neighbours in the level before."""
    n = width * depth
    r = np.arange(n)
    e = []
    for d in range(-(count // 2), count - count // 2):
        some = r[(r >= width) & (r % width + d >= 0) & (r % width + d < width)]
        e.append(np.stack([some, some - width + d], 1))
    e = np.concatenate(e)
    rows, cols = np.concatenate([r, e[:, 0], e[:, 1]]), np.concatenate([r, e[:, 1], e[:, 0]])
    o = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return n, rp, cols[o]


# Two to seven steps a level against the level-scheduled sweep, by what both
# measured at these widths (ns a level, local / level-scheduled); 0: the
# level-scheduled sweep is the faster one.
@pytest.mark.parametrize("count,width,bs,ssor,warps", [
    (3, 600, 1, False, 4),     # 623 / 785
    (3, 900, 1, False, 0),
    (7, 384, 2, False, 4),     # 717 / 799
    (7, 512, 2, False, 0),     # 991 / 819: 24 rows a task
    (7, 640, 2, False, 0),     # 1,170 / 825
    (3, 600, 1, True, 4),      # 844 / 880
    (3, 512, 64, True, 0),     # 1,579 / 1,324: the values are copied at every apply
    (3, 128, 64, True, 4),     # 433 / 1,013
    (7, 640, 2, True, 4),      # 1,457 / 1,833: two rounds of entries there
])
def test_the_cheaper_schedule_is_taken(native, count, width, bs, ssor, warps):
    n, rp, ci = couples(width, 30, count)
    assert native.local_schedule_plan(n, bs, rp, ci, ssor=ssor).warps == warps
