"""Gradients of the learned network where a lost row would be most of them: the
loss's gradient sits on one vertex, at an end of the vertices, of a tile (128) or
of an outer product's chunk (64 rows of a block's range).  Checked against the
same system numbered backwards, in which that vertex is elsewhere in its tile.

A vertex's own arithmetic does not depend on its number; only the order of FP32
sums does.  Another order moves such a sum by about 2^-24 of its size, which
moves one in some 10^4 of the BF16 activations behind it by 2^-8: less than 1e-3
of a gradient.  A lost or doubled row changes it by half or more."""
import numpy as np
import pytest

from test_learned_gpu import bf16_weights, unflat

pytestmark = pytest.mark.gpu

BOUND = 1e-2


def backwards(n, bs, rowptr, cols, vals):
    rows = np.repeat(np.arange(n), np.diff(rowptr))
    rows, cols = n - 1 - rows, n - 1 - np.asarray(cols)
    o = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rp[1:])
    return rp, cols[o], vals.reshape(-1, bs)[o].reshape(-1)


def turned(a, n, bs):
    return np.ascontiguousarray(a.reshape(n, bs)[::-1]).reshape(-1)


@pytest.mark.parametrize("nx,ny,bs", [(2, 1, 3), (127, 1, 1), (128, 1, 3), (43, 3, 8), (64, 5, 2), (16385, 1, 2),
                                      (211, 190, 3)])
def test_gradient_of_one_vertex(native, ctx, problems, nx, ny, bs):
    rng = np.random.default_rng(nx)
    xy, edges = problems.lattice(nx, ny, 0.2, rng)
    s = problems.component_diagonal_system(xy, edges, bs, rng)
    n = s.owned
    w = bf16_weights(bs, 11)
    nets = []
    for rp, ci, v in [(s.rowptr, s.cols, s.vals), backwards(n, bs, s.rowptr, s.cols, s.vals)]:
        m = native.Matrix(ctx, "bsr", n, 0, bs, rp, ci, v)
        net = native.Learned(m, seed=3)
        net.set_loss_weights(1.0, 0.0)
        net.set_parameters(w)
        nets.append(net)
    r = rng.uniform(-1, 1, n * bs)
    rv, out = native.Vector(ctx, n, 0, bs).upload(r), native.Vector(ctx, n, 0, bs)
    nets[0].apply(rv, out)
    out = out.download()
    for target in sorted({t for t in (0, 63, 64, 127, 128, n // 2, n - 1) if t < n}):
        e = out.copy()
        e[target * bs:(target + 1) * bs] += 1e3 * np.abs(out).max() * rng.uniform(0.5, 1.0, bs)
        got = []
        for net, turn in zip(nets, (False, True)):
            a, b = (turned(x, n, bs) if turn else x for x in (r, e))
            loss, g = net.loss_grad(native.Vector(ctx, n, 0, bs).upload(a), native.Vector(ctx, n, 0, bs).upload(b),
                                    want_grads=True)
            got.append((loss, unflat(g, bs)))
        assert abs(got[0][0] - got[1][0]) <= 1e-4 * got[0][0]
        one, two = got[0][1], got[1][1]
        for name, a, b in [("we", one["we"], two["we"]), ("wd", one["wd"], two["wd"])] + \
                [(f"wl{k}", one["wl"][k], two["wl"][k]) for k in range(4)]:
            assert np.linalg.norm(a) > 0
            assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(a), (target, name)
