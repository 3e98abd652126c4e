"""Gradients of the learned network at the edges of the backward kernels'
tiles (128 vertices), staging chunks and grids, against the FP64 restatement:
the cosine and relative bounds of test_learned_gpu.py, which come from the
BF16 activations and weight copies, not from the sums over the vertices."""
import numpy as np
import pytest

from test_learned_gpu import bf16_weights, unflat

pytestmark = pytest.mark.gpu


# 2 and 127-129 vertices (one tile, its edges), 64 * 256 + 1 (a row more than
# the outer products' chunks hold), more than two tiles per CTA.
@pytest.mark.parametrize("nx,ny,bs", [(2, 1, 3), (127, 1, 1), (128, 1, 3), (43, 3, 8), (16385, 1, 2), (211, 190, 3)])
def test_gradients_at_tile_edges(native, ctx, problems, nx, ny, bs):
    from oracle import gnn
    rng = np.random.default_rng(nx)
    xy, edges = problems.lattice(nx, ny, 0.2, rng)
    s = problems.component_diagonal_system(xy, edges, bs, rng)
    n = s.owned
    m = native.Matrix(ctx, "bsr", n, 0, bs, s.rowptr, s.cols, s.vals)
    net = native.Learned(m, seed=3)
    net.set_loss_weights(1.0, 0.0)
    w = bf16_weights(bs, 11)
    net.set_parameters(w)
    r, e = rng.uniform(-1, 1, n * bs), rng.uniform(-1, 1, n * bs)
    loss, got = net.loss_grad(native.Vector(ctx, n, 0, bs).upload(r), native.Vector(ctx, n, 0, bs).upload(e),
                              want_grads=True)
    want_loss, want = gnn.loss_and_grad(gnn.Graph(n, bs, s.rowptr, s.cols, s.vals), unflat(w, bs), r, e, we=1.0, wr=0.0)
    assert abs(loss - want_loss) <= 5e-2 * want_loss
    got = unflat(got, bs)
    for name, a, b in [("we", got["we"], want["we"]), ("wd", got["wd"], want["wd"])] + \
            [(f"wl{k}", got["wl"][k], want["wl"][k]) for k in range(4)]:
        a, b = a.reshape(-1), b.reshape(-1)
        assert a @ b >= 0.99 * np.linalg.norm(a) * np.linalg.norm(b), name
        assert np.linalg.norm(a - b) <= 0.1 * np.linalg.norm(b), name
