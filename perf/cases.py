"""The work that programs using this library have it do, as measurable cases.

A case is a dict of plain values; `listed()` gives the standing ones and
`draw(rng)` more of the same ranges.  `prepare` builds what a program holds
before the call (matrix, preconditioner or network handles, vectors, a
workspace), `run` is one pass through the public entry points, `exact` the
same outputs in 64-bit torch without the library's code.

Meshes are jittered triangulated lattices like those of
owtk_b200/problems.py, each cell split along a random diagonal, so vertices
have 2 to 8 neighbours as on an unstructured mesh.  The mesh belongs to the
case; coefficients, right-hand sides and network inputs come from the seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "owt-krylov_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from owtk_b200 import checkpoint, native  # noqa: E402

_WEIGHTS = os.path.join(_PKG, "weights", "learned_anisotropic_bs3.owtkgnn")
_SOLVER = {"fgmres": native.FGMRES, "bicgstab": native.BICGSTAB, "pipelined_bicgstab": native.PIPELINED_BICGSTAB,
           "comm_hiding_bicgstab": native.COMM_HIDING_BICGSTAB, "idrs": native.IDRS}
_PC = {"jacobi": native.PC_JACOBI, "ssor": native.PC_SSOR, "ilu": native.PC_ILU}
_SSOR_OMEGA = 1.0
# Iterations these systems take to 1e-8 (FGMRES, learned and mixed: their own
# tolerances), for work() only.
_ITERATIONS = {"jacobi": 34, "ssor": 12, "ilu": 9, "learned": 12, "mixed": 9, "batch": 32}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # An application's smallest product: a split diagonal/edge view (borrowed
        # device coefficients), where the launch is most of the call.
        {"name": "spmv_split_5k", "op": "spmv", "kind": "split", "nx": 73, "ny": 69, "bs": 4, "dtype": "f64",
         "order": "natural"},
        # The headline product: component-diagonal blocks, 2M vertices, larger than L2.
        {"name": "spmv_bsr_2m", "op": "spmv", "kind": "bsr", "nx": 1451, "ny": 1379, "bs": 3, "dtype": "f64",
         "order": "rcm"},
        # One block-Jacobi ILU(0) apply at scale, the larger part of a plain solve.
        {"name": "ilu0_apply_1m", "op": "ilu", "nx": 1013, "ny": 989, "bs": 3, "dtype": "f64", "order": "rcm"},
        # SSOR in an application's own numbering, as the SpecWave solver ids use it.
        {"name": "ssor_apply_90k", "op": "ssor", "nx": 311, "ny": 290, "bs": 2, "dtype": "f64", "order": "natural"},
        # A time step's numeric update: coefficients of the same pattern in device
        # memory re-gathered, ILU(0) refactored and applied.
        {"name": "ilu0_refactor_50k", "op": "refactor", "nx": 253, "ny": 198, "bs": 4, "dtype": "f64",
         "order": "rcm"},
        # The small plain solve: 64 x 64 lattice, BiCGSTAB + Jacobi, latency-bound.
        {"name": "bicgstab_jacobi_4096", "op": "solve", "solver": "bicgstab", "pc": "jacobi", "nx": 64, "ny": 64,
         "bs": 3, "dtype": "f64", "order": "natural"},
        # The plain method at an ordinary size: GMRES(30) + ILU(0).
        {"name": "gmres_ilu0_200k", "op": "solve", "solver": "fgmres", "pc": "ilu", "nx": 449, "ny": 447, "bs": 3,
         "dtype": "f64", "order": "rcm"},
        # Mixed precision: dense 3x3 blocks, BF16 factors under FP64 FGMRES, rtol 1e-10.
        {"name": "mixed_dense_100k", "op": "mixed", "nx": 331, "ny": 303, "bs": 3, "storage": "bf16", "inner": 0,
         "order": "rcm"},
        # Many uneven systems in one persistent launch.
        {"name": "batch_bicgstab_24", "op": "batch", "count": 24, "n_min": 1000, "n_max": 40000, "mix": 5},
        # The learned preconditioner alone, with the committed weights.
        {"name": "learned_apply_600k", "op": "learned", "nx": 787, "ny": 769, "bs": 3, "order": "rcm"},
        # The headline solve: learned-preconditioned FGMRES with one damped Jacobi
        # correction and ILU(0) fallback, anisotropic coefficients.
        {"name": "learned_fgmres_150k", "op": "solve", "solver": "fgmres", "pc": "learned", "nx": 391, "ny": 387,
         "bs": 3, "dtype": "f64", "order": "rcm"},
        # One training step of the network: loss, gradients and Adam.
        {"name": "learned_train_100k", "op": "train", "nx": 317, "ny": 313, "bs": 3, "order": "rcm"},
    ]


def draw(rng):
    """One more case: a path, then sizes log-uniform over its range."""
    def lattice(lo, hi):
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        nx = max(8, round(math.sqrt(n * rng.uniform(0.5, 2.0))))
        return {"nx": nx, "ny": max(8, round(n / nx))}

    op = rng.choice(["spmv", "spmv", "ilu", "ssor", "refactor", "solve", "solve", "mixed", "batch", "learned",
                     "train"])
    c = {"op": op}
    if op == "spmv":
        c.update(kind=rng.choice(["bsr", "split", "dense"]), bs=rng.choice([1, 2, 3, 4, 5, 8]),
                 dtype=rng.choice(["f64", "f64", "f32"]), order=rng.choice(["rcm", "natural", "hilbert"]))
        c.update(lattice(2000, 2000000 if c["bs"] <= 3 and c["kind"] != "dense" else 250000))
    elif op in ("ilu", "ssor", "refactor"):
        c.update(bs=rng.choice([1, 2, 3, 4, 8]) if op == "ilu" else rng.randint(1, 4), dtype="f64",
                 order=rng.choice(["rcm", "rcm", "natural", "hilbert"]) if op != "refactor" else "rcm")
        c.update(lattice(1000, 20000 if c["order"] == "hilbert" else 1000000 if op == "ilu" and c["bs"] <= 3
                         else 200000))
        if op != "refactor":
            c["dtype"] = rng.choice(["f64", "f64", "f32"])
    elif op == "solve":
        c.update(solver=rng.choice(["fgmres", "fgmres", "bicgstab", "pipelined_bicgstab", "comm_hiding_bicgstab",
                                    "idrs"]),
                 pc=rng.choice(["jacobi", "ssor", "ilu"]), bs=rng.randint(1, 4), dtype="f64",
                 order=rng.choice(["rcm", "natural"]))
        if c["solver"] == "fgmres" and rng.random() < 0.4:
            c.update(pc="learned", bs=3, order="rcm")
        c.update(lattice(1000, 200000))
    elif op == "mixed":
        c.update(bs=rng.randint(2, 4), storage=rng.choice(["bf16", "f32"]), inner=rng.choice([0, 0, 1, 2]),
                 order="rcm")
        c.update(lattice(2000, 100000))
    elif op == "batch":
        c.update(count=rng.randint(3, 32), n_min=1000, n_max=rng.choice([5000, 20000, 30000]),
                 mix=rng.randrange(1, 1 << 20))
    else:
        c.update(bs=3, order="rcm")
        c.update(lattice(2000, 600000 if op == "learned" else 100000))
    return c


# ------------------------------------------------------------------ meshes
class _Mesh:
    """Pattern of one lattice: CSR on the host (the API's arrays), and on the
    device where each entry's value comes from and the padded row table."""


def _native_mesh(nx, ny):
    rng = np.random.default_rng([nx, ny])
    hx, hy = 1.0 / max(nx - 1, 1), 1.0 / max(ny - 1, 1)
    gx, gy = np.meshgrid(np.arange(nx) * hx, np.arange(ny) * hy)
    xy = np.stack([gx.ravel(), gy.ravel()], axis=1)
    xy += rng.uniform(-0.2, 0.2, size=xy.shape) * np.array([hx, hy])
    idx = np.arange(nx * ny).reshape(ny, nx)
    flip = (rng.random((ny - 1, nx - 1)) < 0.5).ravel()
    a = np.where(flip, idx[:-1, 1:].ravel(), idx[:-1, :-1].ravel())
    b = np.where(flip, idx[1:, :-1].ravel(), idx[1:, 1:].ravel())
    edges = np.concatenate([np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()], axis=1),
                            np.stack([idx[:-1, :].ravel(), idx[1:, :].ravel()], axis=1),
                            np.stack([a, b], axis=1)])
    return xy, edges


def _csr(n, i, j):
    """Sorted pattern of diagonal + both directions of every edge: (rowptr, rows, cols, source of each entry)."""
    ar = torch.arange(n, device="cuda")
    rows, cols = torch.cat([ar, i, j]), torch.cat([ar, j, i])
    key, src = torch.sort(rows * n + cols)
    rows, cols = key // n, key % n
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return rowptr, rows, cols, src


def _host(t, dtype=np.uint64):
    return np.ascontiguousarray(t.cpu().numpy().astype(dtype))


@functools.lru_cache(maxsize=48)
def _mesh(nx, ny, order):
    xy, edges = _native_mesh(nx, ny)
    m = _Mesh()
    m.n = n = nx * ny
    e = torch.from_numpy(edges).cuda()
    m.new_to_old = None
    if order != "natural":
        if order == "rcm":
            rowptr, _, cols, _ = _csr(n, e[:, 0], e[:, 1])
            perm = native.rcm_order(n, _host(rowptr), _host(cols))
        else:
            perm = native.hilbert_order(xy)
        m.new_to_old = torch.from_numpy(perm).cuda()
        inverse = torch.empty_like(m.new_to_old)
        inverse[m.new_to_old] = torch.arange(n, device="cuda")
        e_new = inverse[e]
    else:
        e_new = e
    m.xy, m.edges = torch.from_numpy(xy).cuda(), e          # original numbering
    rowptr, rows, m.cols, m.src = _csr(n, e_new[:, 0], e_new[:, 1])
    m.rows, m.nnz = rows, int(m.cols.numel())
    m.is_diag = m.cols == rows
    m.h_rowptr, m.h_cols = _host(rowptr), _host(m.cols)
    off_rowptr = rowptr - torch.arange(n + 1, device="cuda")
    m.h_off_rowptr, m.h_off_cols = _host(off_rowptr), _host(m.cols[~m.is_diag])
    pos = torch.arange(m.nnz, device="cuda") - rowptr[rows]
    m.width = int(pos.max()) + 1
    m.table = torch.full((n, m.width), -1, dtype=torch.int64, device="cuda")   # CSR entries of each row
    m.table[rows, pos] = torch.arange(m.nnz, device="cuda")
    m.table_cols = torch.where(m.table >= 0, m.cols[m.table.clamp(min=0)], 0)
    return m


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(0x9e3779b9 ^ int(seed))


def _uniform(shape, lo, hi, g):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) * (hi - lo) + lo


def _reorder(m, nodes):
    return nodes if m.new_to_old is None else nodes[m.new_to_old]


def _spread(m, entries):
    """(n, width, ...) table of per-entry values, zero where a row has fewer."""
    t = entries[m.table.clamp(min=0)]
    return torch.where((m.table >= 0).reshape(m.table.shape + (1,) * (t.dim() - 2)), t, 0)


def _edge_weights(m, bs, g, anisotropic):
    """a_ij, a_ji per edge and component: -w (1 + s), -w (1 - s)."""
    edges = m.edges.shape[0]
    if anisotropic:   # w = 1 + 1e4 (e . d)^2, d rotated by a smooth random angle field
        p, q = m.xy[m.edges[:, 0]], m.xy[m.edges[:, 1]]
        mid, ev = 0.5 * (p + q), q - p
        k = torch.randint(-3, 4, (6, 2), device="cuda", generator=g).double()
        amp = torch.randn(6, dtype=torch.float64, device="cuda", generator=g) / 6.0
        phase = _uniform((6,), 0.0, 2.0 * math.pi, g)
        theta = math.pi * (torch.sin(2.0 * math.pi * (mid[:, :1] * k[:, 0] + mid[:, 1:] * k[:, 1]) + phase) * amp).sum(1)
        ev = ev / ev.square().sum(1, keepdim=True).sqrt()
        w = (1.0 + 1e4 * (ev[:, 0] * theta.cos() + ev[:, 1] * theta.sin()) ** 2)[:, None].expand(edges, bs)
    else:
        w = _uniform((edges, bs), 0.5, 1.5, g)
    s = _uniform((edges, bs), -0.3, 0.3, g)
    return -w * (1.0 + s), -w * (1.0 - s)


def _values(m, bs, g, anisotropic=False):
    """Component-diagonal values [entry][component] of a diagonally dominant system."""
    fwd, bwd = _edge_weights(m, bs, g, anisotropic)
    noise = _uniform((m.n, bs), 0.0, 0.1, g)
    v = torch.cat([torch.zeros((m.n, bs), dtype=torch.float64, device="cuda"), fwd, bwd])[m.src]
    v[m.is_diag] = 1.05 * _spread(m, v.abs()).sum(1) + _reorder(m, noise)
    return v


def _dense_values(m, bs, g):
    """Dense blocks: off-diagonal -w (I + 0.3 R), diagonal 1.1 sum |off|_1 I + 0.05 N(0, 1)."""
    edges = m.edges.shape[0]
    eye = torch.eye(bs, dtype=torch.float64, device="cuda")
    w = _uniform((edges, 1, 1), 0.5, 1.5, g)

    def normal(*shape):
        return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)

    fwd, bwd = (-w * (eye + 0.1 * normal(edges, bs, bs)) for _ in range(2))
    noise = 0.05 * normal(m.n, bs, bs)
    v = torch.cat([torch.zeros((m.n, bs, bs), dtype=torch.float64, device="cuda"), fwd, bwd])[m.src]
    size = v.abs().sum(1).amax(1)
    v[m.is_diag] = 1.1 * _spread(m, size).sum(1)[:, None, None] * eye + _reorder(m, noise)
    return v


def _torch_dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.float64


def _system(case, seed):
    """(mesh, matrix values, right-hand side) in the matrix's numbering and type."""
    m, bs, g, t = _mesh(case["nx"], case["ny"], case["order"]), case["bs"], _generator(seed), _torch_dtype(case)
    if case["op"] == "mixed" or case.get("kind") == "dense":
        v = _dense_values(m, bs, g)
    else:
        v = _values(m, bs, g, case["op"] in ("learned", "train") or case.get("pc") == "learned")
    b = _reorder(m, _uniform((m.n, bs), -1.0, 1.0, g))
    return m, v.to(t), b.to(t).contiguous()


def _batch_parts(case, seed):
    rng = np.random.default_rng(case["mix"])
    for i in range(case["count"]):
        n = math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))
        ny = max(2, round(math.sqrt(n / rng.uniform(1.0, 4.0))))
        part = {"op": "solve", "pc": "jacobi", "order": "natural", "nx": max(2, round(n / ny)), "ny": ny,
                "bs": int(rng.integers(1, 5))}
        yield part, int(seed) * 1000 + i


def _network_input(case, seed):
    """Training pair: an error e and the residual r = A e it leaves."""
    m, v, e = _system(case, seed)
    return m, v, (_spread(m, v) * e[m.table_cols]).sum(1), e


# --------------------------------------------------------------- the library
@functools.lru_cache(maxsize=1)
def _context():
    return native.Context(0)


class _State:
    pass


def _vector(ctx, t, owned, bs):
    """The library's view of a torch tensor."""
    return native.Vector.view(ctx, owned, 0, bs, t.data_ptr(), t.numel(),
                              np.float32 if t.dtype == torch.float32 else np.float64)


def prepare(case, seed):
    ctx, s = _context(), _State()
    s.case, op = case, case["op"]
    if op == "batch":
        systems, rhs = [], []
        for part, k in _batch_parts(case, seed):
            m, v, b = _system(part, k)
            systems.append((m.n, part["bs"], m.h_rowptr, m.h_cols, v.cpu().numpy().reshape(-1)))
            rhs.append(b.reshape(-1))
        s.batch = native.Batch(ctx, systems)
        s.t_in = torch.cat(rhs)
        s.t_out = torch.zeros_like(s.t_in)
        s.x, s.y = (_vector(ctx, t, t.numel(), 1) for t in (s.t_in, s.t_out))
        s.options = native.default_options()
        torch.cuda.synchronize()
        return s
    bs = case["bs"]
    if op == "train":
        m, v, s.t_in, s.t_out = _network_input(case, seed)
        s.t_in, s.t_out = s.t_in.contiguous(), s.t_out.contiguous()
    else:
        m, v, s.t_in = _system(case, seed)
        s.t_out = torch.zeros_like(s.t_in)
    n, np_dtype = m.n, np.float32 if _torch_dtype(case) == torch.float32 else np.float64
    if case.get("kind") == "split":
        s.diag, s.off = v[m.is_diag].contiguous(), v[~m.is_diag].contiguous()
        torch.cuda.synchronize()
        s.matrix = native.Matrix(ctx, "split", n, 0, bs, m.h_off_rowptr, m.h_off_cols, diag_ptr=s.diag.data_ptr(),
                                 off_ptr=s.off.data_ptr(), dtype=np_dtype)
    elif op == "refactor":
        # The application's arrays in its own numbering; the matrix is the permuted gather.
        own = _mesh(case["nx"], case["ny"], "natural")
        w = _values(own, bs, _generator(seed))
        s.t_diag, s.t_off = w[own.is_diag].contiguous(), w[~own.is_diag].contiguous()
        s.diag = _vector(ctx, s.t_diag, n, bs)
        s.off = _vector(ctx, s.t_off, s.t_off.shape[0], bs)
        s.permutation = native.Permutation(ctx, m.new_to_old.cpu().numpy())
        torch.cuda.synchronize()
        s.matrix = s.permutation.permuted_split_matrix(bs, own.h_off_rowptr, own.h_off_cols, s.diag, s.off)
    else:
        kind = "dense" if op == "mixed" or case.get("kind") == "dense" else "bsr"
        s.matrix = native.Matrix(ctx, kind, n, 0, bs, m.h_rowptr, m.h_cols, v.cpu().numpy().reshape(-1),
                                 dtype=np_dtype)
    s.x, s.y = _vector(ctx, s.t_in, n, bs), _vector(ctx, s.t_out, n, bs)
    pc = case.get("pc", {"refactor": "ilu"}.get(op, op))
    if pc in ("learned", "train"):
        s.net = native.Learned(s.matrix, seed=1)
        checkpoint.load_network(_WEIGHTS, s.net)
    if op == "mixed":
        storage = native.BF16 if case["storage"] == "bf16" else native.F32
        s.pc = native.Preconditioner(s.matrix, native.PC_BLOCK_ILU, 0, storage=storage, mixed_inner=case["inner"])
    elif pc in _PC:
        s.pc = native.Preconditioner(s.matrix, _PC[pc], _SSOR_OMEGA if pc == "ssor" else 0.0)
    elif op == "solve":
        s.fallback = native.Preconditioner(s.matrix, native.PC_ILU, 0)
        s.pc = native.LearnedPreconditioner(s.net, s.fallback)
        s.pc.set_correction(1, 0.7)
    s.kind = _SOLVER[case.get("solver", "fgmres")]
    s.options = native.default_options(restart=30, relative_tolerance=1e-10 if op == "mixed" else 1e-8)
    s.workspace = native.Workspace(ctx)
    torch.cuda.synchronize()
    ctx.synchronize()
    return s


def run(s):
    op = s.case["op"]
    if op == "spmv":
        s.matrix.apply(s.x, s.y)
    elif op in ("ilu", "ssor"):
        s.pc.apply(s.x, s.y)
    elif op == "refactor":
        native.update_permuted_split(s.matrix, s.diag, s.off)
        s.pc.update_values(s.matrix)
        s.pc.apply(s.x, s.y)
    elif op in ("solve", "mixed"):
        s.y.fill(0.0)
        r = native.solve(s.kind, s.matrix, s.pc, s.x, s.y, s.options, s.workspace)
        return {"x": s.t_out, "status": int(r.status)}
    elif op == "batch":
        s.y.fill(0.0)
        results = s.batch.solve(s.x, s.y, s.options)
        return {"x": s.t_out, "status": np.array([r.status for r in results])}
    elif op == "learned":
        s.net.apply(s.x, s.y)
    else:
        loss, grads = s.net.loss_grad(s.x, s.y, want_grads=True)
        s.net.adam_step(3e-4)
        return {"loss": loss, "grads": grads}
    return s.t_out


# ------------------------------------------------------------------- floors
def _counts(case):
    nx, ny = case["nx"], case["ny"]
    n, edges = nx * ny, nx * (ny - 1) + ny * (nx - 1) + (nx - 1) * (ny - 1)
    return n, n + 2 * edges


def work(case):
    op = case["op"]
    if op == "batch":
        parts = [work(p) for p, _ in _batch_parts(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nnz = _counts(case)
    bs, sv = case["bs"], 4 if case.get("dtype") == "f32" else 8
    per = bs * bs if op == "mixed" or case.get("kind") == "dense" else bs
    vec = n * bs * sv
    mat, mflops = nnz * (per * sv + 4) + (n + 1) * 4, 2 * nnz * per
    spmv = mat + 2 * vec
    if op == "spmv":
        return {"bytes": spmv, "flops": mflops}
    if op in ("ilu", "ssor"):      # factors (or matrix) and diagonal once, both sweeps' vectors
        return {"bytes": mat + 5 * vec, "flops": mflops + 2 * n * bs}
    if op == "refactor":           # values in, matrix and factors out, then the apply
        return {"bytes": 2 * nnz * bs * sv + 2 * mat + 6 * vec, "flops": 3 * mflops}
    # The network: per vertex and layer its row in and out, once more for the
    # gathered rows' slot list (8 columns and BF16 weights); 64 x 128 products.
    net = {"bytes": n * (4 * (2 * 128 + 48) + 4 * bs * 8), "flops": n * (4 * 2 * 128 * 64 + 2 * 64 * 24)}
    if op == "learned":
        return net
    if op == "train":              # forward, the two products of the backward, their operands kept
        return {"bytes": 3 * net["bytes"] + 2 * spmv, "flops": 3 * net["flops"]}
    its = _ITERATIONS["mixed" if op == "mixed" else case["pc"]]
    if op == "mixed":
        apply_bytes = nnz * (per * (2 if case["storage"] == "bf16" else 4) + 4) + 4 * vec
    elif case["pc"] == "learned":
        apply_bytes = net["bytes"] + spmv + 3 * vec
    else:
        apply_bytes = mat + 5 * vec if case["pc"] in ("ilu", "ssor") else 3 * vec
    if case.get("solver", "fgmres") == "fgmres":      # two Gram-Schmidt passes over a basis of half the count
        each = spmv + apply_bytes + (its + 3) * vec
        flops = mflops + 4 * its * n * bs
    else:
        each = 2 * (spmv + apply_bytes) + 15 * vec
        flops = 2 * mflops + 30 * n * bs
    if case.get("pc") == "learned":
        flops += net["flops"]
    return {"bytes": its * each, "flops": its * flops}


# -------------------------------------------------------------------- exact
def _matvec(m, table, x):
    """y = A x from the (n, width, bs[, bs]) table of values."""
    g = x[m.table_cols]
    if table.dim() == 4:
        return (table @ g[..., None])[..., 0].sum(1)
    return (table * g).sum(1)


def _settle(step, x, limit=3000):
    """x = step(x) to its fixed point in 64 bits."""
    for k in range(limit):
        y = step(x)
        if k % 20 == 19 and float((y - x).abs().max()) <= 2e-16 * float(y.abs().max()):
            return y
        x = y
    return x


def _solution(m, v, b):
    """A^-1 b of a diagonally dominant system: Jacobi iteration until it stands still."""
    v, b = v.double(), b.double()
    table = _spread(m, v)
    d = v[m.is_diag]
    d = torch.diagonal(d, dim1=1, dim2=2) if v.dim() == 3 else d
    return _settle(lambda x: x + (b - _matvec(m, table, x)) / d, b / d)


def _ilu0(m, a):
    """ILU(0) values in the pattern (unit lower part, upper part with the
    diagonal): the defining equations iterated to their fixed point."""
    n, key = m.n, m.rows * m.n + m.cols
    lower = torch.nonzero(m.cols < m.rows)[:, 0]
    left, up, target = [], [], []
    for j in range(m.width):           # entry (k, c) of slot j of row k, for every lower entry (i, k)
        e = m.table[m.cols[lower], j]
        ok = (e >= 0) & (m.cols[e.clamp(min=0)] > m.cols[lower])
        l, u = lower[ok], e[ok]
        want = m.rows[l] * n + m.cols[u]
        at = torch.searchsorted(key, want).clamp(max=m.nnz - 1)
        hit = key[at] == want
        left.append(l[hit])
        up.append(u[hit])
        target.append(at[hit])
    left, up, target = torch.cat(left), torch.cat(up), torch.cat(target)
    diag_at = torch.nonzero(m.is_diag)[:, 0]
    is_lower = (m.cols < m.rows)[:, None]

    def step(f):
        w = a.index_add(0, target, f[left] * f[up], alpha=-1.0)
        return torch.where(is_lower, w / f[diag_at[m.cols]], w)

    return _settle(step, torch.where(is_lower, a / a[diag_at[m.cols]], a), 400)


def _ilu_apply(m, a, b):
    f = _ilu0(m, a)
    below, above = (m.cols < m.rows)[:, None], (m.cols > m.rows)[:, None]
    d = f[m.is_diag]
    lo, hi = _spread(m, torch.where(below, f, 0)), _spread(m, torch.where(above, f, 0))
    y = _settle(lambda x: b - _matvec(m, lo, x), b, 1000)
    return _settle(lambda x: (y - _matvec(m, hi, x)) / d, y / d, 1000)


def _ssor_apply(m, a, b):
    d = a[m.is_diag]
    lo = _spread(m, torch.where((m.cols < m.rows)[:, None], _SSOR_OMEGA * a, 0))
    hi = _spread(m, torch.where((m.cols > m.rows)[:, None], _SSOR_OMEGA * a, 0))
    y = _settle(lambda x: (b - _matvec(m, lo, x)) / d, b / d)
    return _settle(lambda x: (d * y - _matvec(m, hi, x)) / d, y)


def _network(m, v, r, p, bs):
    """The message-passing network in 64 bits; p: encoder, layers, decoder."""
    d = v[m.is_diag]
    w = torch.where(m.is_diag, 0.0, -(v / d[m.rows]).mean(1))
    wt, q = _spread(m, w)[..., None], r / d
    sr, sq = r.square().mean().sqrt(), q.square().mean().sqrt()
    x = torch.cat([r / sr, q / sq, torch.zeros((m.n, 16 - 2 * bs), dtype=torch.float64, device="cuda")], 1)
    h = x @ p[0].T
    for wl in p[1:5]:
        agg = torch.zeros_like(h)
        for j in range(m.width):
            agg = agg + wt[:, j] * h[m.table_cols[:, j]]
        h = h + torch.relu(torch.cat([h, agg], 1) @ wl.T)
    return q + sq * (h @ p[5][:bs].T)


def _parameters():
    flat = torch.from_numpy(checkpoint.load(_WEIGHTS)["parameters"]).cuda().double()
    parts = list(torch.split(flat, [64 * 16] + [64 * 128] * 4 + [8 * 64]))
    return [parts[0].reshape(64, 16)] + [t.reshape(64, 128) for t in parts[1:5]] + [parts[5].reshape(8, 64)]


def _permuted(m, own, w):
    """Values of P A P^T: edges keep their place in the source list, nodes are relabelled."""
    sourced = torch.empty_like(w)
    sourced[own.src] = w
    return torch.cat([sourced[:m.n][m.new_to_old], sourced[m.n:]])[m.src]


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        xs = [_solution(*_system(p, k)).reshape(-1) for p, k in _batch_parts(case, seed)]
        return {"x": torch.cat(xs), "status": None}
    if op == "train":
        m, v, r, e = _network_input(case, seed)
        p = [t.requires_grad_() for t in _parameters()]
        z = _network(m, v, r, p, case["bs"])
        table = _spread(m, v)
        loss = (0.1 * (z - e).square().sum() / e.square().sum()
                + (r - _matvec(m, table, z)).square().sum() / r.square().sum())
        grads = torch.autograd.grad(loss, p)
        return {"loss": loss.detach(), "grads": torch.cat([t.reshape(-1) for t in grads])}
    if op == "refactor":
        own = _mesh(case["nx"], case["ny"], "natural")
        w = _values(own, case["bs"], _generator(seed))
        m, _, b = _system(case, seed)
        return _ilu_apply(m, _permuted(m, own, w), b)
    m, v, b = _system(case, seed)
    if op == "spmv":
        return _matvec(m, _spread(m, v.double()), b.double())
    if op == "ilu":
        return _ilu_apply(m, v.double(), b.double())
    if op == "ssor":
        return _ssor_apply(m, v.double(), b.double())
    if op == "learned":
        return _network(m, v, b, _parameters(), case["bs"])
    return {"x": _solution(m, v, b), "status": None}
