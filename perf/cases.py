"""The solver work that this library's performance is measured on.

The matrices are the benchmark's own families (2-D and 3-D Poisson, 3-D
convection-diffusion, Q1 elasticity, random-coefficient diffusion) at their
configured sizes, and `draw` spreads sizes, shapes, precisions and methods over
the ranges a user meets.  Every pass goes through the public Python mirror or
the C ABI on vectors that are already where the caller keeps them: device
pointers for the operator, preconditioner and solver calls of a resident
application, host arrays for the drop-in SMatrix call."""
import importlib.util
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_ctx = None
_generated = {}


def _b2s():
    if "b2s" not in sys.modules:
        pkg = os.path.join(_ROOT, "cpp-fem-solver_b200")
        spec = importlib.util.spec_from_file_location("b2s", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["b2s"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["b2s"]


def _context():
    """One context for the program, as an application keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = _b2s().Context(0)
    return _ctx


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the operator of a small 2-D system, applied once: a single short launch
        {"name": "spmv_poisson2d_512", "kind": "spmv", "problem": "poisson2d", "n": 512},
        # the operator of the largest 3-D system: a stream through memory
        {"name": "spmv_poisson3d_128", "kind": "spmv", "problem": "poisson3d", "n": 128},
        # 3x3 block operator of 3-D elasticity (27-point block rows)
        {"name": "matvec_elasticity_64", "kind": "matvec", "n": 64},
        # one IC(0) apply inside a user's own Krylov loop, 2-D random-coefficient diffusion, exact FP64 solves
        {"name": "ic0_apply_grf_512", "kind": "apply", "pc": "ic0", "problem": "grf", "n": 512, "precision": "fp64"},
        # one ILU(0) apply on the 3-D 7-point system, FP64, the drop-in's default
        {"name": "ilu0_apply_poisson3d_128", "kind": "apply", "pc": "ilu0", "problem": "poisson3d", "n": 128,
         "precision": "fp64"},
        # the same on a trilinear finite-element matrix (27 entries a row): no stencil of the grid schedules
        {"name": "ilu0_apply_q1_40", "kind": "apply", "pc": "ilu0", "problem": "q1", "n": 40, "precision": "fp64"},
        # block ILU(0) apply of 3-D elasticity
        {"name": "bilu0_apply_elasticity_64", "kind": "apply", "pc": "bilu0", "problem": "elasticity", "n": 64,
         "precision": "fp64"},
        # a whole solve of one 3-D system: multigrid set-up and PCG to the library's default tolerance
        {"name": "amg_pcg_poisson3d_128", "kind": "amg_pcg", "problem": "poisson3d", "n": 128},
        # the drop-in call with host arrays, on a 2-D system: hundreds of short iterations
        {"name": "smatrix_pcg_diag_256", "kind": "smatrix_pcg", "pc": "diag", "n": 256},
        # mixed precision on a nonsymmetric system: FP32 ILU(0) kept from step to step inside FP64 GMRES(30)
        {"name": "gmres_ilu0_convdiff_96", "kind": "krylov", "method": "gmres", "n": 96, "precision": "fp32"},
        # the learned preconditioner, set-up and solve, on the configuration the headline is quoted on
        {"name": "learned_pcg_grf_512", "kind": "learned_pcg", "n": 512},
        # one training step of its network on a system of the training set: forward and backward
        {"name": "learner_step_grf_512", "kind": "learner_step", "n": 512, "probes": 4},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["spmv", "matvec", "ic0", "ilu0", "ilu0", "q1", "bilu0", "amg_pcg", "smatrix_pcg", "krylov",
                       "learned_pcg", "learner_step"])
    precision = rng.choice(["fp64", "fp32"])
    if kind == "spmv":
        if rng.random() < 0.5:
            return {"kind": "spmv", "problem": "poisson2d", "n": _log(rng, 512, 1400)}
        return {"kind": "spmv", "problem": "box", "nx": _log(rng, 56, 128), "ny": _log(rng, 56, 128),
                "nz": _log(rng, 56, 128)}
    if kind == "matvec":
        return {"kind": "matvec", "n": _log(rng, 16, 64)}
    if kind == "ic0":
        if rng.random() < 0.5:
            return {"kind": "apply", "pc": "ic0", "problem": "grf", "n": _log(rng, 96, 512), "precision": precision}
        return {"kind": "apply", "pc": "ic0", "problem": "box", "nx": _log(rng, 64, 700), "ny": _log(rng, 64, 700),
                "nz": 1, "precision": precision}
    if kind == "ilu0":
        return {"kind": "apply", "pc": "ilu0", "problem": "box", "nx": _log(rng, 16, 128), "ny": _log(rng, 16, 128),
                "nz": _log(rng, 16, 128), "precision": precision}
    if kind == "q1":
        return {"kind": "apply", "pc": rng.choice(["ilu0", "ic0"]), "problem": "q1", "n": _log(rng, 12, 48),
                "precision": precision}
    if kind == "bilu0":
        return {"kind": "apply", "pc": "bilu0", "problem": "elasticity", "n": _log(rng, 12, 64),
                "precision": precision}
    if kind == "amg_pcg":
        if rng.random() < 0.5:
            return {"kind": "amg_pcg", "problem": "poisson3d", "n": _log(rng, 32, 128)}
        return {"kind": "amg_pcg", "problem": "elasticity", "n": _log(rng, 10, 48)}
    if kind == "smatrix_pcg":
        return {"kind": "smatrix_pcg", "pc": rng.choice(["diag", "ic0", "ssor"]), "n": _log(rng, 64, 256)}
    if kind == "krylov":
        return {"kind": "krylov", "method": rng.choice(["gmres", "fgmres", "bicgstab"]), "n": _log(rng, 24, 96),
                "precision": precision}
    if kind == "learned_pcg":
        return {"kind": "learned_pcg", "n": _log(rng, 128, 512)}
    return {"kind": "learner_step", "n": _log(rng, 96, 512), "probes": rng.choice([2, 4])}


# ------------------------------------------------------------------ systems

def _box(nx, ny, nz, seed):
    """-div(k grad u) on an nx x ny x nz grid (x fastest), face coefficients
    lognormal, Dirichlet outside: (n, rp, ci, v) of an SPD 5- or 7-point matrix."""
    g = np.random.default_rng(seed)
    dims, strides, n = [nx, ny] + ([nz] if nz > 1 else []), [1, nx, nx * ny], nx * ny * nz
    i = np.arange(n)
    low, high, diag = [], [], np.zeros(n)
    for d, m in enumerate(dims):
        face = np.exp(g.standard_normal(n + strides[d]))  # face[i]: below point i, face[i + stride]: above it
        at = i // strides[d] % m
        lo, hi = face[:n], face[strides[d]:]
        diag += lo + hi
        low.append(np.where(at > 0, -lo, 0.0))
        high.append(np.where(at < m - 1, -hi, 0.0))
    cols = [i - strides[d] for d in reversed(range(len(dims)))] + [i] + [i + strides[d] for d in range(len(dims))]
    vals = list(reversed(low)) + [diag] + high
    c, v = np.stack(cols, 1), np.stack(vals, 1)
    keep = v != 0.0
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.uint32)
    return n, rp, c[keep].astype(np.uint32), v[keep]


def _system(case, seed):
    """(rows, rp, ci, values) of a case's matrix; blocks of 3 x 3 for elasticity."""
    b2s = _b2s()
    problem, n = case["problem"], case.get("n")
    if problem == "grf":
        return b2s.gen_grf_diffusion(n, seed)
    if problem == "box":
        return _box(case["nx"], case["ny"], case["nz"], seed)
    if (problem, n) not in _generated:  # no seed in these: generated once a process
        if problem == "q1":
            # the x-x component of the elasticity matrix: a scalar operator on the trilinear elements' pattern
            nb, rp, ci, v = b2s.gen_elasticity_q1(n)
            made = nb, rp, ci, np.ascontiguousarray(v.reshape(-1, 9)[:, 0])
        else:
            made = {"poisson2d": b2s.gen_poisson2d, "poisson3d": b2s.gen_poisson3d, "convdiff": b2s.gen_convdiff3d,
                    "elasticity": b2s.gen_elasticity_q1}[problem](n)
        if len(_generated) > 3:
            _generated.clear()
        _generated[problem, n] = made
    return _generated[problem, n]


def _handle(case, seed):
    n, rp, ci, v = _system(case, seed)
    b2s, ctx = _b2s(), _context()
    if case["problem"] == "elasticity":
        return b2s.BAIJ(ctx, 3, n, n, rp, ci, v)
    return b2s.CSR(ctx, n, n, rp, ci, v)


def _full(case):
    """A solver case with the problem its kind stands for."""
    return dict({"problem": {"smatrix_pcg": "poisson2d", "krylov": "convdiff", "learned_pcg": "grf",
                             "learner_step": "grf", "matvec": "elasticity"}.get(case["kind"])}, **case)


def _kind(name):
    b2s = _b2s()
    return {"ic0": b2s.PC_IC0, "ilu0": b2s.PC_ILU0, "bilu0": b2s.PC_BILU0}[name]


def prepare(case, seed):
    b2s, ctx = _b2s(), _context()
    case = _full(case)
    kind, s = case["kind"], {"case": case}
    if kind == "smatrix_pcg":
        n, rp, ci, v = _system(case, seed)
        s["A"] = b2s.SMatrix(n, n, v, row_ptr=rp, col_idx=ci)
        s["b"] = b2s.uniform(seed, n)
        return s
    A = s["A"] = _handle(case, seed)
    if kind == "learner_step":
        s["net"] = b2s.Learner(ctx, weights=b2s.WEIGHTS, loss=b2s.LOSS_SWEEPS)
        s["net"].set_sweeps(trsv_sweeps=6, factor_sweeps=5)
        s["seed"] = seed
        return s
    if kind == "learned_pcg":
        s["net"] = b2s.Learner(ctx, weights=b2s.WEIGHTS)
    precision = b2s.FP32 if case.get("precision") == "fp32" else b2s.FP64
    if kind == "apply":
        s["pc"] = b2s.Precond(ctx, A, _kind(case["pc"]), precision=precision)
    if kind == "krylov":
        s["pc"] = b2s.Precond(ctx, A, b2s.PC_ILU0, precision=precision)
    s["in"] = torch.from_numpy(b2s.uniform(seed, A.n)).cuda()
    s["out"] = torch.zeros_like(s["in"])
    return s


def run(s):
    b2s, ctx, case, A = _b2s(), _context(), s["case"], s["A"]
    kind = case["kind"]
    if kind == "smatrix_pcg":
        x, _ = b2s.SMatrix.pcg(A, s["b"], case["pc"])
        return x
    if kind == "learner_step":
        loss, grad = s["net"].step(A, nprobes=case["probes"], seed=s["seed"], update=False, want_grad=True)
        return {"loss": loss, "grad": grad}
    x, y = s["in"].data_ptr(), s["out"].data_ptr()
    if kind == "spmv":
        A.spmv_device(x, y)
    elif kind == "matvec":
        ctx.check(b2s.lib().b2s_baij_matvec_device(ctx.h, A.h, x, y))
    elif kind == "apply":
        ctx.check(b2s.lib().b2s_pc_apply_device(ctx.h, s["pc"].h, x, y))
    elif kind == "amg_pcg":
        M = b2s.Precond(ctx, A, b2s.PC_BSA_AMG if case["problem"] == "elasticity" else b2s.PC_SA_AMG)
        b2s.solve_device(ctx, A, x, y, b2s.PCG, M)
    elif kind == "krylov":
        method = {"gmres": b2s.GMRES, "fgmres": b2s.FGMRES, "bicgstab": b2s.BICGSTAB}[case["method"]]
        b2s.solve_device(ctx, A, x, y, method, s["pc"], restart=30)
    else:
        M = s["net"].precond(A, precision=b2s.FP32, trsv=b2s.TRSV_JACOBI, trsv_sweeps=6, factor_sweeps=5)
        b2s.solve_device(ctx, A, x, y, b2s.PCG, M, maxit=20000)
    return s["out"]


# ------------------------------------------------------------------ work

def _sizes(case):
    """(rows, entries, block size) of a case's matrix, from its closed form."""
    p, n = case["problem"], case.get("n")
    if p in ("poisson2d", "grf"):
        return n * n, 5 * n * n - 4 * n, 1
    if p in ("poisson3d", "convdiff"):
        return n ** 3, 7 * n ** 3 - 6 * n * n, 1
    if p == "box":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        m = nx * ny * nz
        return m, m + 2 * (3 * m - ny * nz - nx * nz - nx * ny), 1
    # n^3 trilinear elements, the clamped face's nodes eliminated
    return n * (n + 1) ** 2, (3 * n - 2) * (3 * n + 1) ** 2, 3 if p == "elasticity" else 1


def work(case):
    case = _full(case)
    n, nnz, bs = _sizes(case)
    kind, n8 = case["kind"], 8 * n * bs
    A = nnz * (8 * bs * bs + 4) + 4 * (n + 1)
    mul = 2.0 * nnz * bs * bs
    if kind in ("spmv", "matvec"):
        return {"bytes": A + 2 * n8, "flops": mul}
    if kind == "apply":
        value = 4 if case["precision"] == "fp32" else 8
        kept = nnz if case["pc"] != "ic0" else (nnz + n) // 2  # IC(0) keeps one triangle and applies it twice
        return {"bytes": kept * (value * bs * bs + 4) + 4 * (n + 1) + 2 * n8, "flops": mul}
    if kind == "learner_step":
        # node states of three 64-wide layers read and written, forward and backward; two dense products each way
        return {"bytes": A + 3 * 2 * 2 * 256 * n, "flops": 3 * 3 * 2.0 * 64 * 128 * n}
    # a Krylov iteration: the operator and the preconditioner once, five vectors; iterations as measured on these
    # families at a relative residual of 1e-10
    if kind == "amg_pcg":
        its = 27 if bs == 1 else 60
    elif kind == "krylov":
        its = 28
    elif kind == "smatrix_pcg":
        its = 3.4 * case["n"] if case["pc"] == "diag" else 1.05 * case["n"]
    else:
        its = 1.3 * case["n"]
    its = max(1.0, its)
    return {"bytes": its * (2 * A + 5 * n8), "flops": its * (2 * mul + 10.0 * n * bs)}


# ------------------------------------------------------------------ 64-bit values

def _rows(n, rp, ci, v, bs):
    """Rows padded to the widest: columns (n, w), -1 where there is none, and blocks (n, w, bs, bs)."""
    count = np.diff(rp.astype(np.int64))
    w = int(count.max())
    row = np.repeat(np.arange(n), count)
    slot = np.arange(len(ci)) - np.repeat(rp[:-1].astype(np.int64), count)
    cols = np.full((n, w), -1, np.int64)
    cols[row, slot] = ci
    vals = np.zeros((n, w, bs, bs))
    vals[row, slot] = v.reshape(-1, bs, bs)
    return cols, vals


def _levels(n, cols):
    """Rows grouped so that each group's lower neighbours lie in earlier groups."""
    lower = (cols >= 0) & (cols < np.arange(n)[:, None])
    left, done = lower.sum(1), np.zeros(n, bool)
    order = np.argsort(cols, axis=None, kind="stable")
    order = order[lower.reshape(-1)[order]]  # lower entries by column: who waits for a row
    start = np.searchsorted(cols.reshape(-1)[order], np.arange(n + 1))
    who = order // cols.shape[1]
    now, groups = np.nonzero(left == 0)[0], []
    while len(now):
        groups.append(now)
        done[now] = True
        size = start[now + 1] - start[now]
        hit = who[np.repeat(start[now], size) + np.arange(size.sum()) - np.repeat(np.cumsum(size) - size, size)]
        np.subtract.at(left, hit, 1)
        now = np.unique(hit[left[hit] == 0])
    return groups


def _ilu0_apply(n, rp, ci, v, bs, r, upper_only):
    """z = (LU)^-1 r of the zero-fill (block) factorisation, which for a symmetric matrix is IC(0)'s operator too.
    upper_only: the scalar ILU(0) of the library, as the reference's, updates the kept entries of U alone."""
    cols, f = _rows(n, rp, ci, v, bs)
    row = np.arange(n)
    at = np.argmax(cols == row[:, None], axis=1)  # the diagonal's slot
    groups, w = _levels(n, cols), cols.shape[1]
    inv = np.zeros((n, bs, bs))
    for g in groups:
        for k in range(int(at[g].max())):
            sub = g[at[g] > k]
            j = cols[sub, k]
            f[sub, k] = f[sub, k] @ inv[j]
            for m in range(int(at[j].min()) + 1, w):
                ok = (m > at[j]) & (cols[j, m] >= 0)
                i, jj = sub[ok], j[ok]
                hit = cols[i] == cols[jj, m][:, None]
                slot = np.argmax(hit, axis=1)
                there = hit[np.arange(len(i)), slot] 
                if upper_only:
                    there &= slot >= at[i]
                i, jj, slot = i[there], jj[there], slot[there]
                f[i, slot] -= f[i, k] @ f[jj, m]
        inv[g] = np.linalg.inv(f[g, at[g]])
    z = r.reshape(n, bs, 1).copy()
    for g in groups:
        for k in range(int(at[g].max())):
            sub = g[at[g] > k]
            z[sub] -= f[sub, k] @ z[cols[sub, k]]
    for g in reversed(groups):  # upper entries lie in later groups of a matrix with a symmetric pattern
        for k in range(int(at[g].min()) + 1, w):
            sub = g[(at[g] < k) & (cols[g, k] >= 0)]
            z[sub] -= f[sub, k] @ z[cols[sub, k]]
        z[g] = inv[g] @ z[g]
    return z.reshape(-1)


def _poisson(n, dims, b):
    """The Dirichlet Poisson solution by sine transforms."""
    x = torch.from_numpy(b).reshape([n] * dims)
    for d in range(dims):
        x = _dst(x, d)
    lam = 2 - 2 * torch.cos(torch.arange(1, n + 1, dtype=torch.float64) * (np.pi / (n + 1)))
    total = sum(lam.reshape([n if e == d else 1 for e in range(dims)]) for d in range(dims))
    x = x / total
    for d in range(dims):
        x = _dst(x, d) * (2.0 / (n + 1))
    return x.reshape(-1)


def _dst(x, d):
    x = x.movedim(d, -1)
    zero = torch.zeros_like(x[..., :1])
    odd = torch.cat([zero, x, zero, -x.flip(-1)], -1)
    return (-torch.fft.fft(odd).imag[..., 1:x.shape[-1] + 1] / 2).movedim(-1, d)


def exact(case, seed):
    case = _full(case)
    kind, problem = case["kind"], case["problem"]
    if kind in ("smatrix_pcg", "amg_pcg") and problem in ("poisson2d", "poisson3d"):
        dims = 2 if problem == "poisson2d" else 3
        x = _poisson(case["n"], dims, _b2s().uniform(seed, case["n"] ** dims))
        return x.numpy() if kind == "smatrix_pcg" else x
    if kind not in ("spmv", "matvec", "apply"):
        return None
    n, rp, ci, v = _system(case, seed)
    bs = 3 if problem == "elasticity" else 1
    x = _b2s().uniform(seed, n * bs)
    if kind in ("spmv", "matvec"):
        terms = np.einsum("kij,kj->ki", v.reshape(-1, bs, bs), x.reshape(n, bs)[ci])
        return torch.from_numpy(np.add.reduceat(terms, rp[:-1].astype(np.int64), axis=0).reshape(-1))
    if n * bs * bs > 800_000 and problem in ("elasticity", "q1"):
        return None  # over about 20 seconds
    return torch.from_numpy(_ilu0_apply(n, rp, ci, v, bs, x, case["pc"] == "ilu0"))
