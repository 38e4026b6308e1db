"""Multicolour SSOR on the GPU (array.cpp:2947-3164): colouring and
renumbering identical to the restatement, apply bit-exact, PCG parity."""
import numpy as np
import pytest

import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mat", ["bipartite", "greedy", "convdiff"])
def test_ssor_colouring_and_apply(b2s, ctx, orc, mat):
    n, rp, ci, v = {"bipartite": lambda: P.poisson2d(45), "greedy": lambda: P.random_spd(1200, 0.005, 9),
                    "convdiff": lambda: P.convdiff2d(40)}[mat]()
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    for omega in (1.2, 0.7):
        M = b2s.Precond(ctx, A, b2s.PC_SSOR, omega=omega)
        po = orc.pc(orc.csr(n, n, rp, ci, v), "ssor", omega)
        nc, cptr, nid, perm, d2 = orc.colour_export(po)
        rp_, ci_, v_ = M.export("ssor.colour")
        assert len(rp_) == nc + 1 and np.array_equal(rp_, cptr)
        assert np.array_equal(ci_, nid) and np.array_equal(v_, d2)
        r = b2s.uniform(41, n)
        assert np.array_equal(M.apply(r), po.apply(r))


@pytest.mark.parametrize("n,links", [(1, 0), (7, 0), (2, 1), (300, 1), (301, 1), (301, 3)])
def test_ssor_colour_counts(b2s, ctx, orc, n, links):
    # one colour (no links), two (a path or an even ring), three and more (an odd
    # ring, longer links), with entries on one side of the diagonal only among them
    rng = np.random.default_rng(n + links)
    d = np.zeros((n, n))
    for k in range(1, links + 1):
        for i in range(n):
            d[i, (i + k) % n] = rng.uniform(-1, 1)
            if i % 3:
                d[(i + k) % n, i] = rng.uniform(-1, 1)
    d[np.arange(n), np.arange(n)] = rng.uniform(4, 8, n) * rng.choice([-1, 1], n)
    row, col = np.nonzero(d)
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.uint32)
    ci, v = col.astype(np.uint32), d[row, col]
    M = b2s.Precond(ctx, b2s.CSR(ctx, n, n, rp, ci, v), b2s.PC_SSOR)
    r = rng.uniform(-1, 1, n)
    r[::5] = -0.0
    z, want = M.apply(r), orc.pc(orc.csr(n, n, rp, ci, v), "ssor", 1.2).apply(r)
    assert np.array_equal(z, want) and np.array_equal(np.signbit(z), np.signbit(want))


@pytest.mark.parametrize("n,entries", [(40, 240), (40, 241), (500, 8000), (600, 300)])
def test_ssor_two_colours(b2s, ctx, orc, n, entries):
    # two colours on both sides of the row length (7 n entries with the diagonal)
    # from which the first one's values are stored and read, not formed by their readers
    rng = np.random.default_rng(entries)
    half, d = n // 2, np.zeros((n, n))
    at = rng.permutation(2 * half * half)[:entries]
    i, j = at % (half * half) // half, half + at % half
    d[np.where(at < half * half, i, j), np.where(at < half * half, j, i)] = rng.uniform(-1, 1, entries)
    d[np.arange(n), np.arange(n)] = rng.uniform(4, 8, n) * rng.choice([-1, 1], n)
    row, col = np.nonzero(d)
    assert len(row) == n + entries
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.uint32)
    ci, v = col.astype(np.uint32), d[row, col]
    M = b2s.Precond(ctx, b2s.CSR(ctx, n, n, rp, ci, v), b2s.PC_SSOR)
    r = rng.uniform(-1, 1, n)
    assert np.array_equal(M.apply(r), orc.pc(orc.csr(n, n, rp, ci, v), "ssor", 1.2).apply(r))


def test_ssor_bad_omega(b2s, ctx):
    n, rp, ci, v = P.poisson2d(5)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    for w in (0.0, 2.0, -1.0):
        with pytest.raises(ValueError):
            b2s.Precond(ctx, A, b2s.PC_SSOR, omega=w)


@pytest.mark.parametrize("method", [0, 1, 2])
def test_ssor_solver_parity(b2s, ctx, orc, method):
    n, rp, ci, v = P.poisson2d(40) if method == 0 else P.convdiff2d(40)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    b = b2s.uniform(42, n)
    M = b2s.Precond(ctx, A, b2s.PC_SSOR)
    x, st = b2s.solve(ctx, A, b, method, M, tol=1e-8, maxit=2000, restart=30)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), method, "ssor", b, 1e-8, 2000, 30)
    assert abs(st["it"] - io) <= 2
    assert np.linalg.norm(x - xo) / np.linalg.norm(xo) < 1e-9
