"""GPU parity of the core path through the C ABI: SpMV, dot, BAIJ matvec and
the Krylov solvers with identity / diagonal / block-Jacobi preconditioners,
against the C restatement (oracle/b2s_oracle.c).

Tolerances: SpMV and BAIJ matvec rows are summed in the reference's order,
so they must be bit-exact.  Solver results differ from the oracle only by the
association of the dot products (fixed-order tree on the GPU, ascending on
the CPU): iteration counts within +/-2, relative solution difference below
1e-10 unless the problem is ill-conditioned (stated per case)."""
import numpy as np
import pytest

import problems as P

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def long_row_matrix(n=5000):
    """Row 0 is dense (n nonzeros, > the staging capacity), row 1 empty."""
    R, Cc, V = [], [], []
    for j in range(n):
        R.append(0); Cc.append(j); V.append(1.0 / (j + 1))
    for i in range(2, n):
        R += [i, i]; Cc += [i, i - 1]; V += [2.0, -0.5]
    rp, ci, v = P.coo_to_csr(n, n, R, Cc, V)
    return n, rp, ci, v


@pytest.mark.parametrize("case", ["poisson", "random", "longrow", "tiny", "rect", "big3d", "rows33"])
def test_spmv_bit_exact(b2s, ctx, orc, case):
    # one thread per row below 2^20 rows of <= 32 nonzeros ("poisson", "random",
    # "rect", "tiny"); the warp kernel above ("big3d": 102^3 rows; "longrow",
    # "rows33": a row longer than 32)
    if case == "rect":
        n, m = 300, 500
        rng = np.random.default_rng(0)
        dense = (rng.random((n, m)) < 0.02) * rng.uniform(-1, 1, (n, m))
        rp = np.concatenate([[0], np.cumsum((dense != 0).sum(1))]).astype(np.uint32)
        ci = np.nonzero(dense)[1].astype(np.uint32)
        v = dense[dense != 0]
    else:
        n, rp, ci, v = {"poisson": lambda: P.poisson2d(100), "random": lambda: P.random_spd(3000, 0.004, 1),
                        "big3d": lambda: b2s.gen_poisson3d(102), "rows33": lambda: long_row_matrix(33),
                        "longrow": long_row_matrix, "tiny": lambda: P.coo_to_csr(1, 1, [0], [0], [3.0]) and
                        (1, *P.coo_to_csr(1, 1, [0], [0], [3.0]))}[case]()
        m = n
    A = b2s.CSR(ctx, n, m, rp, ci, v)
    x = np.random.default_rng(5).uniform(-1, 1, m)
    y = A.spmv(x)
    yo = orc.spmv(orc.csr(n, m, rp, ci, v), x)
    assert np.array_equal(y, yo)


def test_dot_deterministic(b2s, ctx):
    rng = np.random.default_rng(1)
    for n in (0, 1, 255, 256, 100003, 3_000_000):
        a, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        d1, d2 = b2s.dot(ctx, a, b), b2s.dot(ctx, a, b)
        assert d1 == d2
        ref = float(np.dot(a, b))
        assert abs(d1 - ref) <= 1e-13 * max(1.0, np.abs(a * b).sum())


@pytest.mark.parametrize("bs", [1, 2, 3, 4])
def test_baij_matvec_bit_exact(b2s, ctx, orc, bs):
    n, rp, ci, v = P.make_test_scalar(40, 3) if bs == 3 else P.poisson2d(60)
    Ao = orc.csr(n, n, rp, ci, v)
    nb = n // bs
    Bo = orc.blk_condense(bs, Ao, nb, nb)
    brp, bci, bv = Bo.export()
    B = b2s.BAIJ(ctx, bs, nb, nb, brp, bci, bv)
    x = P.drand(np.arange(n))
    assert np.array_equal(B.matvec(x), orc.blk_matvec(Bo, x))


@pytest.mark.parametrize("bs", [2, 3, 4])
def test_baij_matvec_irregular(b2s, ctx, orc, bs):
    # ragged block rows: empty rows, single blocks and rows of 100+ blocks,
    # which span several passes of the warp kernel
    rng = np.random.default_rng(bs)
    nb = 700
    lens = rng.integers(0, 12, nb)
    lens[::97] = 0
    lens[5] = 150
    lens[400] = 90
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    ci = np.concatenate([np.sort(rng.choice(nb, size=k, replace=False)) for k in lens]).astype(np.uint32)
    v = rng.uniform(-1, 1, len(ci) * bs * bs)
    B = b2s.BAIJ(ctx, bs, nb, nb, rp, ci, v)
    Bo = orc.blk(bs, nb, nb, rp, ci, v)
    x = rng.uniform(-1, 1, nb * bs)
    assert np.array_equal(B.matvec(x), orc.blk_matvec(Bo, x))


@pytest.mark.parametrize("bs", [2, 3, 4])
@pytest.mark.parametrize("nb", [1, 3553, 60001])
def test_baij_matvec_streams(b2s, ctx, orc, bs, nb):
    # a warp's range of several row groups: empty groups and ranges, rows longer
    # than the ring of dots, ranges that start at any block
    rng = np.random.default_rng(nb)
    lens = rng.integers(0, 30, nb)
    lens[nb // 3:nb // 3 + 50] = 0
    lens[::1009] = 1 if nb == 1 else 300
    rp = np.concatenate([[0], np.cumsum(lens)])
    gaps = rng.integers(1, 4, rp[-1])
    walk = np.concatenate([[0], np.cumsum(gaps)])
    start = rng.integers(0, max(1, nb - 1200), nb)
    row = np.repeat(np.arange(nb), lens)
    ci = (start[row] + walk[:-1] - walk[rp[row]]).astype(np.uint32)
    rp = rp.astype(np.uint32)
    v = rng.uniform(-1, 1, len(ci) * bs * bs)
    B = b2s.BAIJ(ctx, bs, nb, nb, rp, ci, v)
    Bo = orc.blk(bs, nb, nb, rp, ci, v)
    x = rng.uniform(-1, 1, nb * bs)
    assert np.array_equal(B.matvec(x), orc.blk_matvec(Bo, x))


def test_baij_elasticity_matvec(b2s, ctx, orc):
    nbr, rp, ci, v = b2s.gen_elasticity_q1(10)
    B = b2s.BAIJ(ctx, 3, nbr, nbr, rp, ci, v)
    Bo = orc.blk(3, nbr, nbr, rp, ci, v)
    x = b2s.uniform(3, 3 * nbr)
    assert np.array_equal(B.matvec(x), orc.blk_matvec(Bo, x))


SOLVER_CASES = [
    (b"pcg", 0, "none"), (b"pcg", 0, "diag"), (b"pcg", 0, "cg"),
    (b"bicgstab", 1, "none"), (b"bicgstab", 1, "diag"),
    (b"gmres", 2, "none"), (b"gmres", 2, "diag"),
]


@pytest.mark.parametrize("name,method,pc", SOLVER_CASES)
def test_solver_parity(b2s, ctx, orc, name, method, pc):
    n, rp, ci, v = P.poisson2d(48) if method == 0 else P.convdiff2d(48)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    b = b2s.uniform(11, n)
    kind = b2s.pc_kind_from_name(method, pc)
    M = b2s.Precond(ctx, A, kind) if kind != b2s.PC_NONE else None
    x, st = b2s.solve(ctx, A, b, method, M, tol=1e-8, maxit=3000, restart=20)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), method, pc, b, 1e-8, 3000, 20)
    assert st["status"] == 0
    assert abs(st["it"] - io) <= 2, (st["it"], io)
    assert st["relres_true"] < 1e-8 * 1.5
    assert rel(x, xo) < 1e-9, rel(x, xo)


def test_pcg_maxit_and_zero_rhs(b2s, ctx, orc):
    n, rp, ci, v = P.poisson2d(30)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    x, st = b2s.solve(ctx, A, np.zeros(n), b2s.PCG, None, tol=1e-8)
    assert st["it"] == 0 and not x.any()
    b = b2s.uniform(1, n)
    x, st = b2s.solve(ctx, A, b, b2s.PCG, None, tol=1e-12, maxit=5)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), 0, "none", b, 1e-12, 5)
    assert st["it"] == io == 4
    assert rel(x, xo) < 1e-12


def test_pcg_not_spd_raises(b2s, ctx):
    n, rp, ci, v = P.poisson2d(10)
    v = v.copy()
    rows = np.repeat(np.arange(n), np.diff(rp))
    v[(rows == ci) & (rows == 3)] = -4.0
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    with pytest.raises(RuntimeError):
        b2s.Precond(ctx, A, b2s.PC_DIAG)
    S = b2s.SMatrix(n, n, v, row_ptr=rp, col_idx=ci)
    with pytest.raises(RuntimeError):
        b2s.SMatrix.pcg(S, np.ones(n), "diag", 1e-8, 100)
    with pytest.raises(ValueError):
        b2s.SMatrix.pcg(S, np.ones(n + 1), "none")
    with pytest.raises(ValueError):
        b2s.SMatrix.pcg(S, np.ones(n), "bogus")


def test_smatrix_mirror(b2s, orc):
    n, rp, ci, v = P.poisson2d(25)
    rows = np.repeat(np.arange(n), np.diff(rp))
    S = b2s.SMatrix(n, n, v, rows, ci)
    assert np.array_equal(S.row_ptr(), rp) and np.array_equal(S.col_idx(), ci)
    b = b2s.uniform(2, n)
    x, it = b2s.SMatrix.pcg(S, b, "jacobi", 1e-8, 2000)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), 0, "jacobi", b, 1e-8, 2000)
    assert abs(it - io) <= 2 and rel(x, xo) < 1e-9
    assert np.array_equal(b2s.SMatrix.spmv(S, b), orc.spmv(orc.csr(n, n, rp, ci, v), b))


def test_block_gmres_bjacobi(b2s, ctx, orc):
    n, rp, ci, v = P.make_test_scalar(20, 3)
    Bo = orc.blk_condense(3, orc.csr(n, n, rp, ci, v), n // 3, n // 3)
    brp, bci, bv = Bo.export()
    B = b2s.BAIJ(ctx, 3, n // 3, n // 3, brp, bci, bv)
    b = 1.0 + 0.5 * P.drand(np.arange(n) + 7)
    M = b2s.Precond(ctx, B, b2s.PC_BJACOBI)
    x, st = b2s.solve(ctx, B, b, b2s.GMRES, M, tol=1e-8, maxit=500, restart=30)
    xo, io = orc.blk_gmres(Bo, b, "blockjacobi", 1e-8, 500, 30)
    assert abs(st["it"] - io) <= 2 and rel(x, xo) < 1e-9
    x2, st2 = b2s.solve(ctx, B, b, b2s.PCG, M, tol=1e-8, maxit=500)
    assert st2["relres_true"] < 1e-8 * 1.5


def test_host_preconditioner(b2s, ctx, orc):
    n, rp, ci, v = P.poisson2d(20)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    d = v[np.repeat(np.arange(n), np.diff(rp)) == ci]
    M = b2s.HostPrecond(ctx, n, lambda r: r / d)
    b = b2s.uniform(4, n)
    x, st = b2s.solve(ctx, A, b, b2s.GMRES, M, tol=1e-8, maxit=500, restart=10, use_graphs=0)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), 2, "diag", b, 1e-8, 500, 10)
    assert abs(st["it"] - io) <= 2 and rel(x, xo) < 1e-9


def test_graphs_match_eager(b2s, ctx):
    n, rp, ci, v = P.poisson2d(40)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    b = b2s.uniform(9, n)
    M = b2s.Precond(ctx, A, b2s.PC_DIAG)
    x1, s1 = b2s.solve(ctx, A, b, b2s.PCG, M, tol=1e-8, use_graphs=1, check_every=8)
    x2, s2 = b2s.solve(ctx, A, b, b2s.PCG, M, tol=1e-8, use_graphs=0, check_every=3)
    assert np.array_equal(x1, x2) and s1["it"] == s2["it"]


@pytest.mark.parametrize("flexible", [False, True])
def test_gmres_cgs2(b2s, ctx, orc, flexible):
    """Classical Gram-Schmidt twice is a different algorithm from the
    reference's MGS (the same Krylov space, other rounding), so it is held to
    accuracy, not to the reference's iterates: the same iteration count within
    +/-2, and an error against the FP64 solution (rtol 1e-13) no larger than
    twice the reference MGS solve's own error at the same tolerance."""
    n, rp, ci, v = P.convdiff2d(60)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    b = b2s.uniform(13, n)
    M = b2s.Precond(ctx, A, b2s.PC_ILU0)
    method = b2s.FGMRES if flexible else b2s.GMRES
    x, st = b2s.solve(ctx, A, b, method, M, tol=1e-8, maxit=2000, restart=30, orth=b2s.ORTH_CGS2)
    Ao = orc.csr(n, n, rp, ci, v)
    xo, io = orc.solve(Ao, 2, "ilu", b, 1e-8, 2000, 30)
    xt, _ = orc.solve(Ao, 2, "ilu", b, 1e-13, 2000, 30)
    assert abs(st["it"] - io) <= 2
    assert rel(x, xt) <= 2 * rel(xo, xt) + 1e-13, (rel(x, xt), rel(xo, xt))
    assert st["relres_true"] < 2e-8


def test_fgmres_fp32_refinement(b2s, ctx):
    """FP32 ILU(0) inside FP64 FGMRES with iterative refinement reaches 1e-10."""
    n, rp, ci, v = b2s.gen_convdiff3d(24)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    b = b2s.uniform(14, n)
    M = b2s.Precond(ctx, A, b2s.PC_ILU0, precision=b2s.FP32)
    x, st = b2s.solve(ctx, A, b, b2s.FGMRES, M, tol=1e-10, maxit=500, restart=30, ir_steps=5, ir_inner_tol=1e-6)
    assert st["relres_true"] < 1e-10
    r = b - A.spmv(x)
    assert np.linalg.norm(r) / np.linalg.norm(b) < 1e-10


def rect_random(n, m, density, seed):
    rng = np.random.default_rng(seed)
    dense = (rng.random((n, m)) < density) * rng.uniform(-1, 1, (n, m))
    rp = np.concatenate([[0], np.cumsum((dense != 0).sum(1))]).astype(np.uint32)
    return rp, np.nonzero(dense)[1].astype(np.uint32), dense[dense != 0]


@pytest.mark.parametrize("case", ["poisson_sq", "rect", "wide", "diag"])
def test_csr_matmul_transpose(b2s, ctx, orc, ref, case):
    """C = A B and A^T on the device (b2s_csr_matmul / b2s_csr_transpose) equal
    the restatement bit for bit: sorted columns, each entry summed in the
    reference's order.  Where every product column is touched by two or more
    rows the compiled reference gives the same arrays; "diag" is a product
    whose columns are each touched by one row, where the reference's marker
    array (not reset between its passes) drops them (tested on the CPU in
    test_oracle_pin.py::test_reference_spgemm_single_touch_defect)."""
    if case == "poisson_sq":
        n, rp, ci, v = P.poisson2d(40)
        a, b = (n, n, rp, ci, v), (n, n, rp, ci, v)
    elif case == "rect":
        a = (300, 500) + rect_random(300, 500, 0.02, 1)
        b = (500, 200) + rect_random(500, 200, 0.03, 2)
    elif case == "wide":  # product rows wider than the symbolic hash table (512 columns)
        a = (64, 64) + rect_random(64, 64, 0.5, 3)
        b = (64, 2000) + rect_random(64, 2000, 0.5, 4)
    else:
        n = 1000
        rp = np.arange(n + 1, dtype=np.uint32)
        d = np.linspace(1.0, 2.0, n)
        a = b = (n, n, rp, rp[:-1].copy(), d)
    A, B = b2s.CSR(ctx, *a), b2s.CSR(ctx, *b)
    C = A.matmul(B)
    Ao, Bo = orc.csr(*a), orc.csr(*b)
    Co = orc.matmul(Ao, Bo).export()
    assert np.array_equal(C.rp, Co[0]) and np.array_equal(C.ci, Co[1]) and np.array_equal(C.v, Co[2])
    if case != "diag":
        Cr = ref.matmul(ref.csr(*a), ref.csr(*b)).export()
        assert all(np.array_equal(x, y) for x, y in zip(Co, Cr))
    T = A.transpose()
    To = orc.transpose(Ao).export()
    assert (T.n, T.m) == (a[1], a[0])
    assert np.array_equal(T.rp, To[0]) and np.array_equal(T.ci, To[1]) and np.array_equal(T.v, To[2])
    Tr = ref.transpose(ref.csr(*a)).export()
    assert all(np.array_equal(x, y) for x, y in zip(To, Tr))
    # the product is a usable operator: its SpMV equals A (B x)
    x = np.random.default_rng(6).uniform(-1, 1, b[1])
    assert rel(C.spmv(x), A.spmv(B.spmv(x))) < 1e-13


@pytest.mark.parametrize("n,width", [(1, 1), (3, 40), (255, 16), (257, 17), (1000, 64), (40, 2048), (70, 6000)])
def test_baij1_long_rows(b2s, ctx, orc, n, width):
    """Scalar-block matvec with 16 and more entries a row: rows of no entry,
    of a whole pass of a CTA, of several; one row; CTAs of 256 rows."""
    rng = np.random.default_rng(n)
    m = max(n, 2 * width)
    lens = rng.integers(0, 2 * width, n)
    lens[-1] = 2 * width - 1
    lens[: n // 2 : 3] = 0
    lens[n // 2 :] = np.maximum(lens[n // 2 :], min(width + width // 2, m))
    cols = [np.sort(rng.choice(m, size=int(k), replace=False)) for k in lens]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    ci, v, x = np.concatenate(cols).astype(np.uint32), rng.uniform(-1, 1, int(rp[-1])), rng.uniform(-1, 1, m)
    y = b2s.BAIJ(ctx, 1, n, m, rp, ci, v).matvec(x)
    assert np.array_equal(y, orc.spmv(orc.csr(n, m, rp, ci, v), x))


@pytest.mark.parametrize("n", [1, 33, 1000, 60001])
def test_spmv_warp_groups(b2s, ctx, orc, n):
    """CSR product by groups of 32 rows: a last group of one row, empty rows
    and whole empty groups, rows longer than a warp's chunk, several groups a
    warp.  One row of 700 entries keeps the matrix off the row kernel."""
    rng = np.random.default_rng(n)
    m = max(n, 1024)
    lens = rng.integers(0, 12, n)
    lens[32 * 5 : 32 * 9] = 0
    lens[[0, -1]] = 700
    lens[n // 2] = 257
    cols = [np.sort(rng.choice(m, size=int(k), replace=False)) if k > 20 else np.unique(rng.integers(0, m, int(k)))
            for k in lens]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.uint32)
    ci, v, x = np.concatenate(cols).astype(np.uint32), rng.uniform(-1, 1, int(rp[-1])), rng.uniform(-1, 1, m)
    assert np.array_equal(b2s.CSR(ctx, n, m, rp, ci, v).spmv(x), orc.spmv(orc.csr(n, m, rp, ci, v), x))


@pytest.mark.parametrize("mean", [1, 8, 16, 40])
def test_csr_matmul_row_widths(b2s, ctx, orc, mean):
    """Product rows on both sides of every size of the symbolic hash table
    (32, 128, 256 and 512 columns), of one table filled to the last slot, and
    empty ones, for each group of lanes that walks a row of B."""
    widths = [0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 700]
    rng = np.random.default_rng(mean)
    nb, m = 1500, 1024
    cols = [np.sort(rng.choice(m, size=int(k), replace=False)) for k in rng.integers(0, 2 * mean + 1, nb)]
    brp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.uint32)
    b = (nb, m, brp, np.concatenate(cols).astype(np.uint32), rng.uniform(-1, 1, int(brp[-1])))
    rows = []
    for w in widths:  # rows of B until the product row has about w columns
        seen, row = set(), []
        for k in rng.permutation(nb):
            if len(seen | set(cols[k])) <= w and len(row) < 400:
                seen |= set(cols[k])
                row.append(k)
            if len(seen) == w:
                break
        rows.append(np.sort(np.array(row, np.int64)))
    arp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    a = (len(rows), nb, arp, np.concatenate(rows).astype(np.uint32), rng.uniform(-1, 1, int(arp[-1])))
    C = b2s.CSR(ctx, *a).matmul(b2s.CSR(ctx, *b))
    Co = orc.matmul(orc.csr(*a), orc.csr(*b)).export()
    assert np.array_equal(C.rp, Co[0]) and np.array_equal(C.ci, Co[1]) and np.array_equal(C.v, Co[2])


def test_csr_matmul_shape_error(b2s, ctx):
    n, rp, ci, v = P.poisson2d(8)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    B = b2s.CSR(ctx, 3, 3, np.zeros(4, np.uint32), np.zeros(0, np.uint32), np.zeros(0))
    with pytest.raises(b2s.B2SInvalidArgument):
        A.matmul(B)
    M = b2s.SMatrix(n, n, v, row_ptr=rp, col_idx=ci)
    with pytest.raises(ValueError):
        M * b2s.SMatrix(3, 3, np.zeros(0), row_ptr=np.zeros(4, np.uint32), col_idx=np.zeros(0, np.uint32))
    P2 = M * M
    assert P2.rows() == n and np.array_equal(M.transpose().col_idx(), ci)


@pytest.mark.parametrize("N,restart", [(1, 5), (2, 30), (7, 6), (8, 30), (31, 30), (97, 30)])
def test_gmres_orthogonalisation_sizes(b2s, ctx, orc, N, restart):
    """The one-launch Gram-Schmidt column at the sizes where it can go wrong: one
    row, fewer rows than a warp, an odd count (a slice's last pair half empty),
    a last CTA with fewer rows than the others, restarts.  GMRES and FGMRES
    against the restatement."""
    n, rp, ci, v = P.convdiff2d(N)
    A, b = b2s.CSR(ctx, n, n, rp, ci, v), b2s.uniform(N, n)
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), 2, "none", b, 1e-10, 2000, restart)
    for method in (b2s.GMRES, b2s.FGMRES):
        x, st = b2s.solve(ctx, A, b, method, None, tol=1e-10, maxit=2000, restart=restart)
        assert abs(st["it"] - io) <= 2 and st["relres_true"] < 1e-9
        # two solutions of relative residual 1e-10, condition numbers below 1e3 at these sizes
        assert np.linalg.norm(x - xo) <= 1e-7 * np.linalg.norm(xo)


@pytest.mark.parametrize("pc", ["none", "diag"])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (16, 16, 1), (257, 1, 1), (199, 190, 1), (41, 37, 29), (67, 64, 63)])
def test_pcg_one_launch_sizes(b2s, ctx, orc, pc, nx, ny, nz):
    """The one-launch PCG loop against the launch-by-launch one and the
    restatement: one row, exactly one CTA, one row more, one to four rows a
    thread, a last CTA with fewer rows."""
    if nz > 1:
        n, rp, ci, v = P.diffusion3d(nx, ny, nz, seed=nx)
    elif ny > 1:
        n, rp, ci, v = P.diffusion2d(nx, ny, seed=nx)
    else:  # a chain
        n, rp, ci, v = nx, *P.coo_to_csr(nx, nx, *zip(*[(i, j, 2.5 if i == j else -1.0) for i in range(nx)
                                                        for j in (i - 1, i, i + 1) if 0 <= j < nx]))
    A, b = b2s.CSR(ctx, n, n, rp, ci, v), b2s.uniform(nx + nz, n)
    M = b2s.Precond(ctx, A, b2s.PC_DIAG) if pc == "diag" else None
    got = [b2s.solve(ctx, A, b, b2s.PCG, M, tol=1e-8, maxit=5000, persistent=k) for k in (b2s.PERSIST_AUTO, b2s.PERSIST_OFF)]
    xo, io = orc.solve(orc.csr(n, n, rp, ci, v), 0, pc, b, 1e-8, 5000)
    for x, st in got:
        assert st["status"] == 0 and st["relres_true"] < 2e-8
        # iteration counts by the association of the dots alone; solutions of the same relative residual
        assert abs(st["it"] - io) <= max(2, io // 50)
        assert np.linalg.norm(x - xo) <= 1e-5 * np.linalg.norm(xo)


@pytest.mark.parametrize("loop", ["pcg", "pcg_diag", "pcg_tiles", "gmres", "fgmres"])
def test_persistent_wait_timeout_reported(b2s, ctx, loop):
    """The persistent kernels' CTAs wait for one another's sums a bounded number
    of polls.  With the bound cut to one poll the first sums of some 30 and more
    CTAs, which start microseconds apart, cannot all be there: the solve ends with
    B2S_TIMEOUT, at once (GMRES's host loop too, which goes on until the device
    says that a column is done), and with the default bounds the same solve gives
    the same bits as before."""
    import time
    N = 200
    if loop.startswith("pcg"):
        n, rp, ci, v = P.poisson2d(N)
    else:
        n, rp, ci, v = P.convdiff2d(N)
    A, b, M = b2s.CSR(ctx, n, n, rp, ci, v), b2s.uniform(5, n), None
    if loop == "pcg_diag":
        M = b2s.Precond(ctx, A, b2s.PC_DIAG)
    if loop == "pcg_tiles":
        M = b2s.Precond(ctx, A, b2s.PC_IC0, precision=b2s.FP32, trsv=b2s.TRSV_JACOBI, trsv_sweeps=6)
        assert M.sizes("pcg.tiles")[0] > 1
    method = {"gmres": b2s.GMRES, "fgmres": b2s.FGMRES}.get(loop, b2s.PCG)
    x0, _ = b2s.solve(ctx, A, b, method, M, tol=1e-3, maxit=2000)
    ctx.set_wait_limits(1, 0)
    try:
        t0 = time.perf_counter()
        with pytest.raises(RuntimeError) as e:
            b2s.solve(ctx, A, b, method, M, tol=1e-3, maxit=2000)
        dt = time.perf_counter() - t0
    finally:
        ctx.set_wait_limits(0, 0)
    assert e.value.status == b2s.TIMEOUT
    assert dt < 0.5, dt
    x, _ = b2s.solve(ctx, A, b, method, M, tol=1e-3, maxit=2000)
    assert np.array_equal(x, x0)


@pytest.mark.parametrize("bs", [2, 3, 4])
@pytest.mark.parametrize("where", ["first", "middle", "last", "hub", "hub_first"])
def test_baij_matvec_adjacent_long_rows(b2s, ctx, orc, bs, where):
    """Block matvec where rows dealt evenly would give a few warps most of the
    blocks, so that they are dealt by their blocks: long rows next to one another
    among short and empty ones, one row longer than all the rest; shares of no
    row, of one, of many."""
    n = 9001  # more rows than warps in a wave
    rng = np.random.default_rng(bs)
    lens = rng.integers(0, 4, n)
    lens[100:400] = 0
    at = {"first": 0, "middle": 4000, "last": n - 120}.get(where)
    if at is None:
        lens[0 if where == "hub_first" else n - 1] = 8000
    else:
        lens[at:at + 120] = rng.integers(200, 700, 120)
    cols = [np.sort(rng.choice(n, size=int(k), replace=False)) for k in lens]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint32)
    ci, v = np.concatenate(cols).astype(np.uint32), rng.uniform(-1, 1, int(rp[-1]) * bs * bs)
    x = rng.uniform(-1, 1, n * bs)
    y = b2s.BAIJ(ctx, bs, n, n, rp, ci, v).matvec(x)
    assert np.array_equal(y, orc.blk_matvec(orc.blk(bs, n, n, rp, ci, v), x))


@pytest.mark.parametrize("where", [0, 1500, 2999])
@pytest.mark.parametrize("columns", [33, 129, 257, 513])
def test_csr_matmul_one_wide_row(b2s, ctx, orc, where, columns):
    """A product of which one row alone does not fit the first table sizes, first,
    amid and last of 3,000: its counts stop the others' at whatever row they are."""
    n = 3000
    cols = [np.unique([i, (7 * i + 1) % n]) for i in range(n)]
    cols[where] = np.unique(np.concatenate([[where], np.arange(columns) * (n // columns)]))
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.uint32)
    a = (n, n, rp, np.concatenate(cols).astype(np.uint32), b2s.uniform(columns, int(rp[-1])))
    i = np.arange(n)
    b = (n, n, np.arange(n + 1, dtype=np.uint32), i.astype(np.uint32), 1.0 + b2s.uniform(1, n))
    for x, y in ((a, b), (a, a)):
        C = b2s.CSR(ctx, *x).matmul(b2s.CSR(ctx, *y))
        Co = orc.matmul(orc.csr(*x), orc.csr(*y)).export()
        assert np.array_equal(C.rp, Co[0]) and np.array_equal(C.ci, Co[1]) and np.array_equal(C.v, Co[2])


def test_pcg_wide_band_costs_no_launch(b2s, ctx):
    """An operator that the one-launch loop refuses for its band (2,500 of 2,048)
    is refused by what its handle knows: as many launches as with the loop off."""
    n, rp, ci, v = P.diffusion3d(50, 50, 30, seed=1)
    A, b = b2s.CSR(ctx, n, n, rp, ci, v), b2s.uniform(1, n)
    M = b2s.Precond(ctx, A, b2s.PC_DIAG)
    count = []
    for k in (b2s.PERSIST_AUTO, b2s.PERSIST_OFF):
        l0 = ctx.kernel_launches
        b2s.solve(ctx, A, b, b2s.PCG, M, tol=1e-8, maxit=16, persistent=k)
        count.append(ctx.kernel_launches - l0)
    assert count[0] == count[1]


def test_pcg_one_launch_on_a_product(b2s, ctx):
    """A device-built operator, whose band the first solve reads: the one-launch
    loop runs from the first solve on and gives the host-built operator's bits."""
    n, rp, ci, v = P.poisson2d(60)
    A = b2s.CSR(ctx, n, n, rp, ci, v)
    C = A.matmul(A)
    H, b = b2s.CSR(ctx, n, n, C.rp, C.ci, C.v), b2s.uniform(1, n)
    want, _ = b2s.solve(ctx, H, b, b2s.PCG, None, tol=1e-6, maxit=200)
    for _ in range(2):
        l0 = ctx.kernel_launches
        x, _ = b2s.solve(ctx, C, b, b2s.PCG, None, tol=1e-6, maxit=200)
        assert ctx.kernel_launches - l0 < 20
        assert np.array_equal(x, want)


@pytest.mark.parametrize("n", [1, 256, 257, 37889, 60001, 100003, 151553, 200001, 303105, 700001, 1000003, 1300001,
                               1700001, 1818624, 1818625])
def test_gmres_column_launch_bits(b2s, ctx, n):
    """The one-launch Gram-Schmidt column against a launch a step, bit for bit, over
    one to eight blocks a CTA (37,888 rows a block count on 148 SMs) and one to six
    elements a thread of each (303,104 rows), with odd remainders; one row more
    than the SMs hold keeps the launch a step."""
    rp = np.concatenate([[0], np.cumsum(np.full(n, 3) - (np.arange(n) == 0) - (np.arange(n) == n - 1))]).astype(np.uint32)
    i = np.arange(n)
    cols = i[:, None] + np.array([-1, 0, 1])
    keep = (cols >= 0) & (cols < n)
    v = np.where(cols == i[:, None], 2.5 + b2s.uniform(1, n)[:, None], np.array([-1.0, 0.0, -0.5]))[keep]
    A, b = b2s.CSR(ctx, n, n, rp, cols[keep].astype(np.uint32), v), b2s.uniform(2, n)
    got = []
    for k in (b2s.PERSIST_AUTO, b2s.PERSIST_OFF):
        l0 = ctx.kernel_launches
        x, st = b2s.solve(ctx, A, b, b2s.GMRES, None, tol=1e-14, maxit=9, restart=6, persistent=k)
        got.append((x, st["it"], st["relres"], ctx.kernel_launches - l0))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1:3] == got[1][1:3]
    assert got[0][3] < got[1][3] if n < 1818625 else got[0][3] == got[1][3]


@pytest.mark.parametrize("pc", ["none", "diag"])
@pytest.mark.parametrize("nx,ny,one", [(300, 300, True), (400, 333, True), (512, 512, True), (551, 550, True),
                                       (2048, 61, True), (2049, 61, False), (552, 552, False)])
def test_pcg_one_launch_rows_and_band(b2s, ctx, pc, nx, ny, one):
    """The one-launch PCG loop against the launch-by-launch one with two and four
    rows a thread (609 to 2,048 rows a CTA) and at both sides of its limits, a
    band of 2,048 and 2,048 rows a CTA.  The two differ by the association of the
    dots, some 1e-15 of them an iteration, which 40 iterations of these operators
    (conditions of 1e5 and below) cannot raise past 1e-9 of the iterate."""
    i = np.arange(nx * ny)
    n, rng = nx * ny, np.random.default_rng(nx)
    x_, y_ = i % nx, i // nx
    cx, cy = rng.uniform(0.5, 2.0, n), rng.uniform(0.5, 2.0, n)  # of (i, i + 1) and (i, i + nx)
    w, e = np.where(x_ > 0, np.roll(cx, 1), 0.0), np.where(x_ < nx - 1, cx, 0.0)
    s, t = np.where(y_ > 0, np.roll(cy, nx), 0.0), np.where(y_ < ny - 1, cy, 0.0)
    cols = i[:, None] + np.array([-nx, -1, 0, 1, nx])
    vals = np.stack([-s, -w, w + e + s + t + 0.1, -e, -t], 1)
    keep = vals != 0
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.uint32)
    A, b = b2s.CSR(ctx, n, n, rp, cols[keep].astype(np.uint32), vals[keep]), b2s.uniform(nx, n)
    M = b2s.Precond(ctx, A, b2s.PC_DIAG) if pc == "diag" else None
    got = []
    for k in (b2s.PERSIST_AUTO, b2s.PERSIST_OFF):
        l0 = ctx.kernel_launches
        x, st = b2s.solve(ctx, A, b, b2s.PCG, M, tol=1e-12, maxit=40, persistent=k)
        got.append((x, st, ctx.kernel_launches - l0))
    (x, st, l), (xr, sr, lr) = got
    assert (l < 20 < lr) if one else l == lr
    assert st["iterations"] == sr["iterations"] == 40
    assert np.linalg.norm(x - xr) <= 1e-9 * np.linalg.norm(xr)


@pytest.mark.parametrize("method", [0, 1])
def test_graph_replay_matches_eager(b2s, ctx, method):
    """Iterations captured and replayed against launched ones, for PCG with its
    one-launch loop off and for BiCGSTAB: the same bits."""
    n, rp, ci, v = P.poisson2d(40)
    A, b = b2s.CSR(ctx, n, n, rp, ci, v), b2s.uniform(9, n)
    M = b2s.Precond(ctx, A, b2s.PC_DIAG)
    o = dict(tol=1e-8, persistent=b2s.PERSIST_OFF)
    x1, s1 = b2s.solve(ctx, A, b, method, M, use_graphs=1, check_every=8, **o)
    x2, s2 = b2s.solve(ctx, A, b, method, M, use_graphs=0, check_every=3, **o)
    assert s1["it"] > 8 and s1["it"] == s2["it"] and np.array_equal(x1, x2)
