"""Whole-solve parity: the GPU tree walk against the oracle and the golden KAT.

* the reference's known-answer test, generated on the device, against the
  committed dense solutions (tests/golden) and against the oracle;
* seeded Gaussian systems (balanced and unbalanced trees) against the
  oracle's fused FP64 solve, both node forms;
* the factor/solve split and the mixed-precision refined solve, whose
  relative residual must reach 1e-12;
* the FP64 HODLR matvec against the oracle's.
FP64 tolerance: 1e-12 relative (Frobenius), the reference's Err formula.
"""
import numpy as np
import pytest

from gpu_util import dev, host, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-12


def gpu_system(fs, s):
    h = fs.HodlrMatrix(s.m, s.N, int(s.tree[1, 1]) if s.tree.shape[0] > 1 else 1,
                       _threshold_of(s))
    h.create_tree()
    h.set_matrix(s.D, s.U if s.U.shape[1] else None, s.V if s.V.shape[1] else None)
    h.set_rhs(s.B)
    return h


def _threshold_of(s):
    return s.threshold


def make_gauss(oracle, N, m, r, t, seed):
    s = oracle.gaussian_system(N, m, r, t, seed=seed)
    s.threshold = t
    return s


@pytest.mark.parametrize("name", ["kat_n480", "kat_n201", "kat_n1000"])
def test_kat_on_device(fs, oracle, golden, cuda, name):
    g = golden(name)
    N, m, r, t = (int(g[k]) for k in ("N", "nrhs", "rank", "threshold"))
    h = fs.HodlrMatrix(m, N, r, t).create_tree()
    h.init_rhs(int(g["seed"]))
    h.init_circulant_matrix(float(g["diag"]))
    s = oracle.kat_system(N=N, nrhs=m, rank=r, threshold=t, diag=float(g["diag"]),
                          seed=int(g["seed"]))
    D, U, V, B = h.get_matrix()
    np.testing.assert_array_equal(B, g["B"])
    np.testing.assert_array_equal(D, s.D)
    np.testing.assert_array_equal(U, s.U)
    np.testing.assert_array_equal(V, s.V)
    fs.FastSolver().bfs_solve(h)
    x = h.solution()
    assert oracle.rel_error(x, g["X"]) < TOL           # the reference's Err vs dense
    Xo, _ = oracle.bfs_solve(s)
    assert relerr(x, Xo[:, :m]) < TOL                  # vs the restated HODLR walk


CASES = [(4096, 1, 30, 256), (4096, 8, 16, 300), (3001, 5, 12, 200), (777, 2, 8, 100),
         (20000, 4, 24, 512), (8192, 16, 64, 512), (65537, 3, 20, 1000)]


@pytest.mark.parametrize("N,m,r,t", CASES)
@pytest.mark.parametrize("schur2", [False, True])
def test_fused_fp64_vs_oracle(fs, oracle, cuda, N, m, r, t, schur2):
    s = make_gauss(oracle, N, m, r, t, seed=N + m)
    h = gpu_system(fs, s)
    fs.FastSolver().bfs_solve(h, schur2=schur2)
    x = h.solution()
    Xo, _ = oracle.bfs_solve(s, nthreads=8, schur2=schur2)
    assert relerr(x, Xo[:, :m]) < TOL
    assert oracle.relres(s, x) < 1e-13


@pytest.mark.parametrize("N,m,r,t", [(4096, 4, 16, 256), (20000, 3, 24, 512)])
def test_factor_then_solve_new_rhs(fs, oracle, cuda, N, m, r, t):
    s = make_gauss(oracle, N, m, r, t, seed=11)
    h = gpu_system(fs, s)
    solver = fs.FastSolver()
    solver.factor(h, fs.PREC_FP64)
    B2 = np.asfortranarray(np.random.default_rng(5).standard_normal((N, m)))
    h.set_rhs(B2)
    solver.solve(h)
    s.B = B2
    Xo, _ = oracle.bfs_solve(s, nthreads=8)
    assert relerr(h.solution(), Xo[:, :m]) < TOL


@pytest.mark.parametrize("N,m,r,t", [(4096, 1, 30, 256), (20000, 4, 24, 512),
                                     (65536, 8, 50, 512), (3001, 5, 12, 200)])
def test_mixed_refined_reaches_1e12(fs, oracle, cuda, N, m, r, t):
    s = make_gauss(oracle, N, m, r, t, seed=3 * N)
    h = gpu_system(fs, s)
    it, rr = fs.FastSolver().solve_refined(h, fs.PREC_MIXED, tol=1e-12, maxiter=10)
    assert rr <= 1e-12
    x = h.solution()
    assert oracle.relres(s, x) <= 2e-12   # the oracle's matvec agrees
    Xo, _ = oracle.bfs_solve(s, nthreads=8)
    assert relerr(x, Xo[:, :m]) < 1e-11   # forward error vs the FP64 oracle


def test_matvec_vs_oracle(fs, oracle, cuda):
    s = make_gauss(oracle, 9000, 6, 20, 300, seed=4)
    h = gpu_system(fs, s)
    import torch
    x = np.asfortranarray(np.random.default_rng(9).standard_normal((9000, 6)))
    y = torch.zeros((6, 9000), dtype=torch.float64, device="cuda").T
    h.matvec(dev(x), y)
    assert relerr(host(y), oracle.matvec(s, x)) < 1e-13


def test_gaussian_generator_distribution(fs, oracle, cuda):
    N, m, r, t = 4096, 2, 16, 256
    h = fs.HodlrMatrix(m, N, r, t).create_tree()
    h.init_gaussian(1234, 0.5)
    D, U, V, B = h.get_matrix()
    tree = h.tree_nodes()
    s = oracle.System(tree, D, U, V, B)
    A = s.dense()
    F = oracle.F
    for p in range(tree.shape[0]):
        if tree[p, F["is_leaf"]]:
            continue
        c0, c1 = tree[p, F["lchild"]], tree[p, F["rchild"]]
        rs0 = slice(tree[c0, 2], tree[c0, 2] + tree[c0, 0])
        rs1 = slice(tree[c1, 2], tree[c1, 2] + tree[c1, 0])
        assert abs(np.linalg.norm(A[rs0, rs1], 2) - 0.5) < 1e-6
    assert abs(B.mean()) < 0.05 and abs(B.std() - 1) < 0.05
    leaf = D[:256, :256]
    off = (leaf - 2 * np.eye(256)) * 16.0
    assert abs(off.std() - 1) < 0.02
    # and the generated system solves like any other
    fs.FastSolver().bfs_solve(h)
    Xo, _ = oracle.bfs_solve(s, nthreads=8)
    assert relerr(h.solution(), Xo[:, :m]) < TOL


def test_solve_before_factor_is_state_error(fs, cuda):
    h = fs.HodlrMatrix(1, 1000, 8, 100).create_tree()
    with pytest.raises(fs.HodlrError) as e:
        fs.FastSolver().solve(h)
    assert e.value.status == fs.ERR_STATE


def test_singular_leaf_reported(fs, oracle, cuda):
    s = make_gauss(oracle, 2000, 1, 8, 250, seed=1)
    s.D[300, :] = 0.0   # zero row in leaf 2 -> exact zero pivot
    h = gpu_system(fs, s)
    with pytest.raises(fs.HodlrError) as e:
        fs.FastSolver().bfs_solve(h)
    assert e.value.status > 0


def test_save_solution_reference_format(fs, cuda, tmp_path):
    h = fs.HodlrMatrix(2, 480, 30, 60, name=str(tmp_path / "global")).create_tree()
    h.init_rhs(1245667)
    h.init_circulant_matrix(1.0e4)
    fs.FastSolver().bfs_solve(h)
    h.save_solution()
    rows = open(h.file_soln).read().splitlines()
    assert len(rows) == 480
    vals = np.array([[float(v) for v in r.split("\t") if v] for r in rows])
    np.testing.assert_array_equal(vals, h.solution())


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_graph_replay_new_rhs(fs, oracle, cuda, precision):
    """On a side stream the refined solve is captured as CUDA graphs on its
    first call and replayed afterwards: a second right-hand side loaded into
    the same system must be solved as accurately as the first, and the fused
    FP64 solve replayed on a third one must match the oracle."""
    import torch
    N, m, r, t = 8192, 3, 20, 256
    s = make_gauss(oracle, N, m, r, t, seed=11)
    h = gpu_system(fs, s)
    prec = fs.PREC_MIXED if precision == "mixed" else fs.PREC_FP64
    st = torch.cuda.Stream()
    sol = fs.FastSolver()
    rng = np.random.default_rng(5)
    for trial in range(3):
        B = np.asfortranarray(rng.standard_normal((N, m)))
        h.set_rhs(B, stream=st)
        s.B = B
        it, rr = sol.solve_refined(h, prec, tol=1e-12, maxiter=10, stream=st)
        st.synchronize()
        assert rr <= 1e-12, (trial, rr)
        x = h.solution(stream=st)
        Xo, _ = oracle.bfs_solve(s, nthreads=8)
        assert relerr(x, Xo[:, :m]) < 1e-11
    for trial in range(2):
        B = np.asfortranarray(rng.standard_normal((N, m)))
        h.set_rhs(B, stream=st)
        s.B = B
        sol.bfs_solve(h, stream=st)
        st.synchronize()
        Xo, _ = oracle.bfs_solve(s, nthreads=8)
        assert relerr(h.solution(stream=st), Xo[:, :m]) < 1e-12


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_solve_refined_host_matches_device_path(fs, oracle, cuda, precision):
    """The host-to-host refined solve (inputs copied in, V's copy under the
    leaf factorization for the mixed path, the solution copied out) gives
    bit for bit the solution of the device-resident solve, from pinned
    tensors on a side stream and from pageable arrays on the legacy stream,
    and repeated calls replay it unchanged."""
    import torch
    N, m, r, t = 20000, 4, 40, 512
    s = make_gauss(oracle, N, m, r, t, seed=31)
    prec = fs.PREC_MIXED if precision == "mixed" else fs.PREC_FP64
    h = gpu_system(fs, s)
    it1, rr1 = fs.FastSolver().solve_refined(h, prec, tol=1e-12, maxiter=10)
    x1 = h.solution()
    assert rr1 <= 1e-12

    def pinned(a):  # column-major pinned CPU tensor
        return torch.from_numpy(np.ascontiguousarray(np.asfortranarray(a).T)).pin_memory().t()

    h2 = fs.HodlrMatrix(m, N, r, t).create_tree()
    st = torch.cuda.Stream()
    sol = fs.FastSolver()
    x2, it2, rr2 = sol.solve_refined_host(h2, pinned(s.D), pinned(s.U), pinned(s.V), pinned(s.B),
                                          precision=prec, stream=st)
    assert it2 == it1 and rr2 == rr1
    np.testing.assert_array_equal(x2, x1)
    for _ in range(2):
        x3, it3, _ = sol.solve_refined_host(h2, s.D, s.U, s.V, s.B, precision=prec)
        assert it3 == it1
        np.testing.assert_array_equal(x3, x1)
    Xo, _ = oracle.bfs_solve(s, nthreads=8)
    assert relerr(x1, Xo[:, :m]) < 1e-11


@pytest.mark.parametrize("n", [5, 20, 32, 33, 63, 100, 257, 511, 512, 513, 1024])
def test_leaf_panels_ties_and_zero_columns(fs, cuda, n):
    """The leaf panel LU at the edges of its sub-blocks, panels and threads, on
    matrices full of equal pivot candidates, and its INFO for a zero column."""
    rng = np.random.default_rng(n)
    A = rng.integers(-1, 2, (n, n)).astype(np.float64) + 3 * np.eye(n) * rng.choice([-1, 1], n)
    A = A[rng.permutation(n)]                    # pivots off the diagonal
    B = rng.standard_normal((n, 3))
    X = np.linalg.solve(A, B)
    h = fs.HodlrMatrix(3, n, 1, 1024).create_tree()
    h.set_matrix(A)
    h.set_rhs(B)
    solver = fs.FastSolver()
    solver.bfs_solve(h)
    cond = np.linalg.cond(A)
    # both solvers: backward error of a few n u, growth of partial pivoting included
    assert np.linalg.norm(h.solution() - X) <= 50 * n * cond * 2.0 ** -53 * np.linalg.norm(X)
    it, rr = solver.solve_refined(h, fs.PREC_MIXED, tol=1e-12, maxiter=30)
    assert rr <= 1e-12
    j = int(rng.integers(0, n))
    A[:, j] = 0.0
    h.set_matrix(A)
    for call in (lambda: solver.bfs_solve(h), lambda: solver.factor(h, fs.PREC_MIXED)):
        with pytest.raises(fs.HodlrError) as e:
            call()
        assert e.value.status == j + 1


@pytest.mark.parametrize("m", [1, 8, 9, 17, 32, 40])
@pytest.mark.parametrize("n", [3, 16, 17, 33, 64, 130, 255, 500, 512, 513, 700, 1024])
def test_leaf_apply_edges(fs, cuda, n, m):
    """Kept leaf factors applied to new right-hand sides, at the edges of the
    panels, tiles and column chunks, FP64 and FP32."""
    rng = np.random.default_rng(100 * n + m)
    A = rng.standard_normal((n, n)) / np.sqrt(n) + 2 * np.eye(n)
    A = A[rng.permutation(n)]
    h = fs.HodlrMatrix(m, n, 1, 1024).create_tree()
    h.set_matrix(A)
    h.set_rhs(rng.standard_normal((n, m)))
    solver = fs.FastSolver()
    cond = np.linalg.cond(A)
    for prec, u in ((fs.PREC_FP64, 2.0 ** -53), (fs.PREC_MIXED, 2.0 ** -15)):
        # FP32 factors carry the split-BF16 updates' 2^-15 per product
        solver.factor(h, prec)
        B = rng.standard_normal((n, m))
        h.set_rhs(B)
        solver.solve(h)
        X = np.linalg.solve(A, B)
        lim = (50 * n if prec == fs.PREC_FP64 else 8) * cond * u
        assert np.linalg.norm(h.solution() - X) <= lim * np.linalg.norm(X)


@pytest.mark.parametrize("ob64", [64, 128])
@pytest.mark.parametrize("n", [15, 16, 17, 33, 64, 65, 100, 127, 128, 129, 177, 241, 300])
def test_fp64_block_row_solves_edges(fs, cuda, n, ob64):
    """The triangular products of the two-level FP64 leaf LU, whose zero half
    is left out by 16-row fragments, at the remainders of blocks and fragments."""
    rng = np.random.default_rng(10 * n + ob64)
    A = rng.standard_normal((n, n)) / np.sqrt(n) + 2 * np.eye(n)
    A = A[rng.permutation(n)]
    B = rng.standard_normal((n, 40))
    h = fs.HodlrMatrix(40, n, 1, 1024).create_tree()
    h.schedule = dict(leaf_ob64=ob64)
    h.set_matrix(A)
    h.set_rhs(B)
    fs.FastSolver().bfs_solve(h)
    X = np.linalg.solve(A, B)
    lim = 50 * n * np.linalg.cond(A) * 2.0 ** -53
    assert np.linalg.norm(h.solution() - X) <= lim * np.linalg.norm(X)


def _gepp(A):
    """(L, U, row order) of Gaussian elimination with partial pivoting."""
    A, n = A.copy(), A.shape[0]
    p = np.arange(n)
    for k in range(n):
        j = k + int(np.argmax(np.abs(A[k:, k])))
        A[[k, j]], p[[k, j]] = A[[j, k]], p[[j, k]]
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    return np.tril(A, -1) + np.eye(n), np.triu(A), p


def _smooth_kernel(n, s, shift):
    x = np.linspace(0, 1, n)
    return np.exp(-((x[:, None] - x) / s) ** 2) + shift * np.eye(n)


@pytest.mark.parametrize("prec,n,s,shift", [("fp64", 32, 0.1, 1e-8), ("fp64", 32, 0.2, 1e-8),
                                            ("fp64", 32, 0.3, 1e-8), ("mixed", 48, 0.1, 1e-6),
                                            ("mixed", 64, 0.1, 1e-7), ("mixed", 64, 0.05, 1e-7)])
def test_panel_inverse_residual(fs, cuda, prec, n, s, shift):
    """Kept factors of one panel whose triangles are ill-conditioned: the explicit
    inverses Y of the triangles T have |T Y - I| <= n u |T| |Y|, so that a solve
    with them leaves the residual below, where inverses whose error grows with
    the square of the condition number do not."""
    u, prec = (2.0 ** -53, fs.PREC_FP64) if prec == "fp64" else (2.0 ** -24, fs.PREC_MIXED)
    dt = np.float64 if prec == fs.PREC_FP64 else np.float32
    A = _smooth_kernel(n, s, shift).astype(dt).astype(np.float64)
    B = np.random.default_rng(n).standard_normal((n, 4)).astype(dt).astype(np.float64)
    h = fs.HodlrMatrix(4, n, 1, 1024).create_tree()
    h.set_matrix(A)
    h.set_rhs(B)
    solver = fs.FastSolver()
    solver.factor(h, prec)
    solver.solve(h)
    L, U, p = _gepp(A)
    a = np.abs
    w = a(np.linalg.inv(L)) @ a(B[p])
    # |b - L y| <= 2 n u |L| |Y_L| |b|, likewise for U, and L U = P A + n u |L| |U|
    lim = n * u * (2 * a(L) @ w + 3 * a(L) @ (a(U) @ (a(np.linalg.inv(U)) @ w)))
    r = a((B - A.astype(np.longdouble) @ h.solution()).astype(np.float64))[p]
    assert (r <= lim).all()


@pytest.mark.parametrize("call", ["leaf", 0, 16, 128, 256])
@pytest.mark.parametrize("n,s", [(17, 0.5), (31, 0.3), (33, 0.3), (100, 0.1), (128, 0.1), (129, 0.1),
                                 (257, 0.1), (512, 0.02), (512, 0.1), (513, 0.1), (1000, 0.1)])
def test_ill_conditioned_leaf_residual(fs, cuda, call, n, s):
    """A leaf of a smooth kernel, as the leaf task body and as a whole solve (by
    its outer block width): triangles with max|T| max|T^{-1}| above 2^7 are
    solved by substitution, so the residual is that of the factors plus what
    the inverses of the others leave."""
    A = _smooth_kernel(n, s, 1e-12)
    B = np.random.default_rng(n).standard_normal((n, 70))
    order = 32 if n <= 512 else 16
    if call == "leaf":
        D, X = dev(A, n + 1), dev(B, n + 3)
        import torch
        assert fs.leaf_solve(D, X, torch.zeros(n, dtype=torch.int32, device="cuda")) == 0
        x = host(X)
    else:
        h = fs.HodlrMatrix(70, n, 1, 1024).create_tree()
        h.schedule = dict(leaf_ob64=call)
        h.set_matrix(A)
        h.set_rhs(B)
        fs.FastSolver().bfs_solve(h)
        x = h.solution()
    if call == 128 or (n > 512 and call != 16):
        order = 128
    L, U, p = _gepp(A)
    # per triangle |b - T x| <= 2 n u |T| |Y| |T| |x| with (|T| |Y|)_ij <= 2^7 order
    lim = n * 2.0 ** -53 * (3 + 2 * 2 ** 7 * order ** 1.5) * np.linalg.norm(
        np.abs(L) @ (np.abs(U) @ np.abs(x)), axis=0)
    r = np.linalg.norm((B - A.astype(np.longdouble) @ x).astype(np.float64), axis=0)
    assert (r <= lim).all()


def test_block_inverse_memory(fs, cuda):
    """The outer blocks' inverses take one block of 128 columns per leaf where that
    is over 32 MB (256 leaves), and both node forms use the same leaf buffers."""
    import torch
    r, leaf, used = 8, 512, []
    # (the small systems first: code is loaded at a kernel's first launch)
    for N, ob in ((2048, 16), (2048, 128), (131072, 16), (131072, 128)):
        h = fs.HodlrMatrix(1, N, r, leaf).create_tree()
        h.schedule = dict(leaf_ob64=ob)
        D = torch.zeros((leaf, N), dtype=torch.float64, device="cuda").T
        at = torch.arange(N, device="cuda")
        D[at, at % leaf] = 2.0
        h.set_matrix(D, *(torch.zeros((r * h.max_depth, N), dtype=torch.float64, device="cuda").T
                          for _ in range(2)))
        h.set_rhs(torch.ones((1, N), dtype=torch.float64, device="cuda").T)
        del D
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        fs.FastSolver().bfs_solve(h)
        used.append(before - torch.cuda.mem_get_info()[0])
        np.testing.assert_array_equal(h.solution(), 0.5)
        cols = h.ncols
        del h
    slack = 16 << 20  # descriptors, node blocks, V^T products, the allocator's granularity
    assert used[3] - used[2] <= 8 * N // leaf * 128 * 128 + slack
    # X, the factors, Y and row orders and, once, the panels' inverses (2 x 32 columns)
    assert used[2] <= 8 * N * (cols + leaf + 64 + 2) + slack


@pytest.mark.parametrize("r", [104, 105, 144])
def test_mixed_large_ranks(fs, oracle, cuda, r):
    """The mixed node factorization on both sides of the rank up to which the V^T u
    blocks are staged in shared memory, and at the largest rank."""
    s = make_gauss(oracle, 1500, 3, r, 400, seed=r)
    h = gpu_system(fs, s)
    it, rr = fs.FastSolver().solve_refined(h, fs.PREC_MIXED, tol=1e-12, maxiter=10)
    assert rr <= 1e-12
    X, _ = oracle.bfs_solve(s, nthreads=8)
    assert relerr(h.solution(), X[:, :3]) < 1e-11
