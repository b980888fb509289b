"""The kernels' forms at the sizes where one gives way to another, and at the
edges of their tiles, against numpy or the CPU oracle.

Tolerances.  A product: each entry within 2 (K + 4) eps (|alpha| |A| |B| + |beta|
|C|), the bound of a K-term FP64 sum in any order, for both sides.  Solves and
factorizations: the scaled residuals of tests/test_gpu_parity.py (<= 4).  A
triangular solve multiplies by inverted diagonal blocks, so its residual may
grow with the blocks' condition: T = 2 I + N / n with |N| <= 1 has |T| |T^-1| <= 3
in the 1-norm, and the bound 4 is taken times 3.
"""
import numpy as np
import pytest

import elemental_b200 as eg
from elemental_b200 import inputs
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def cuda(a):
    return eg.colmajor_cuda(a)


def host(t):
    return np.asfortranarray(t.cpu().numpy())


def solve_bwd(A, X, B):
    return np.linalg.norm(A @ X - B, 1) / (np.linalg.norm(A, 1) * np.linalg.norm(X, 1) * A.shape[0] * EPS)


# small products (K <= 256), the eight-warp engine, its long-k form (K >= 1024, many tiles)
@pytest.mark.parametrize("mnk", [(31, 33, 1), (32, 32, 7), (33, 65, 129), (130, 18, 256), (130, 18, 258),
                                 (1201, 1203, 17), (1290, 1282, 130), (3100, 3102, 1027)])
@pytest.mark.parametrize("oa", [eg.NORMAL, eg.TRANSPOSE])
@pytest.mark.parametrize("ob", [eg.NORMAL, eg.TRANSPOSE])
def test_product_forms(handle, oa, ob, mnk):
    m, n, k = mnk
    A = inputs.uniform(*((m, k) if oa == eg.NORMAL else (k, m)), 1)
    B = inputs.uniform(*((k, n) if ob == eg.NORMAL else (n, k)), 2)
    C = inputs.uniform(m, n, 3)
    dC = cuda(C)
    handle.gemm(oa, ob, -0.5, cuda(A), cuda(B), 2.0, dC)
    a, b = (A if oa == eg.NORMAL else A.T), (B if ob == eg.NORMAL else B.T)
    ref = -0.5 * (a @ b) + 2.0 * C
    bound = 2 * (k + 4) * EPS * (0.5 * (np.abs(a) @ np.abs(b)) + 2.0 * np.abs(C))
    assert (np.abs(host(dC) - ref) <= bound).all()


@pytest.mark.parametrize("uplo", [eg.LOWER, eg.UPPER])
@pytest.mark.parametrize("nk", [(33, 5), (1250, 129), (2300, 300)])
def test_rank_k_forms_leave_the_other_triangle(handle, uplo, nk):
    n, k = nk
    A, C = inputs.uniform(n, k, 4), inputs.uniform(n, n, 5)
    dC = cuda(C)
    handle.herk(uplo, eg.NORMAL, 1.0, cuda(A), 1.0, dC)
    own = np.tril(np.ones((n, n), dtype=bool)) if uplo == eg.LOWER else np.triu(np.ones((n, n), dtype=bool))
    got = host(dC)
    bound = 2 * (k + 4) * EPS * (np.abs(A) @ np.abs(A).T + np.abs(C))
    assert (np.abs(got - (A @ A.T + C)) <= bound)[own].all()
    assert np.array_equal(got[~own], C[~own])


def test_product_into_rows_below_its_operand(handle):
    """C and B are row blocks of one matrix: they interleave in memory and share nothing."""
    k, m, n = 64, 90, 70
    G, A = inputs.uniform(k + m, n, 6), inputs.uniform(m, k, 7)
    dG = cuda(G)
    handle.gemm(eg.NORMAL, eg.NORMAL, -1.0, cuda(A), dG[:k], 1.0, dG[k:])
    got = host(dG)
    bound = 2 * (k + 4) * EPS * (np.abs(A) @ np.abs(G[:k]) + np.abs(G[k:]))
    assert np.array_equal(got[:k], G[:k])
    assert (np.abs(got[k:] - (G[k:] - A @ G[:k])) <= bound).all()


# in-place multiplies by an inverted block: 16 or 32 rows (columns) per CTA, then the engine
@pytest.mark.parametrize("other", [2368, 2369, 4736, 4737])
@pytest.mark.parametrize("side", [eg.LEFT, eg.RIGHT])
def test_triangular_solve_across_in_place_forms(handle, side, other):
    nt = 131
    T = np.asfortranarray(np.tril(inputs.uniform(nt, nt, 8) / nt, -1) + 2.0 * np.eye(nt))
    B = inputs.uniform(*((nt, other) if side == eg.LEFT else (other, nt)), 9)
    dB = cuda(B)
    handle.trsm(side, eg.LOWER, eg.NORMAL, eg.NON_UNIT, 1.0, cuda(T), dB)
    X = host(dB)
    R = (T @ X if side == eg.LEFT else X @ T) - B
    assert np.linalg.norm(R, 1) <= 4 * 3 * nt * EPS * np.linalg.norm(T, 1) * np.linalg.norm(X, 1)


# rows per thread and per CTA of the LU panel change at 128, 2048, 4096, 8192
@pytest.mark.parametrize("m", [33, 127, 128, 129, 2048, 2049, 4096, 4097, 8193, 16384])
def test_lu_panel_heights(handle, m):
    n = 33  # two whole sub-panels and one column
    A = inputs.uniform(m, n, 10)
    dA = cuda(A)
    import torch
    p = torch.zeros(n, dtype=torch.int32, device="cuda")
    handle.lu(dA, p)
    ref, pref, st = orc.lu(A, nb=128)
    assert st == 0
    assert np.array_equal(p.cpu().numpy(), pref)
    assert np.abs(host(dA) - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("m", [5, 64, 300, 2500, 9000])
def test_lu_panel_ties_take_the_lowest_row(handle, m):
    """Entries +-1: many rows tie in every column, and three columns stay exact."""
    import torch
    A = np.asfortranarray(np.sign(inputs.uniform(m, 3, 11)))
    dA = cuda(A)
    p = torch.zeros(3, dtype=torch.int32, device="cuda")
    handle.lu(dA, p)
    ref, pref, st = orc.lu(A, nb=128)
    assert st == 0
    assert np.array_equal(p.cpu().numpy(), pref)
    assert np.array_equal(host(dA), ref)


@pytest.mark.parametrize("col", [1, 2, 15, 16, 17, 18, 33, 128, 129, 145])
def test_cholesky_reports_the_failing_column(handle, col):
    n = 145
    A = inputs.spd_ggt(n, 12)
    A[col - 1, col - 1] = -1.0
    with pytest.raises(eg.NonHPDError) as e:
        handle.cholesky(cuda(A), eg.LOWER)
    assert e.value.column == col


@pytest.mark.parametrize("n", [15, 16, 17, 31, 33, 113])
@pytest.mark.parametrize("uplo", [eg.LOWER, eg.UPPER])
def test_cholesky_leaf_edges(handle, n, uplo):
    A = inputs.spd_ggt(n, 13)
    dA = cuda(A)
    handle.cholesky(dA, uplo)
    F = host(dA)
    L = np.tril(F) if uplo == eg.LOWER else np.triu(F).T
    assert np.linalg.norm(A - L @ L.T, 1) <= 4 * n * EPS * np.linalg.norm(A, 1)


# right-hand sides in groups of 8, and of 16 (82 block rows of 16 at 64 columns)
@pytest.mark.parametrize("nrhs", [8, 9, 16, 17, 63, 64])
@pytest.mark.parametrize("n,nb", [(131, 128), (700, 128), (1301, 16)])
@pytest.mark.parametrize("uplo", [eg.LOWER, eg.UPPER])
def test_solve_sweeps_in_groups(handle, uplo, n, nb, nrhs):
    A, B = inputs.spd_ggt(n, 14), inputs.normal(n, nrhs, 15)
    ld = n + (n & 1)
    old = handle.blocksize()
    handle.set_blocksize(nb)
    try:
        dA, dB = eg.empty_colmajor(n, n, ld=ld), eg.empty_colmajor(n, nrhs, ld=ld)
        dA.copy_(cuda(A))
        dB.copy_(cuda(B))
        handle.hpd_solve(dA, dB, uplo=uplo)
    finally:
        handle.set_blocksize(old)
    assert solve_bwd(A, host(dB), B) <= 4


@pytest.mark.parametrize("nrhs", [1, 8, 64, 65])
@pytest.mark.parametrize("n", [130, 331])
def test_gaussian_elimination_routes(handle, n, nrhs):
    A, B = inputs.uniform(n, n, 16), inputs.normal(n, nrhs, 17)
    dA, dB = cuda(A), cuda(B)
    handle.gaussian_elimination(dA, dB)
    assert solve_bwd(A, host(dB), B) <= 4


def tiny_block(n, rows, cols):
    """I + 2^-55 in a block: a row's products with x = 1 vanish against 1 one by
    one (half an ulp below 1 is 2^-54), their sum of w 2^-55 does not."""
    A = np.eye(n)
    A[rows, cols] = 2.0 ** -55
    return np.asfortranarray(A)


@pytest.mark.parametrize("nrhs", [1, 16, 64])
def test_last_solve_sums_a_block_before_it_meets_b(handle, nrhs):
    A = tiny_block(256, slice(0, 128), slice(128, 256))
    dB = cuda(np.ones((256, nrhs), order="F"))
    handle.gaussian_elimination(cuda(A), dB)
    assert (host(dB)[:128] == 1.0 - 2.0 ** -48).all() and (host(dB)[128:] == 1.0).all()


@pytest.mark.parametrize("n", [7, 100, 257])
def test_cholesky_of_a_diagonal_matrix_is_its_roots(handle, n):
    d = np.abs(inputs.normal(n, 1, 25))[:, 0] + 0.01
    A = np.asfortranarray(np.diag(d))
    for batched in (False, True):
        dA, dB = cuda(A), cuda(np.ones((n, 1), order="F"))
        if batched:
            assert handle.hpd_solve_batched([dA], [dB]) == [0]
        else:
            handle.hpd_solve(dA, dB)
        assert np.array_equal(np.tril(host(dA)), np.diag(np.sqrt(d)))


# an infinite pivot: its root, zeros below it, and the others' solution with x = 0 there
@pytest.mark.parametrize("n,at", [(40, 7), (40, 39), (100, 16), (300, 150)])
def test_batched_hpd_infinite_diagonal_entry(handle, n, at):
    A, B = inputs.spd_ggt(n, 26), inputs.normal(n, 2, 27)
    G = A.copy(order="F")
    G[at, at] = np.inf
    dA, dB = cuda(G), cuda(B)
    assert handle.hpd_solve_batched([dA], [dB]) == [0]
    L, X = np.tril(host(dA)), host(dB)
    assert L[at, at] == np.inf and (L[at + 1:, at] == 0.0).all()
    assert (X[at] == 0.0).all()
    keep = np.arange(n) != at
    assert solve_bwd(A[np.ix_(keep, keep)], X[keep], B[keep]) <= 4


# products of 32 columns (16-column panels: two sums) right of or left of the diagonal
@pytest.mark.parametrize("n", [64, 320])
@pytest.mark.parametrize("lower", [False, True])
def test_batched_solve_sums_a_block_before_it_meets_b(handle, lower, n):
    first, last = slice(0, 32), slice(n - 32, n)
    A = tiny_block(n, last, first) if lower else tiny_block(n, first, last)
    dB = [cuda(np.ones((n, 3), order="F"))]
    assert handle.gaussian_elimination_batched([cuda(A)], dB) == [0]
    want = np.ones((n, 3))
    want[last if lower else first] = 1.0 - 2.0 ** -50
    assert np.array_equal(host(dB[0]), want)


# block sizes that the one-launch sweeps do not take, and the smallest that they do
@pytest.mark.parametrize("nb", [2, 6, 8])
@pytest.mark.parametrize("n,nrhs", [(20, 3), (50, 64)])
def test_solves_with_small_block_sizes(handle, n, nrhs, nb):
    import torch
    A, S, B = inputs.uniform(n, n, 22), inputs.spd_ggt(n, 23), inputs.normal(n, nrhs, 24)
    old = handle.blocksize()
    handle.set_blocksize(nb)
    try:
        dX, dY, dZ, dF, p = cuda(B), cuda(B), cuda(B), cuda(A), torch.zeros(n, dtype=torch.int32, device="cuda")
        handle.gaussian_elimination(cuda(A), dX)
        handle.hpd_solve(cuda(S), dY)
        handle.lu(dF, p)
        handle.lu_solve_after(dF, p, dZ)
    finally:
        handle.set_blocksize(old)
    assert solve_bwd(A, host(dX), B) <= 4
    assert solve_bwd(S, host(dY), B) <= 4
    assert solve_bwd(A, host(dZ), B) <= 4


# the shapes change with the largest order; block edges at multiples of 16 and 32
@pytest.mark.parametrize("sizes", [(1, 2, 15, 16, 17, 31, 32, 33, 47, 64, 255, 256), (48, 257, 300, 511, 512)])
def test_batched_block_edges(handle, sizes):
    nr = [1 + (5 * i) % 9 for i in range(len(sizes))]
    for hpd in (True, False):
        As = [inputs.spd_ggt(n, 20 + n) if hpd else inputs.uniform(n, n, 20 + n) for n in sizes]
        Bs = [inputs.normal(n, k, 40 + n) for n, k in zip(sizes, nr)]
        dA, dB = [cuda(a) for a in As], [cuda(b) for b in Bs]
        info = (handle.hpd_solve_batched if hpd else handle.gaussian_elimination_batched)(dA, dB)
        assert info == [0] * len(sizes)
        for a, b, x in zip(As, Bs, dB):
            assert solve_bwd(a, host(x), b) <= 4


@pytest.mark.parametrize("panel,threads", [(32, 256), (16, 256), (16, 128)])
@pytest.mark.parametrize("kind", [0, 1])
def test_batched_block_edges_in_every_shape(handle, kind, panel, threads):
    sizes = (1, 15, 16, 17, 31, 32, 33, 64, 257, 300, 512)
    As = [inputs.spd_ggt(n, 60 + n) if kind == 0 else inputs.uniform(n, n, 60 + n) for n in sizes]
    Bs = [inputs.normal(n, 1 + i % 9, 80 + n) for i, n in enumerate(sizes)]
    dA, dB = [cuda(a) for a in As], [cuda(b) for b in Bs]
    plan = eg.BatchPlan(handle, kind, dA, dB)
    plan.set_shape(panel, threads)
    plan.run()
    assert plan.info() == [0] * len(sizes)
    for a, b, x in zip(As, Bs, dB):
        assert solve_bwd(a, host(x), b) <= 4
    plan.close()


def test_batched_lu_ties_and_singular_column(handle):
    A = np.asfortranarray(np.sign(inputs.uniform(40, 40, 18)))
    Z = inputs.uniform(40, 40, 19)
    Z[:, 35] = 0.0
    dA = [cuda(A), cuda(Z)]
    B = inputs.normal(40, 1, 21)
    dB = [cuda(B), cuda(B)]
    info = handle.gaussian_elimination_batched(dA, dB)
    assert info == [0, 36]
    assert solve_bwd(A, host(dB[0]), B) <= 4
