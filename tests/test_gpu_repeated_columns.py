"""Matrices whose rows hold a column more than once (assembled without summing
entries), the diagonal among them: marking takes such links one by one, as the
reference does, and the elimination adds them up, whichever kernel a row falls
to."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)


def _split(ia, ja, a, share, rng, diagonal=False):
    """Splits a share of the off-diagonal links in two or three, both ways
    alike, the parts anywhere among the row's links; with `diagonal` every fifth
    row's diagonal too."""
    rows = np.repeat(np.arange(len(ia) - 1), np.diff(ia))
    lo, hi = np.minimum(rows, ja).astype(np.uint64), np.maximum(rows, ja).astype(np.uint64)
    links, at = np.unique(lo * np.uint64(len(ia)) + hi, return_inverse=True)
    kind = np.where(rng.random(len(links)) < share, rng.integers(1, 3, len(links)), 0)[at]
    out_ia, out_ja, out_a = [0], [], []
    for i in range(len(ia) - 1):
        r = []
        for j in range(ia[i] + 1, ia[i + 1]):
            parts = ([1.0], [0.625, 0.375], [0.5, 0.3125, 0.1875])[kind[j]]
            r += [(ja[j], a[j] * p) for p in parts]
        diag = a[ia[i]]
        if diagonal and i % 5 == 0:
            r.append((i, -0.25 * diag))
            diag *= 1.25
        r = [r[k] for k in rng.permutation(len(r))]
        out_ja += [i] + [c for c, _ in r]
        out_a += [diag] + [v for _, v in r]
        out_ia.append(len(out_ja))
    return np.array(out_ia, np.uint32), np.array(out_ja, np.uint32), np.array(out_a)


def _sparse(csr, shape):
    ia, ja, a = csr
    return sp.csr_matrix((a, ja.astype(np.int64), ia.astype(np.int64)), shape=shape)  # repeated entries add up


def _close(x, y, rtol):
    d = abs(x - y)
    return d.nnz == 0 or d.max() <= rtol * abs(y).max()


def _check_solution(A, S, b, x, eps):
    """The recursive residual reaches eps of ||r0||; the true one stays within
    rounding of it."""
    import ml_prec_b200 as M
    r0 = np.linalg.norm(b - S @ M.api.generate_x0(A.n))
    scale = r0 * eps + A.n ** 0.5 * 2.0 ** -52 * abs(S).max() * np.abs(x).max() * 8
    assert np.linalg.norm(b - S @ x) <= 4 * scale


# rows by a warp, by groups of lanes and by threads; few and many repeats
@pytest.mark.parametrize("dims,c,share", [((8, 11, 5), 1.0, 0.5), ((16, 22, 8), 0.1, 0.02), ((16, 22, 8), 1.0, 0.5),
                                          ((30, 40, 20), 0.1, 0.2), ((59, 61, 29), 1.0, 0.2)])
def test_repeated_links(dims, c, share):
    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    from oracle import oracle as O
    Ao, b = O.assemble(*dims, *fields.field("layered", 9), c, True)
    arrays = _split(Ao.ia, Ao.ja, Ao.a, share, np.random.default_rng(3))
    Ao = O.Matrix(*arrays)
    A = M.CSRMatrix.from_arrays(*arrays)
    P, Po = M.MultiSplitPrec(A, **MS), O.Prec(Ao, "msplit", **MS)
    lv, lo = P.level(0), Po.level(0)
    for k in ("N", "nnz", "M", "Md"):
        assert lv[k] == lo[k], k
    np.testing.assert_array_equal(lv["map"], lo["map"])
    N, M_, R = lv["N"], lv["M"], lv["N"] - lv["Md"]
    # a factor entry is a sum of a few terms: 1e-13 of the largest entry
    assert _close(_sparse(lv["L"], (R, R)), _sparse(lo["L"], (R, R)), 1e-13)
    assert _close(_sparse(lv["U"], (M_, R)), _sparse(lo["U"], (M_, R)), 1e-13)
    n = R - M_
    l1, lo1 = P.level(1), Po.level(1)
    assert l1["N"] == lo1["N"] == n
    assert _close(_sparse(l1["A"], (n, n)), _sparse(lo1["A"], (n, n)), 1e-13)
    for l in range(P.nlevels):  # no column repeats in what the elimination leaves
        for k in ("L", "U"):
            m = P.level(l).get(k)
            if m is not None:
                rows = np.repeat(np.arange(len(m[0]) - 1), np.diff(m[0])).astype(np.uint64)
                key = rows * np.uint64(N) + m[1]
                assert len(np.unique(key)) == len(key)
    # a second build is the same, bit for bit
    f = np.random.default_rng(5).standard_normal(A.n)
    np.testing.assert_array_equal(P.solve(f), M.MultiSplitPrec(A, **MS).solve(f))
    _check_solution(A, _sparse(arrays, (A.n, A.n)), b, M.PCGSolver(A, b, P, eps=1e-10, flexible=True), 1e-10)


@pytest.mark.parametrize("dims,kw", [((8, 11, 5), {}), ((16, 22, 8), {}), ((30, 40, 20), {}),
                                     ((8, 11, 5), dict(max_levels=1)), ((16, 22, 8), dict(max_levels=2))])
def test_repeated_diagonal(dims, kw):
    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    from oracle import oracle as O
    Ao, b = O.assemble(*dims, *fields.field("iid", 3), 1.0, True)
    arrays = _split(Ao.ia, Ao.ja, Ao.a, 0.3, np.random.default_rng(3), diagonal=True)
    A = M.CSRMatrix.from_arrays(*arrays)
    P = M.MultiSplitPrec(A, **dict(MS, **kw))
    _check_solution(A, _sparse(arrays, (A.n, A.n)), b, M.PCGSolver(A, b, P, eps=1e-10, flexible=True), 1e-10)
