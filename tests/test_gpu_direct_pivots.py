"""The coarsest dense inverse takes its pivots in blocks of 32, every entry one
after another: the result of Gauss-Jordan with one pivot at a time, to the last
bit, also on ill-conditioned matrices that are not diagonally dominant."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gauss_jordan(A):
    D = A.copy()
    for k in range(len(D)):
        col = D[:, k].copy()
        row = D[k] * (1 / col[k])
        row[k] = 1 / col[k]
        D[:, k] = 0
        D -= np.outer(col, row)
        D[k] = row
    return D


# a block, its edges, several blocks and an update tile's edges
@pytest.mark.parametrize("n", [1, 7, 32, 33, 40, 64, 65, 100, 131])
@pytest.mark.parametrize("cond", [1e3, 1e9])
def test_inverse_is_that_of_single_pivots(n, cond, monkeypatch):
    import ml_prec_b200 as M
    monkeypatch.setenv("MLP_SMALL_BUDGET", "0")
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    D = (Q * np.logspace(0, -np.log10(cond), n)) @ Q.T
    D = (D + D.T) / 2
    ja = np.array([[i] + [j for j in range(n) if j != i] for i in range(n)])
    A = M.CSRMatrix.from_arrays(np.arange(n + 1) * n, ja.ravel(), np.take_along_axis(D, ja, 1).ravel())
    P = M.MultiSplitPrec(A, q=(0.8,), niter=(5,), max_levels=1, degree_max=2)
    assert P.nlevels == 1 and P.level(0)["direct"]
    got = np.stack([P.solve(e) for e in np.eye(n)], axis=1)  # a column: the other products are zeros
    np.testing.assert_array_equal(got, _gauss_jordan(D))
