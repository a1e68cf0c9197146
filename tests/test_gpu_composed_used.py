"""Where the composed form is used: by the plan's launches, and on natural-order
vectors by the launches an application makes; and where its rows outgrow it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)
ENV = ("MLP_PERSIST", "MLP_MERGE", "MLP_FOLD", "MLP_SMALL_BUDGET", "MLP_DENSE_OP_MAX", "MLP_EXPLICIT")


def _names(P):
    return [n for n, _, _ in P.profile(1)]


@pytest.mark.parametrize("seed,dims,kw", [(4, (30, 60, 20), dict(ncheb=(2,))), (5, (41, 117, 23), dict(ncheb=(4, 2, 3))),
                                          (6, (16, 22, 8), dict(ncheb=(5,))), (6, (16, 22, 8), dict(ncheb=(1,))),
                                          (6, (30, 40, 20), dict(ncheb=(2,), sigma=(2.0,), use_tails=False))])
@pytest.mark.parametrize("fp32", [False, True])
def test_uh_cheb_plan(seed, dims, kw, fp32, monkeypatch):
    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    for var in ENV:
        monkeypatch.delenv(var, raising=False)
    A, _ = M.CSRMatrix.spe(*dims, *fields.field("layered", seed), c=1.0)
    kw = dict(dict(sigma=(3.0,)), **kw)
    P = M.Prec(A, fp32=fp32, **kw)
    monkeypatch.setenv("MLP_MERGE", "1")
    steps = _names(M.Prec(A, fp32=fp32, **kw))
    got = _names(P)
    assert P.nlevels > 1 and not any(n.startswith("sweep") for n in steps)
    # the finest level of at most 2,048 rows below level 0 is tabulated
    system = P.level_info(1)["N"] > 2048 and kw["ncheb"][0] > 1
    assert any(n.startswith("sweep") for n in got) == system
    if kw["ncheb"][0] > 1:
        assert len(got) < len(steps)


@pytest.mark.parametrize("dims,model,c,composed", [((12, 22, 6), "iid", 1.0, True), ((30, 40, 20), "layered", 0.1, True),
                                                   ((60, 220, 20), "iid", 1.0, True), ((30, 40, 20), "iid", 1.0, False)])
@pytest.mark.parametrize("fp32", [False, True])
def test_natural_order_launches(dims, model, c, composed, fp32, monkeypatch):
    """A composed plan makes its own launches and no copies; a step plan one
    copy before and one after."""
    import torch

    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    from ml_prec_b200._capi import check, lib
    for var in ENV:
        monkeypatch.delenv(var, raising=False)
    if not composed:
        monkeypatch.setenv("MLP_MERGE", "1")
    A, _ = M.CSRMatrix.spe(*dims, *fields.field(model, 2), c=c)
    P = M.MultiSplitPrec(A, fp32=fp32, **MS)
    f = torch.from_numpy(np.random.default_rng(5).standard_normal(A.n)).cuda()
    z = torch.empty_like(f)
    torch.cuda.synchronize()

    def count():
        n = C.c_uint64()
        check(lib().mlp_launch_count(C.byref(n)))
        return n.value

    per = len(_names(P))
    before = count()
    check(lib().mlp_prec_apply(P.h, C.c_void_p(f.data_ptr()), C.c_void_p(z.data_ptr()), None))
    assert count() - before == per + (0 if composed else 2)
    torch.cuda.synchronize()


# two chains of cells, nearly no reaction: with 2,500 cells the products' rows fit
# 1,024 entries, with 3,000 and less reaction they do not
@pytest.mark.parametrize("dims,c,composed", [((2500, 2, 1), 1e-4, True), ((3000, 2, 1), 1e-5, False)])
def test_rows_that_outgrow_the_products(dims, c, composed, monkeypatch):
    import ml_prec_b200 as M
    from ml_prec_b200.fields import KN
    for var in ENV:
        monkeypatch.delenv(var, raising=False)
    A, b = M.CSRMatrix.spe(*dims, *(np.ones(KN),) * 3, c=c)
    P = M.MultiSplitPrec(A, **MS)
    assert any(n.startswith("sweep") for n in _names(P)) == composed
    x = M.PCGSolver(A, b, P, eps=1e-10, flexible=True)
    ia, ja, a = A.arrays()
    rows = np.repeat(np.arange(A.n), np.diff(ia))

    def residual(v):
        r = b.copy()
        np.add.at(r, rows, -a * v[ja])
        return np.linalg.norm(r)

    # the recursive residual reaches 1e-10 of ||r0||; the true one stays within rounding of it
    scale = residual(M.api.generate_x0(A.n)) * 1e-10 + A.n ** 0.5 * 2.0 ** -52 * np.abs(a).max() * np.abs(x).max() * 8
    assert residual(x) <= 4 * scale
