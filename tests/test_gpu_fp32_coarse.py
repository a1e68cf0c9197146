"""The FP32-stored hierarchy keeps its coarse operator, however small, in FP64
with FP64 sums: as a launch of its own where a system sweeps above it, which in
the FP64 hierarchy a small operator does not need."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)


def test_small_coarse_operator_stays_fp64(monkeypatch):
    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    for var in ("MLP_PERSIST", "MLP_MERGE", "MLP_FOLD", "MLP_SMALL_BUDGET", "MLP_DENSE_OP_MAX"):
        monkeypatch.delenv(var, raising=False)
    A, _ = M.CSRMatrix.spe(60, 220, 20, *fields.field("iid", 2), c=1.0)
    f = np.random.default_rng(5).standard_normal(A.n)
    names, z = {}, {}
    for fp32 in (False, True):
        P = M.MultiSplitPrec(A, fp32=fp32, **MS)
        assert P.nlevels >= 3 and P.level_info(2)["N"] <= 32
        names[fp32] = [n for n, _, _ in P.profile(1)]
        z[fp32] = P.solve(f)
    assert any(n.startswith("sweep") for n in names[True])
    assert [n for n in names[True] if n != "dense L2"] == names[False]
    assert names[True].count("dense L2") == 1
    # a few FP32 roundings of 6e-8 a sweep
    assert np.linalg.norm(z[True] - z[False]) <= 1e-6 * np.linalg.norm(z[False])
