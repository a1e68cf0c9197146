"""autotune: the step plan with timed launch shapes and the composed plan are
both made and timed at the first build of a shape, and the faster one is kept;
a tuned step plan is the same operator as the untuned one."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)
ENV = ("MLP_PERSIST", "MLP_MERGE", "MLP_FOLD", "MLP_SMALL_BUDGET", "MLP_DENSE_OP_MAX")

CHILD = """
import sys
import ml_prec_b200 as M
from ml_prec_b200 import fields
kind, fp32 = sys.argv[1], sys.argv[2] == "1"
A, b = M.CSRMatrix.spe(30, 40, 20, *fields.field("layered", 9), c=0.1)
for k in range(2):
    if kind == "cheb":
        P = M.Prec(A, sigma=(3.0,), ncheb=(4,), fp32=fp32, autotune=True)
    else:
        P = M.MultiSplitPrec(A, fp32=fp32, autotune=True, q=(0.8,), niter=(5,), max_levels=15, degree_max=2)
    print("SWEEPS", int(any(n.startswith("sweep") for n, _, _ in P.profile(1))))
"""


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("kind", ["msplit", "cheb"])
def test_faster_plan_is_kept(kind, fp32):
    env = {k: v for k, v in os.environ.items() if not k.startswith("MLP_")}
    r = subprocess.run([sys.executable, "-c", CHILD, kind, str(int(fp32))], cwd=ROOT, env=dict(env, MLP_TRACE="1"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    timed = re.findall(r"autotune: composed ([\d.]+) us, steps ([\d.]+) us", r.stderr)
    assert len(timed) == 1  # the second build remembers
    want = float(timed[0][0]) <= float(timed[0][1])
    assert re.findall(r"SWEEPS (\d)", r.stdout) == [str(int(want))] * 2


# row kernels alone, and with the tile kernels among the candidates (levels above 131,072 rows)
@pytest.mark.parametrize("model,dims,c", [("layered", (30, 40, 20), 0.1), ("iid", (60, 220, 20), 1.0)])
@pytest.mark.parametrize("fp32", [False, True])
def test_tuned_steps_equal_untuned(model, dims, c, fp32, monkeypatch):
    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    for var in ENV:
        monkeypatch.delenv(var, raising=False)
    monkeypatch.setenv("MLP_MERGE", "1")  # step plans
    A, b = M.CSRMatrix.spe(*dims, *fields.field(model, 9), c=c)
    f = np.random.default_rng(5).standard_normal(A.n)
    out = []
    for autotune in (False, True):
        P = M.MultiSplitPrec(A, fp32=fp32, autotune=autotune, **MS)
        assert not any(n.startswith("sweep") for n, _, _ in P.profile(1))
        out.append(P.solve(f))
    # another order of a row's sum: 1e-13 (1e-6 with FP32 values) as for the composed form
    assert np.linalg.norm(out[1] - out[0]) <= (1e-6 if fp32 else 1e-13) * np.linalg.norm(out[0])
