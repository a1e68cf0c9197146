"""The composed form is optional: where the device has room for the step plan
but not for the composed operators, the hierarchy is made with the step plan."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import torch
import ml_prec_b200 as M
from ml_prec_b200 import fields

MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)
spare = int(sys.argv[1])  # bytes to leave for the hierarchy, 0: all
torch.zeros(1, device="cuda")
for fp32 in (False, True):  # the kernels are loaded before memory is measured
    A, b = M.CSRMatrix.spe(30, 40, 20, *fields.field("layered", 9), c=0.1)
    M.PCGSolver(A, b, M.MultiSplitPrec(A, fp32=fp32, **MS), eps=1e-8, flexible=True)
A, b = M.CSRMatrix.spe(59, 211, 37, *fields.field("layered", 2), c=0.1)
free = torch.cuda.mem_get_info()[0]
held = [] if not spare else [torch.empty(free - spare, dtype=torch.uint8, device="cuda")]
P = M.MultiSplitPrec(A, **MS)
used = (spare or free) - torch.cuda.mem_get_info()[0]
held.clear()
torch.cuda.empty_cache()
st = M.SolverStats()
M.PCGSolver(A, b, P, stats=st, eps=1e-8, flexible=True)
composed = any(n.startswith("sweep") for n, _, _ in P.profile(1))
print("RESULT", used, int(composed), st.niter)
"""


def _child(spare, **env):
    full = {k: v for k, v in os.environ.items() if not k.startswith("MLP_")}
    r = subprocess.run([sys.executable, "-c", CHILD, str(spare)], cwd=ROOT, env=dict(full, **env),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return [int(t) for t in r.stdout.split("RESULT")[1].split()]


def test_step_plan_where_the_composed_form_does_not_fit():
    steps, composed, its = _child(0, MLP_MERGE="1")
    assert not composed
    full, composed, _ = _child(0)
    assert composed and full > steps + (160 << 20)  # 310 MB more
    _, composed, got = _child(steps + (64 << 20))
    assert not composed and abs(got - its) <= 1
