"""Launches that are resident before their predecessor has written: chains of
applications and products without a synchronisation in between have to give, bit
for bit, what they give one at a time. Vectors change from call to call and are
written in place, so a stale line of one would show."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MS = dict(q=(0.8,), niter=(5,), max_levels=15, degree_max=2)
ENV = ("MLP_PERSIST", "MLP_MERGE", "MLP_FOLD", "MLP_SMALL_BUDGET", "MLP_DENSE_OP_MAX")


def _p(t):
    return C.c_void_p(t.data_ptr())


# composed launches before a step of the plan below them (a one-sweep level, one
# CTA for the small levels); two composed launches; step plans without a graph
@pytest.mark.parametrize("dims,c,kw,env", [((30, 40, 20), 0.1, dict(niter=(1, 3, 1, 4)), {}),
                                           ((30, 40, 20), 0.1, {}, {"MLP_DENSE_OP_MAX": "0"}),
                                           ((31, 117, 23), 1.0, {}, {"MLP_SMALL_BUDGET": "0"}),
                                           ((12, 22, 6), 1.0, {}, {}),
                                           ((7, 11, 5), 1.0, {}, {}),
                                           ((12, 22, 6), 1.0, dict(max_levels=1), {"MLP_MERGE": "1"})])
@pytest.mark.parametrize("fp32", [False, True])
def test_chain_equals_single_calls(dims, c, kw, env, fp32, monkeypatch):
    import torch

    import ml_prec_b200 as M
    from ml_prec_b200 import fields
    from ml_prec_b200._capi import check, lib
    for var in ENV:
        monkeypatch.delenv(var, raising=False)
    for var, v in env.items():
        monkeypatch.setenv(var, v)
    A, _ = M.CSRMatrix.spe(*dims, *fields.field("layered", 9), c=c)
    P = M.MultiSplitPrec(A, fp32=fp32, **dict(MS, **kw))
    stream = torch.cuda.Stream()
    s = C.c_void_p(stream.cuda_stream)
    x0 = torch.from_numpy(np.random.default_rng(5).standard_normal(A.n)).cuda()
    STEPS = 40

    def run(wait):
        x, y, out = x0.clone(), torch.empty_like(x0), []
        kept = [torch.empty_like(x0) for _ in range(STEPS)]
        torch.cuda.synchronize()
        for k in range(STEPS):
            check(lib().mlp_prec_apply(P.h, _p(x), _p(x), s))  # x = B x, in place
            wait()
            check(lib().mlp_spmv(A.h, _p(x), _p(y), s))        # y = A x
            wait()
            check(lib().mlp_prec_apply(P.h, _p(y), _p(x), s))  # x = B y
            wait()
            with torch.cuda.stream(stream):
                kept[k].copy_(y)
            out.append(kept[k])
        torch.cuda.synchronize()
        return out + [x]

    single = run(torch.cuda.synchronize)
    chain = run(lambda: None)
    for a, b in zip(single, chain):
        assert torch.equal(a, b)
    assert bool(torch.isfinite(single[-1]).all())
