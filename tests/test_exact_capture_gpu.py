"""A captured execution of each FP64 plan with an exact contraction follows the
operands of each replay: in range, out of range (the FP64 kernels behind the
flag), and in range again.  Same bits as the plan's ordinary execution, and
within the FP64 parity tests' 1e-12 of the oracle."""
import numpy as np
import pytest

import workload as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NB, NC, NG, NF = 45, 3001, 64, 3


def _dev(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy((a.view(np.float64) if np.iscomplexobj(a) else a).astype(np.float64).copy()).cuda()


def _setup(S, kind):
    """(problem, plan, run(stream), device aqsn, outputs, oracle)"""
    import torch
    zeros = lambda n: torch.zeros(n, dtype=torch.float64, device="cuda")
    if kind == "ff":
        p = W.ff_random(NB, NC, NG, NF, 92)
        e, n, m = (_dev(x) for x in (p.I_epsR, p.aqsntemp, p.aqsmtemp))
        out = zeros(NB * NF * 2)
        plan = S.FfPlan(NB, NC, NG, NF, p.inv_igp_index, p.indinv)
        run = lambda s: plan.execute(e.data_ptr(), n.data_ptr(), m.data_ptr(), out.data_ptr(), stream=s)
        return p, plan, run, n, [out], lambda q: O.ff_schdt(q)
    real = kind == "real"
    p = (W.gpp_real_random if real else W.gpp_random)(NB, 2, NC, NG, 91)
    ops = [_dev(x) for x in (p.wx_array[:3], p.aqsmtemp, p.aqsntemp, p.I_eps_array, p.wtilde_array, p.vcoul)]
    n = 1 if real else 2
    outs = [zeros(3 * n), zeros(3 * n), zeros(NB * n)] + ([zeros(2)] if kind == "half" else [])
    make = {"gpp": S.GppPlan, "real": S.GppRealPlan, "half": S.GppHalfSumPlan}[kind]
    plan = make(NB, 2, NC, NG, p.inv_igp_index, p.indinv)
    want = {"gpp": O.gpp, "real": O.gpp_real, "half": O.gpp_halfsum}[kind]
    return p, plan, lambda s: plan.execute(*ops, *outs, stream=s), ops[2], outs, lambda q: want(q)[0]


@pytest.mark.parametrize("kind", ["gpp", "real", "half", "ff"])
def test_captured_plan_follows_its_operands(sigma_lib, kind):
    import torch
    p, plan, run, aqsn, outs, oracle = _setup(sigma_lib, kind)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        graph.capture_begin()
        run(s.cuda_stream)
        graph.capture_end()
    clean, seen = p.aqsntemp.copy(), []
    for factor in (1.0, 2.0 ** 40, 1.0):
        p.aqsntemp = clean.copy()
        p.aqsntemp[7, 10] *= factor
        aqsn.copy_(_dev(p.aqsntemp).view_as(aqsn))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = [t.cpu().numpy().copy() for t in outs]
        for t in outs:
            t.zero_()
        run(0)
        torch.cuda.synchronize()
        for g, t in zip(got, outs):
            assert np.array_equal(g, t.cpu().numpy())
        g = got[0] if kind == "real" else got[0].view(np.complex128)
        o = np.asarray(oracle(p)).reshape(-1)
        assert np.abs(g - o).max() <= 1e-12 * np.abs(o).max()
        seen.append(got)
    assert all(np.array_equal(a, b) for a, b in zip(seen[0], seen[2]))
    plan.close()
