"""max_it on the mixed path caps each FP32 inner solve: a domain that needs more goes on in the next refinement step,
up to max_refine of them, and is reported as not converged only when these run out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["mg", "block"])
def test_cap_is_per_inner_solve(dtc, precond):
    syn = dtc.synth
    doms = [dtc.Domain(syn.bone_volume((12, 12, 12), 0.4, syn.seed_for(61, i)), E=syn.E_CONST, nu=syn.NU,
                       delta=syn.DELTA, domain_number=i) for i in range(3)]
    kw = dict(precision="mixed", inner_precond=precond, rtol=1e-6, rotation_search=False)
    cap = 9 if precond == "mg" else 40
    with dtc.Solver(**kw) as s:
        refs = s.solve(doms)
    with dtc.Solver(max_it=cap, **kw) as s:
        res = s.solve(doms)
    with dtc.Solver(max_it=2, max_refine=2, **kw) as s:
        short = s.solve(doms)
    for r, f, q in zip(res, refs, short):
        assert f["status"] == r["status"] == dtc.DOMAIN_OK
        assert cap < max(r["iters"]) <= cap * r["refine_steps"]
        assert np.abs(r["c"] - f["c"]).max() <= 2e-5 * np.abs(f["c"]).max()   # about 10 rtol each
        assert q["status"] == dtc.DOMAIN_MAX_IT and max(q["iters"]) <= 2 * 2
