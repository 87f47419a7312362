"""Batches of very small domains on a nearly full card: the passes are cut by all that a domain needs, not by its
nodes alone (27 nodes of a 2^3 domain are 95 KB; its coarsest multigrid level and block CG state 57 KB more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_passes_of_small_domains_fit(dtc):
    torch = pytest.importorskip("torch")
    syn = dtc.synth
    g = np.full((2, 2, 2), 20000, np.int16)
    doms = [dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, domain_number=i) for i in range(5200)]
    kw = dict(precision="mixed", inner_precond="mg", rtol=1e-6, rotation_search=False)
    with dtc.Solver(**kw) as s:
        ref = s.solve(doms[:2])[0]["c"]
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - 640 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        with dtc.Solver(keep_displacements=True, **kw) as s:   # no leading pass for the host's sake
            res = s.solve(doms)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert all(r["status"] == dtc.DOMAIN_OK for r in res)
    assert max(np.abs(r["c"] - ref).max() for r in res) <= 1e-6 * np.abs(ref).max()
