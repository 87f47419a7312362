"""Block CG on bones whose load cases are numerically dependent: two small bones (142 and 567 voxels) in a corner of
a domain of 24^3 and 32^3, each touching two faces, whose 24 right-hand sides span 18 dimensions up to rounding.

A direction made of rounding noise must not enter the iteration: load case by load case these domains take at most
42 iterations, so the block must not need more (it took thousands).  Both alone, which runs the last two multigrid levels
in one kernel, and among more than 128 domains.  Tolerance on C as for the block CG elsewhere: FP64 at rtol 1e-10 carries
about 10 rtol.
"""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BONES = Path(__file__).parent / "golden" / "corner_bones.npz"


@pytest.mark.parametrize("bone", ["a", "b"])
@pytest.mark.parametrize("pad", [0, 1, 130])
def test_dependent_load_cases_converge(dtc, bone, pad):
    syn = dtc.synth
    g = np.load(BONES)[bone]
    E = np.where(g > 0, 5000.0 + 1.5 * (g.astype(np.float64) - 20000.0), 0.0).astype(np.float32)
    kw = dict(E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA)
    doms = [dtc.Domain(g, E_voxel=E, domain_number=0, **kw)]
    if pad == 1:
        doms.append(doms[0])
    else:
        doms += [dtc.Domain(np.full((2, 2, 2), 20000, np.int16), domain_number=1 + i, **kw) for i in range(pad)]
    with dtc.Solver(precision="fp64", rtol=1e-10, rotation_search=False) as s:
        ref = s.solve(doms[:1])[0]
    with dtc.Solver(precision="mixed", rtol=1e-7, rotation_search=False, inner_precond="mg", estimator="energy") as s:
        r = s.solve(doms)[0]
    assert r["status"] == ref["status"] == dtc.DOMAIN_OK
    assert max(r["iters"]) <= 42, r["iters"]
    assert np.abs(r["c"] - ref["c"]).max() <= 1e-8 * np.abs(ref["c"]).max()
