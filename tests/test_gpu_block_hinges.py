"""Block CG on bone with hinges: randomly placed voxels, many of which share an edge or a corner only, so that the
stiffness has null vectors (mechanisms) along which the load cases put no force.  CG load case by load case solves these
consistent systems; the block must too, also with moduli over four decades, and not by way of many refinement steps.

Against the FP64 path at rtol 1e-10 (about 10 rtol in a reaction projection, the energy products' error is quadratic
in the mixed solve's 1e-7): 1e-8 of the tensor.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def domains(dtc, elem, decades, seed):
    syn = dtc.synth
    rng = np.random.default_rng(100 * seed + elem)
    out = []
    for i in range(12):
        shape = tuple(int(x) for x in rng.integers(5, 17 if elem == 8 else 9, 3))
        g = np.where(rng.random(shape) < (0.1, 0.2, 0.3, 0.5)[i % 4], 20000, 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000
        E = np.where(g > 0, 10.0 ** rng.uniform(4 - decades, 4, shape), 0).astype(np.float32)
        out.append(dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=E, elem_type=elem, domain_number=i))
    return out


@pytest.mark.parametrize("seed", [1, 2])
@pytest.mark.parametrize("decades", [0, 4])
@pytest.mark.parametrize("elem", [8, 20])
def test_hinged_bone_is_solved(dtc, elem, decades, seed):
    doms = domains(dtc, elem, decades, seed)
    with dtc.Solver(precision="fp64", rtol=1e-10, rotation_search=False) as s:
        refs = s.solve(doms)
    with dtc.Solver(precision="mixed", rtol=1e-7, rotation_search=False, inner_precond="mg", estimator="energy") as s:
        res = s.solve(doms)
    for r, f in zip(res, refs):
        assert r["status"] == f["status"]
        assert r["refine_steps"] <= 6
        assert np.abs(r["c"] - f["c"]).max() <= 1e-8 * np.abs(f["c"]).max()
