"""Rigid translations cost nothing with quadratic elements: the macro stiffness (24 x 24, nodal) gives no force for a
translation of the whole domain, beyond rounding.

The displacements of a translation are constant in the domain, so any force is a spurious stiffness of the element
operator, counted in every voxel.  Rounding of its products, 1e-16 each with signs as they come, leaves a few 1e-14;
an element matrix off by one rounding in a translation's entries gave 1e-12 and more (and up to 2.8e-9 where FP32 solves
of weakly connected bone lost accuracy to it).  Tolerance between the two: 2e-13.  With the energy estimator the solver's
own error enters squared: below 1e-14 at rtol 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [0.3, 0.45])
@pytest.mark.parametrize("kw", [dict(precision="fp64", rtol=1e-9), dict(precision="mixed", inner_precond="mg", rtol=1e-8)],
                         ids=["fp64", "mixed"])
def test_translations_have_no_stiffness(dtc, kw, nu):
    syn = dtc.synth
    doms = []
    for i, bvtv in enumerate((0.2, 0.35)):
        g = syn.bone_volume((24, 24, 24), bvtv, syn.seed_for(51, i))
        doms.append(dtc.Domain(g, E=syn.E_CONST, nu=nu, delta=syn.DELTA, elem_type=dtc.HEX20, domain_number=i))
    with dtc.Solver(rotation_search=False, estimator="energy", **kw) as s:
        res = s.solve(doms)
    t = np.kron(np.eye(3), np.ones((8, 1)))   # a unit translation along each axis
    for r in res:
        assert r["status"] == dtc.DOMAIN_OK
        assert np.abs(r["kmacro"] @ t).max() <= 2e-13 * np.abs(r["kmacro"]).max()
