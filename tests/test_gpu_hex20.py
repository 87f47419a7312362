"""HEX20 operator on voxel columns at the edges of its columns (8 x 6 voxels, layers by the size of the batch)
against the oracle, constant and per-voxel moduli, FP64 and mixed.

Tolerance: rtol 1e-10 on both sides, a reaction projection's error is about 10 rtol.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# voxels z, y, x: the smallest, one column exactly, one voxel more and less per axis, several columns
SHAPES = [(2, 2, 2), (3, 6, 8), (4, 7, 9), (5, 5, 7), (2, 13, 3), (3, 3, 17)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_columns_at_their_edges(dtc, orc, shape):
    syn = dtc.synth
    rng = np.random.default_rng(sum(shape))
    doms, odoms = [], []
    for i, frac in enumerate((1.0, 0.6)):
        g = np.where(rng.random(shape) < frac, rng.integers(20000, 30001, shape), 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000   # the bone's bounding box is the domain
        E = syn.modulus_of_gray(g) if i else None
        kw = dict(E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=E)
        doms.append(dtc.Domain(g, domain_number=i, elem_type=dtc.HEX20, **kw))
        odoms.append(orc.Domain(g, nen=20, rtol=1e-10, **kw))
    refs = orc.solve_batch(odoms)
    for kw in (dict(precision="fp64"), dict(precision="mixed", inner_precond="block"),
               dict(precision="mixed", inner_precond="mg")):
        with dtc.Solver(rtol=1e-10, rotation_search=False, **kw) as s:
            res = s.solve(doms)
        for r, ref in zip(res, refs):
            assert r["status"] == ref["status"]
            assert (r["ne"], r["nn"], r["nb"]) == (ref["ne"], ref["nn"], ref["nb"])
            for k in ("c", "ff"):
                assert np.abs(r[k] - ref[k]).max() <= 1e-8 * np.abs(ref[k]).max(), (kw, k)
