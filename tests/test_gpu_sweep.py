"""HEX08 sweeps in the voxel's Hadamard basis at the edges of their tiles (16 x 8 x 6 nodes inside the
domain, from node 0 for the reactions) against the oracle, constant and per-voxel moduli.

FP64 path at rtol 1e-10: the reaction projection's error is about 10 rtol on both sides.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# voxels z, y, x: one tile exactly (16 x 8 x 6 inner nodes), one node more and less per axis, one voxel
# thick inner layers, several tiles along each axis
SHAPES = [(7, 9, 17), (8, 10, 18), (6, 8, 16), (2, 2, 2), (3, 20, 5), (13, 7, 34), (19, 18, 3)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_sweeps_at_tile_edges(dtc, orc, shape):
    syn = dtc.synth
    rng = np.random.default_rng(sum(shape))
    doms, odoms = [], []
    for i, frac in enumerate((1.0, 0.6)):
        g = np.where(rng.random(shape) < frac, rng.integers(20000, 30001, shape), 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000   # the bone's bounding box is the domain
        E = syn.modulus_of_gray(g) if i else None
        kw = dict(E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=E)
        doms.append(dtc.Domain(g, domain_number=i, **kw))
        odoms.append(orc.Domain(g, rtol=1e-10, **kw))
    refs = orc.solve_batch(odoms)
    for kw, tol in ((dict(precision="fp64"), 1e-8), (dict(precision="mixed", inner_precond="block"), 1e-8)):
        with dtc.Solver(rtol=1e-10, rotation_search=False, **kw) as s:
            res = s.solve(doms)
        for r, ref in zip(res, refs):
            assert r["status"] == ref["status"]
            assert (r["ne"], r["nn"], r["nb"]) == (ref["ne"], ref["nn"], ref["nb"])
            for k in ("c", "ff"):
                assert np.abs(r[k] - ref[k]).max() <= tol * np.abs(ref[k]).max(), (kw, k)
