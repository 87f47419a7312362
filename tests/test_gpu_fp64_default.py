"""The plain FP64 path at loose tolerances (tile_cg.cuh): its results do not move with the order of summation.

At rtol 1e-3 the iterate stops where rounding decides on the last iteration, so another summation order gives
another tensor (by up to 1e-3) and other iteration counts.  The recorded domains are two node tiles each, whose sums
have one order; the recorded results are those of the kernels that the setting has always had.  Tolerance 1e-9: in
the same order only the reactions' last bits differ.

At the edges of the tiles (16 x 4 x 4 nodes for the operator, 8 x 4 x 4 for the vectors) against the oracle, just
above the tolerance from which the sweeps take over; a reaction projection's error is about 10 rtol on both sides.
"""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).parent / "golden" / "fp64_default.npz"


def test_default_tolerance_keeps_recorded_results(dtc):
    syn = dtc.synth
    f = np.load(GOLDEN)
    doms = [dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=e, domain_number=i)
            for i, (g, e) in enumerate(zip(f["phi"], f["E"]))]
    with dtc.Solver(precision="fp64", rtol=1e-3, rotation_search=False) as s:
        for res in (s.solve(doms), s.solve(doms)):
            for r, c, it in zip(res, f["c"], f["iters"]):
                assert r["status"] == dtc.DOMAIN_OK
                assert np.array_equal(r["iters"], it)
                assert np.abs(r["c"] - c).max() <= 1e-9 * np.abs(c).max()


# voxels z, y, x: one tile exactly, one node more and less per axis, the smallest, several tiles along each axis
SHAPES = [(5, 5, 17), (6, 6, 18), (4, 4, 16), (2, 2, 2), (3, 20, 5), (13, 7, 34), (5, 9, 9)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_node_tiles_at_their_edges(dtc, orc, shape):
    syn = dtc.synth
    rng = np.random.default_rng(sum(shape))
    doms, odoms = [], []
    for i, frac in enumerate((1.0, 0.6)):
        g = np.where(rng.random(shape) < frac, rng.integers(20000, 30001, shape), 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000
        E = syn.modulus_of_gray(g) if i else None
        kw = dict(E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=E)
        doms.append(dtc.Domain(g, domain_number=i, **kw))
        odoms.append(orc.Domain(g, rtol=1e-10, **kw))
    refs = orc.solve_batch(odoms)
    with dtc.Solver(rtol=2e-10, rotation_search=False, precision="fp64") as s:
        res = s.solve(doms)
    for r, ref in zip(res, refs):
        assert r["status"] == ref["status"]
        for k in ("c", "ff"):
            assert np.abs(r[k] - ref[k]).max() <= 1e-8 * np.abs(ref[k]).max(), k
