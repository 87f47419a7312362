"""The last two multigrid levels in one kernel (batches of at most 128 domains) against the same steps as kernels
of their own (the same domains among more than 128), at edges of their grids: levels of 5 to 8 voxels, uneven
halving, boxes that are not cubes, a last level below the first and below the second halving.

Tolerance on C: FP64 refinement to rtol 1e-10, a reaction projection's error is about 10 rtol.  The V-cycles are the
same operator up to FP32 rounding, so the inner iterations agree but for a threshold crossed one sooner or later.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(16, 16, 16), (9, 9, 9), (11, 16, 13), (10, 5, 16), (17, 17, 17), (32, 20, 18), (3, 16, 9)]


def domain(dtc, shape, seed):
    syn = dtc.synth
    rng = np.random.default_rng(seed)
    g = np.where(rng.random(shape) < 0.7, rng.integers(20000, 30001, shape), 0).astype(np.int16)
    g[0, 0, 0] = g[-1, -1, -1] = 20000
    return dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=syn.modulus_of_gray(g), domain_number=seed)


@pytest.mark.parametrize("elem", [8, 20])
def test_tail_matches_separate_kernels(dtc, elem):
    doms = [domain(dtc, s, k) for k, s in enumerate(SHAPES if elem == 8 else SHAPES[1:4])]
    if elem == 20:
        doms = [dtc.Domain(d.phi, E=dtc.synth.E_CONST, nu=dtc.synth.NU, delta=dtc.synth.DELTA, elem_type=dtc.HEX20,
                           domain_number=k) for k, d in enumerate(doms)]
    pad_kw = dict(E=dtc.synth.E_CONST, nu=dtc.synth.NU, delta=dtc.synth.DELTA)
    if elem == 20:
        pad_kw["elem_type"] = dtc.HEX20
    pad = [dtc.Domain(np.full((2, 2, 2), 20000, np.int16), domain_number=100 + k, **pad_kw) for k in range(128)]
    with dtc.Solver(precision="mixed", inner_precond="mg", rtol=1e-10, rotation_search=False) as s:
        few = s.solve(doms)
        many = s.solve(doms + pad)[:len(doms)]
    for a, b in zip(few, many):
        assert a["status"] == b["status"]
        assert np.abs(a["c"] - b["c"]).max() <= 1e-8 * np.abs(b["c"]).max()
        assert np.abs(a["iters"] - b["iters"]).max() <= 3 * max(1, a["refine_steps"]), (a["iters"], b["iters"])
