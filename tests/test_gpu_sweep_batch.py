"""The HEX08 sweeps and the HEX20 columns in batches large enough for their long tiles: sweeps of 16 and 8 nodes in
x (17 and 9 voxels walked, every place of the ring of 5 planes used several times over) and columns of several layers
whose last one is shorter.  Small batches get tiles of 4 nodes and columns of one layer.

Each batch repeats two domains (constant moduli; 60 % bone with a modulus per voxel), which are compared with the
oracle in FP64 and mixed (multigrid: residual and post-smoothing sweeps).  Tolerance: rtol 1e-10 on both sides, a
reaction projection's error is about 10 rtol.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-8


def sweep_length(shapes):
    """Nodes in x of the sweep tiles: halved from 16 while 3 CTAs a tile leave 2 x 148 places empty."""
    up = lambda n, t: -(-(n - 1) // t)
    tiles = sum(up(s[2], 16) * up(s[1], 8) * up(s[0], 6) for s in shapes)
    n = 16
    while n > 4 and 3 * tiles * (16 // n) < 2 * 148:
        n //= 2
    return n


def column_layers(shapes):
    """Layers of a HEX20 column: those whose longest SM walks the fewest, one more per column than it owns."""
    cost = lambda n: -(-sum(3 * math.ceil(s[2] / 8) * math.ceil(s[1] / 6) * math.ceil(s[0] / n) for s in shapes) // 148) * (n + 1)
    return min(range(max(s[0] for s in shapes), 0, -1), key=cost)


def check(dtc, orc, shape, copies, elem, solvers):
    syn = dtc.synth
    rng = np.random.default_rng(sum(shape))
    pair, odoms = [], []
    for i, frac in enumerate((1.0, 0.6)):
        g = np.where(rng.random(shape) < frac, rng.integers(20000, 30001, shape), 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000   # the bone's bounding box is the domain
        kw = dict(E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=syn.modulus_of_gray(g) if i else None)
        pair.append((g, kw))
        odoms.append(orc.Domain(g, rtol=1e-10, **kw, **({"nen": 20} if elem == 20 else {})))
    refs = orc.solve_batch(odoms)
    doms = [dtc.Domain(pair[i % 2][0], domain_number=i, elem_type=elem, **pair[i % 2][1]) for i in range(copies)]
    for kw in solvers:
        with dtc.Solver(rtol=1e-10, rotation_search=False, **kw) as s:
            res = s.solve(doms)
        for i, r in enumerate(res):
            ref = refs[i % 2]
            assert r["status"] == ref["status"]
            for k in ("c", "ff"):
                assert np.abs(r[k] - ref[k]).max() <= TOL * np.abs(ref[k]).max(), (kw, i, k)


# voxels z, y, x and domains: one tile exactly, one node more and less per axis, several tiles with a remainder in x
@pytest.mark.parametrize("shape, copies, length", [
    ((7, 9, 17), 100, 16), ((8, 10, 18), 26, 16), ((6, 8, 16), 100, 16), ((13, 7, 34), 18, 16), ((3, 4, 21), 50, 16),
    ((7, 9, 17), 60, 8), ((6, 8, 12), 50, 8), ((4, 5, 42), 17, 8)])
def test_long_sweep_tiles(dtc, orc, shape, copies, length):
    assert sweep_length([shape] * copies) == length
    check(dtc, orc, shape, copies, 8, (dict(precision="fp64"), dict(precision="mixed", inner_precond="mg")))


# voxels z, y, x, domains and layers: a remainder of one and of two layers, an exact division, several columns
@pytest.mark.parametrize("shape, copies, layers", [
    ((7, 5, 5), 24, 4), ((7, 3, 3), 16, 3), ((6, 6, 8), 24, 3), ((5, 7, 9), 12, 5), ((9, 4, 5), 49, 9)])
def test_columns_of_several_layers(dtc, orc, shape, copies, layers):
    assert column_layers([shape] * copies) == layers
    check(dtc, orc, shape, copies, 20, (dict(precision="fp64"), dict(precision="mixed", inner_precond="mg")))
