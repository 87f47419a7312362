"""Rotation search where its split of the work changes: few tensors (more CTAs a tensor, two threads a
refinement axis), many (64 CTAs, one thread), against the oracle's search of the same tensors bit for bit.

The tensors are ones the bound on a candidate's partial sums could decide wrongly: all candidates tied (zero,
isotropic), squares that underflow or overflow, and criteria that reach exactly zero.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tensors():
    rng = np.random.default_rng(11)
    iso = np.zeros((6, 6))
    iso[:3, :3] = 0.5
    iso[range(6), range(6)] = [1.5, 1.5, 1.5, 0.5, 0.5, 0.5]
    orth = np.zeros((6, 6))
    orth[:3, :3] = [[3.0, 0.7, 0.4], [0.7, 2.0, 0.5], [0.4, 0.5, 1.0]]
    orth[range(3, 6), range(3, 6)] = [0.9, 0.6, 0.4]
    a = rng.standard_normal((6, 6))
    full = a @ a.T + 4 * np.eye(6)
    return [np.zeros((6, 6)), iso, orth, full, full * 1e-162, full * 1e160]


@pytest.fixture(scope="module")
def reference(orc):
    return [orc.rotation_search(e) for e in tensors()]


@pytest.mark.parametrize("n", [1, 6, 13, 14, 31, 32, 70])
def test_rotation_split_matches_oracle(dtc, reference, n):
    ees = tensors()
    pick = [(3 + i) % len(ees) for i in range(n)]   # n = 1: the full tensor
    with dtc.Solver(precision="fp64") as s:
        res = s.rotation_search(np.stack([ees[p] for p in pick]))
    for i, p in enumerate(pick):
        for w in ("cr1", "cr2"):
            got, ref = res[i][w], reference[p][w]
            assert got["iters"] == ref["iters"], (i, p, w)
            assert got["crit"] == ref["crit"], (i, p, w)
            assert got["angle"] == ref["angle"], (i, p, w)
