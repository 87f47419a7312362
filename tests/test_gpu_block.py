"""Block CG of the multigrid inner solve (24 load cases in one Krylov space) against the FP64 path.

Sizes at the edges of its node pieces (fewer nodes than one staged tile, exactly full tiles, pieces of
the largest size) and domains whose load cases are linearly dependent (bone that touches a few
faces only), where the block loses columns.  Tolerance on C: FP64 at rtol 1e-10 carries an error of
about 10 rtol (reaction projection, linear); the energy estimator's is quadratic in 1e-8.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-8


def solid(shape):
    return np.full(shape, 20000, np.int16)


def column(shape, w):
    """A bar along z through the domain: only the two z faces prescribe displacements."""
    g = np.zeros(shape, np.int16)
    y, x = (shape[1] - w) // 2, (shape[2] - w) // 2
    g[:, y:y + w, x:x + w] = 20000
    return g


def cantilever(shape, w):
    """A bar that touches one face."""
    g = column(shape, w)
    g[shape[0] // 2:] = 0
    return g


CASES = {
    "few_nodes": lambda: [solid((2, 2, 2)), solid((4, 4, 4)), column((6, 6, 6), 2)],           # 1, 27, 45 nodes
    "full_tiles": lambda: [solid((5, 5, 5)), solid((9, 9, 9)), solid((3, 9, 5))],              # 64, 512, 64 nodes
    "dependent": lambda: [column((9, 8, 7), 3), cantilever((12, 9, 9), 3), column((5, 12, 12), 1),
                          solid((6, 6, 6))],
    "largest_pieces": lambda: [solid((28, 28, 28)) for _ in range(8)] + [column((17, 17, 17), 5)],
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_block_cg_matches_fp64(dtc, name):
    syn = dtc.synth
    rng = np.random.default_rng(5)
    doms = []
    for i, g in enumerate(CASES[name]()):
        E = np.where(g > 0, rng.uniform(5000.0, 20000.0, g.shape), 0.0).astype(np.float32)
        doms.append(dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=E, domain_number=i))
    with dtc.Solver(precision="fp64", rtol=1e-10, rotation_search=False) as s:
        ref = s.solve(doms)
    with dtc.Solver(precision="mixed", rtol=1e-8, rotation_search=False, inner_precond="mg", estimator="energy") as s:
        res = s.solve(doms)
    for r, f in zip(res, ref):
        assert r["status"] == f["status"] == dtc.DOMAIN_OK
        assert np.abs(r["c"] - f["c"]).max() <= TOL * np.abs(f["c"]).max()
        assert max(r["relres"]) <= 1e-8
