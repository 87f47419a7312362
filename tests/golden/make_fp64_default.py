"""Fixture of the plain FP64 path at the reference's default tolerance (rtol 1e-3): 12 domains of 17 x 5 x 5
voxels, moduli over six decades, and the tensors and iteration counts the library gives for them.  Such a domain is
two node tiles, whose sums do not depend on the order of atomic additions.  Needs a GPU.

    python tests/golden/make_fp64_default.py            # writes tests/golden/fp64_default.npz
"""
import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[2]
sys.path.insert(0, str(ROOT))
import __graft_entry__ as entry   # noqa: E402

SHAPE, COUNT = (5, 5, 17), 12


def inputs():
    phi, E = [], []
    for i in range(COUNT):
        rng = np.random.default_rng(7000 + i)
        g = np.where(rng.random(SHAPE) < 0.6, 20000, 0).astype(np.int16)
        g[0, 0, 0] = g[-1, -1, -1] = 20000   # the bone's bounding box is the domain
        phi.append(g)
        E.append(np.where(g > 0, 10.0 ** rng.uniform(-2, 4, SHAPE), 0).astype(np.float32))
    return np.stack(phi), np.stack(E)


def main():
    dtc = entry.load_package()
    syn = dtc.synth
    phi, E = inputs()
    doms = [dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, E_voxel=e, domain_number=i)
            for i, (g, e) in enumerate(zip(phi, E))]
    with dtc.Solver(precision="fp64", rtol=1e-3, rotation_search=False) as s:
        res = s.solve(doms)
    np.savez_compressed(ROOT / "tests/golden/fp64_default.npz", phi=phi, E=E, c=np.stack([r["c"] for r in res]),
                        iters=np.stack([r["iters"] for r in res]))


if __name__ == "__main__":
    main()
