"""Handles on one GPU do not share state: each solve's Poisson ratio, element, macro order and tensor-core operand
are its own, whatever other handles do in between or at the same time.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# options and Poisson ratio; the tolerances bring every solve to 1e-8 of its tensor or better
KINDS = [
    dict(nu=0.3, precision="mixed", inner_precond="mg", estimator="energy", rtol=1e-7),
    dict(nu=0.15, precision="mixed", inner_precond="mg", estimator="energy", rtol=1e-7, mixed_matvec="tensor"),
    dict(nu=0.2, precision="fp64", rtol=1e-10),
    dict(nu=0.35, precision="fp64", rtol=3e-10, macro_order=2),
    dict(nu=0.25, elem=20, precision="mixed", inner_precond="mg", estimator="energy", rtol=1e-7, device_mesher=True),
    dict(nu=0.1, precision="mixed", inner_precond="block", rtol=1e-9, device_mesher=True),
]


def domains(dtc, nu, elem=8, n=4, L=14):
    syn = dtc.synth
    out = []
    for i in range(n):
        L_i = (L if elem == 8 else L // 2) + i
        g = syn.bone_volume((L_i,) * 3, 0.4, syn.seed_for(31, i))
        out.append(dtc.Domain(g, E=syn.E_CONST, nu=nu, delta=syn.DELTA, elem_type=elem, domain_number=i))
    return out


def test_gradient_after_another_handles_solve(dtc):
    opts = dict(precision="mixed", inner_precond="mg", estimator="energy", rtol=1e-7, rotation_search=False)
    doms, other = domains(dtc, 0.3), domains(dtc, 0.1)
    dl = np.stack([np.eye(6)] * len(doms))

    def grads(between):
        g = [np.zeros(d.phi.shape, np.float32) for d in doms]
        with dtc.Solver(keep_displacements=True, **opts) as a, dtc.Solver(**opts) as b:
            a.solve(doms)
            if between:
                b.solve(other)
            a.energy_grad(dl, g)
        return g

    # two solves agree to their tolerance, and FP32 gradients to their last bits
    for x, y in zip(grads(False), grads(True)):
        assert np.abs(x - y).max() <= 1e-5 * np.abs(x).max()


def test_handles_in_threads(dtc):
    def make(kind):
        kw = dict(kind)
        return domains(dtc, kw.pop("nu"), kw.pop("elem", 8)), dtc.Solver(rotation_search=False, **kw)

    pairs = [make(k) for k in KINDS]
    want = [np.stack([r["c"] for r in s.solve(doms)]) for doms, s in pairs]
    worst, errors = [0.0] * len(pairs), []

    def work(i):
        try:
            doms, s = pairs[i]
            for _ in range(8):
                res = s.solve(doms)
                assert all(r["status"] == dtc.DOMAIN_OK for r in res)
                got = np.stack([r["c"] for r in res])
                worst[i] = max(worst[i], np.abs(got - want[i]).max() / np.abs(want[i]).max())
        except BaseException as e:   # reported by the main thread
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(pairs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for _, s in pairs:
        s.close()
    assert not errors, errors
    assert max(worst) <= 1e-7, worst
