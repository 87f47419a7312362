"""The autotuned operator is chosen for the size of the launch: a batch that fills the card times the candidates
for itself, also after a single domain of the same edge and bone fraction did."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem, L, n", [(8, 13, 96), (20, 7, 96)])
def test_batch_is_not_tuned_by_a_single_domain(dtc, elem, L, n):
    syn = dtc.synth
    g = syn.bone_volume((L, L, L), 0.4, syn.seed_for(41, 0))
    doms = [dtc.Domain(g, E=syn.E_CONST, nu=syn.NU, delta=syn.DELTA, elem_type=elem, domain_number=i) for i in range(n)]

    def timings(batch):
        with dtc.Solver(precision="mixed", inner_precond="mg", mixed_matvec="auto", rtol=1e-6, rotation_search=False,
                        profile_kernels=True) as s:
            s.solve(batch)
            k = s.kernel_stats()
        return k["autotune_simt_sweep"]["ms_total"], k["autotune_tc_sweep"]["ms_total"]

    one, many, again = timings(doms[:1]), timings(doms), timings(doms)
    assert np.all(np.array(many) > 0) and many == again
    assert many != one
