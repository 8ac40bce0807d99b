"""Solves with a hardness on sides with prime factors above 7, whose launched
passes take direct DFT stages (cm_fft.cuh), against the oracle: one such factor
first, after other stages, and twice."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [(11, 26), (22, 121), (57, 74), (53, 64), (143, 30)])
def test_plastic_solve(nb):
    """Same iteration count, fields to 1e-10 and contact set, as for other sides."""
    import contactmechanics_b200 as cm
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=41)
    kw = dict(external_force=2e-3, hardness=0.05 / (nb[0] * nb[1]),
              pentol=1e-8 * (h.max() - h.min()), forcetol=1e-10, maxiter=60)
    o = oc.constrained_conjugate_gradients(oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0)), h, **kw)
    r = cm.constrained_conjugate_gradients(cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0)), h, **kw)
    assert r.nit == o["nit"] and r.success == o["success"]
    for k in ("x", "jac"):
        assert np.linalg.norm(r[k] - o[k]) <= 1e-10 * np.linalg.norm(o[k])
    assert np.array_equal(r.active_set, o["active_set"])
