"""Plastic solves of more than 2^19 points, whose reducing passes have more
tiles than resident blocks, against the oracle: from rest and from forces
(whose first offset is a sum over the whole field)."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    nb = (1024, 1024)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=31)
    kw = dict(external_force=2e-3, hardness=0.05 / (nb[0] * nb[1]),
              pentol=1e-6 * (h.max() - h.min()), forcetol=1e-8, maxiter=200)
    sub = oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0))
    cold = oc.constrained_conjugate_gradients(sub, h, **kw)
    f0 = -cold["jac"]
    warm = oc.constrained_conjugate_gradients(sub, h * 1.01, initial_forces=f0, **kw)
    return nb, h, kw, cold, f0, warm


@pytest.mark.parametrize("start", ["rest", "forces"])
def test_plastic_1024(case, start):
    """Same iteration count, fields to 1e-10; the masks but for points whose gap
    converges to zero (one in a thousand of the plastic ones)."""
    import contactmechanics_b200 as cm
    nb, h, kw, cold, f0, warm = case
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    if start == "rest":
        r, o = cm.constrained_conjugate_gradients(sub, h, **kw), cold
    else:
        r, o = cm.constrained_conjugate_gradients(sub, h * 1.01, initial_forces=f0, **kw), warm
    assert r.success and o["success"] and r.nit == o["nit"]
    for k in ("x", "jac"):
        assert np.linalg.norm(r[k] - o[k]) <= 1e-10 * np.linalg.norm(o[k])
    assert np.count_nonzero(r.active_set != o["active_set"]) <= 1e-3 * np.count_nonzero(o["active_set"])
    assert np.count_nonzero(r.plastic != o["plastic"]) <= 1e-3 * np.count_nonzero(o["plastic"])
