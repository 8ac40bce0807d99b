"""Solves whose persistent launch (cm_solo.cu, cm_solo_gen.cu) is refused, at
their first launch or between two, go on in launched passes."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [(96, 128), (75, 91)])  # register-resident and other sides
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("launches", [0, 1])
def test_refused_launch(nb, precision, launches):
    """The oracle's iterations, contact set and fields (1e-10) in FP64; in mixed
    precision its fields to 1e-6, as in the other mixed tests.  The next solve
    on the plan too, without the kernel."""
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=25)
    kw = dict(external_force=1e-3, pentol=1e-9 * (h.max() - h.min()), forcetol=1e-13, maxiter=2000)
    o = oc.constrained_conjugate_gradients(oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0)), h, **kw)
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    prec = _lib.CM_FP64 if precision == "fp64" else _lib.CM_FP32
    assert _lib.lib().cm_selftest_refuse_solver(sub._plan.ptr, prec, launches) == _lib.CM_OK
    for _ in range(2):
        n0 = _lib.lib().cm_launch_count()
        # (with a time limit a launch is 16 iterations, of 18 at least)
        r = cm.constrained_conjugate_gradients(sub, h, precision=precision, timeout=1e3, **kw)
        assert _lib.lib().cm_launch_count() - n0 > 7 * 8
        assert r.success and o["success"]
        tol = 1e-10 if precision == "fp64" else 1e-6
        for k in ("x", "jac"):
            assert np.linalg.norm(r[k] - o[k]) <= tol * np.linalg.norm(o[k])
        if precision == "fp64":
            assert r.nit == o["nit"]
            assert np.array_equal(r.active_set, o["active_set"])
