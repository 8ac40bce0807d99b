"""The persistent solver of small problems (cm_solo.cu) against the oracle: the
smallest and largest sides it serves, sides 3 * 2^m, sides of any other length
along one axis or both (odd, prime, one row pair), long thin domains (one
pass has many tiles, the other few), free domains whose blocks hold padding
rows only, and domains whose blocks have several tiles each."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu

CASES = [
    ("periodic", (64, 64)),
    ("periodic", (64, 1024)),
    ("periodic", (1024, 64)),
    ("periodic", (96, 768)),
    ("periodic", (768, 96)),
    ("periodic", (512, 256)),
    ("periodic", (1024, 512)),
    ("free", (32, 48)),
    ("free", (128, 128)),
    ("free", (64, 384)),
    ("free", (256, 96)),
    ("periodic", (75, 91)),
    ("periodic", (64, 75)),
    ("periodic", (75, 64)),
    ("periodic", (96, 90)),
    ("periodic", (67, 97)),
    ("periodic", (20, 500)),
    ("periodic", (1000, 30)),
    ("periodic", (900, 700)),
    ("free", (45, 60)),
    ("free", (33, 32)),
    ("free", (125, 90)),
]


def substrates(kind, nb):
    import contactmechanics_b200 as cm
    if kind == "free":
        return cm.FreeFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0)), oc.FreeSubstrate(nb, 1.0, (1.0, 1.0))
    return (cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0)),
            oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0)))


@pytest.mark.parametrize("kind,nb", CASES)
@pytest.mark.parametrize("control", ["load", "offset"])
def test_solve_fp64(kind, nb, control):
    """Same iteration count and active set; fields to 1e-10 as everywhere in FP64."""
    import contactmechanics_b200 as cm
    dev, ref = substrates(kind, nb)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=17)
    span = h.max() - h.min()
    kw = dict(pentol=1e-9 * span, forcetol=1e-12, maxiter=2000)
    if control == "load":
        kw["external_force"] = 1e-3
    else:
        kw["offset"] = -h.max() + 0.2 * span
    r = cm.constrained_conjugate_gradients(dev, h, **kw)
    o = oc.constrained_conjugate_gradients(ref, h, **kw)
    assert r.success and o["success"]
    assert r.nit == o["nit"] and r.nfev == o["nfev"]
    np.testing.assert_array_equal(r.active_set, o["active_set"])
    for k in ("x", "jac"):
        assert np.linalg.norm(r[k] - o[k]) <= 1e-10 * np.linalg.norm(o[k])
    assert abs(r.offset - o["offset"]) <= 1e-10 * abs(o["offset"])


@pytest.mark.parametrize("kind,nb", [("periodic", (64, 1024)), ("periodic", (768, 96)),
                                     ("free", (128, 128)), ("periodic", (1024, 512)),
                                     ("periodic", (75, 91)), ("free", (125, 90))])
def test_solve_mixed(kind, nb):
    """A mixed solve meets the FP64 criteria: within the pentol of 1e-9 of the
    height range of the FP64 solution, like the other mixed tests (1e-6)."""
    import contactmechanics_b200 as cm
    dev, ref = substrates(kind, nb)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=18)
    kw = dict(pentol=1e-9 * (h.max() - h.min()), forcetol=1e-12, maxiter=2000, external_force=1e-3)
    r = cm.constrained_conjugate_gradients(dev, h, precision="mixed", **kw)
    o = oc.constrained_conjugate_gradients(ref, h, **kw)
    assert r.success and r.nit_fp32 > 0
    assert np.linalg.norm(r.x - o["x"]) <= 1e-6 * np.linalg.norm(o["x"])


def test_stops_at_maxiter_across_launches():
    """More iterations than one launch runs, ended by maxiter."""
    import contactmechanics_b200 as cm
    nb = (64, 64)
    dev, ref = substrates("periodic", nb)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=19)
    kw = dict(pentol=1e-30, forcetol=0.0, maxiter=150, external_force=1e-3)
    r = cm.constrained_conjugate_gradients(dev, h, **kw)
    o = oc.constrained_conjugate_gradients(ref, h, **kw)
    assert not r.success and r.nit == o["nit"] == 150
    assert np.linalg.norm(r.x - o["x"]) <= 1e-10 * np.linalg.norm(o["x"])
