"""Which solves run in the persistent kernel (cm_solo.cu, cm_solo_gen.cu) and
which in launched passes, told by the kernels launched: a solve of 40 iterations
is one launch beside its set-up and its result, or at least seven an iteration."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu

NIT = 40

# (kind, topography, persistent)
CASES = [
    # sides with register-resident transforms in the kernel: one tile a block,
    # several tiles, and the largest
    ("periodic", (64, 64), True),
    ("periodic", (1024, 512), True),
    ("periodic", (1024, 768), True),
    ("periodic", (1024, 1024), False),
    ("free", (96, 128), True),
    # longer rows
    ("periodic", (64, 1536), True),
    ("periodic", (384, 1536), False),
    ("periodic", (64, 2048), False),
    ("free", (32, 1024), False),
    # longer columns
    ("periodic", (2048, 64), True),
    ("periodic", (3072, 64), True),
    ("periodic", (2048, 384), False),
    ("periodic", (4096, 64), False),
    # sides of any length: one tile a block, several, long columns
    ("periodic", (75, 91), True),
    ("periodic", (900, 700), True),
    ("periodic", (4000, 100), True),
    ("periodic", (4000, 150), False),
    ("periodic", (75, 64), True),
    ("periodic", (64, 75), True),
]


@pytest.mark.parametrize("kind,nb,persistent", CASES)
def test_route(kind, nb, persistent):
    """The route, and iterations and fields of the oracle (1e-10) where it is quick."""
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    if kind == "free":
        dev, ref = cm.FreeFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0)), oc.FreeSubstrate(nb, 1.0, (1.0, 1.0))
    else:
        dev, ref = (cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0)),
                    oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0)))
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=23)
    kw = dict(external_force=1e-3, pentol=1e-30, forcetol=0.0, maxiter=NIT)
    n0 = _lib.lib().cm_launch_count()
    r = cm.constrained_conjugate_gradients(dev, h, **kw)
    launches = _lib.lib().cm_launch_count() - n0
    assert r.nit == NIT
    assert launches < NIT if persistent else launches >= 7 * NIT
    if nb[0] * nb[1] <= 2 ** 18:
        o = oc.constrained_conjugate_gradients(ref, h, **kw)
        for k in ("x", "jac"):
            assert np.linalg.norm(r[k] - o[k]) <= 1e-10 * np.linalg.norm(o[k])


def test_time_limit_is_read_every_few_iterations():
    """A solve with a time limit launches the persistent kernel for a few
    iterations at a time, and ends in the same state."""
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    nb = (256, 256)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=24)
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    kw = dict(external_force=1e-3, pentol=1e-30, forcetol=0.0, maxiter=NIT)
    free = cm.constrained_conjugate_gradients(sub, h, **kw)
    n0 = _lib.lib().cm_launch_count()
    r = cm.constrained_conjugate_gradients(sub, h, timeout=1e3, **kw)
    launches = _lib.lib().cm_launch_count() - n0
    n0 = _lib.lib().cm_launch_count()
    cm.constrained_conjugate_gradients(sub, h, **kw)
    assert launches == _lib.lib().cm_launch_count() - n0 - 1 + NIT // 8
    assert np.array_equal(r.x, free.x) and np.array_equal(r.jac, free.jac)
