"""The operator's row and column passes on both sides of the rules for their
shapes (cm_op_p2.cu: small blocks or large ones, few columns a block each, or
groups and pairs of blocks), against an FFT in numpy."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu

# rows of 64, 384 and 512 in small and in large blocks; columns of 2048, 3072
# and 4096 in few groups and in many; columns of 512 and 768
SIDES = [(2048, 64), (2048, 512), (2048, 768), (3072, 64), (3072, 256), (3072, 384),
         (4096, 64), (4096, 256), (4096, 384), (512, 512), (512, 1536), (768, 96), (3072, 512),
         (1024, 384), (1536, 384), (6144, 64), (1536, 512), (8192, 64)]


@pytest.mark.parametrize("nb", SIDES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_operators(nb, precision):
    """1e-12 of the maximum in FP64 and 2e-5 in FP32, as for the other sides."""
    import contactmechanics_b200 as cm
    tol = 1e-12 if precision == "fp64" else 2e-5
    f = np.random.default_rng(nb[0] + nb[1]).standard_normal(nb)
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), precision=precision)
    ref = oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0))
    for op in ("evaluate_disp", "evaluate_force"):
        want = getattr(ref, op)(f)
        got = getattr(sub, op)(f)
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
