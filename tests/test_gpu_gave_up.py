"""A wait of the one-launch operator (cm_op_one.cu) that runs out: the result
holds NaN, the next call reports it once, and the one after works.  The waits
end after 1 ms."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [(64, 64), (64, 512), (512, 512)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_operator_reports_a_wait_that_ran_out(nb, precision):
    import torch
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), precision=precision)
    f = torch.from_numpy(np.random.default_rng(21).standard_normal(nb)).cuda()
    f = f.to(torch.float64 if precision == "fp64" else torch.float32)
    want = sub.evaluate_disp(f)
    assert _lib.lib().cm_selftest_operator_barrier(sub._plan.ptr, _lib.PRECISIONS[precision], 1, 1e3) == _lib.CM_OK
    u = sub.evaluate_disp(f)
    assert bool(torch.isnan(u).all())  # (waits for the launch)
    with pytest.raises(_lib.CudaLibraryError, match="ran out"):
        sub.evaluate_disp(f)
    assert torch.equal(sub.evaluate_disp(f), want)


def test_solve_reports_a_wait_that_ran_out():
    """Of an operator call before the solve, and of the solve's first displacement."""
    import torch
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    nb = (64, 64)
    h = oc.self_affine(nb, (1.0, 1.0), 0.8, 0.1, seed=22)
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    kw = dict(external_force=1e-3, pentol=1e-10 * (h.max() - h.min()), forcetol=1e-13)
    first = cm.constrained_conjugate_gradients(sub, h, **kw)

    def lose_one():
        assert _lib.lib().cm_selftest_operator_barrier(sub._plan.ptr, _lib.CM_FP64, 1, 1e3) == _lib.CM_OK

    lose_one()
    sub.evaluate_disp(torch.zeros(nb, dtype=torch.float64, device="cuda")).cpu()
    with pytest.raises(_lib.CudaLibraryError, match="ran out"):
        cm.constrained_conjugate_gradients(sub, h, **kw)
    lose_one()
    with pytest.raises(_lib.CudaLibraryError, match="ran out"):
        cm.constrained_conjugate_gradients(sub, h, initial_forces=-first.jac, **kw)
    again = cm.constrained_conjugate_gradients(sub, h, **kw)
    assert np.array_equal(again.x, first.x)
