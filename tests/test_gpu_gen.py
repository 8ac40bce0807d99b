"""The operator passes for sides of any length (cm_gen.cuh) against an FFT in
numpy: every radix alone and in pairs, direct stages (primes, squares of
primes, two different ones), odd and even lengths along each axis, lengths of
one and two, one axis generic and the other 2^k or 3 * 2^m, padded and odd
domains, and the longest rows and columns."""
import numpy as np
import pytest

from oracle import contact_oracle as oc

pytestmark = pytest.mark.gpu

SIDES = [(3, 5), (7, 6), (9, 10), (12, 14), (15, 16), (8, 4), (25, 49), (81, 45), (11, 13),
         (169, 22), (143, 17), (167, 2), (2, 166), (37, 74), (500, 300), (64, 75), (75, 64),
         (96, 91), (91, 96), (255, 1000), (1001, 30), (30, 1001), (2310, 20), (20, 2310)]


@pytest.mark.parametrize("nb", SIDES)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_operators(nb, precision):
    """Both operators: 1e-12 of the field's maximum in FP64 and 2e-5 in FP32, the
    bounds the transforms of the other sides are held to."""
    import torch
    import contactmechanics_b200 as cm
    tol = 1e-12 if precision == "fp64" else 2e-5
    rng = np.random.default_rng(nb[0] * 10007 + nb[1])
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), precision=precision)
    ref = oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0))
    f = rng.standard_normal(nb)
    for op in ("evaluate_disp", "evaluate_force"):
        want = getattr(ref, op)(f)
        got = getattr(sub, op)(f)
        assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
        dev = getattr(sub, op)(torch.from_numpy(f).cuda())
        assert np.max(np.abs(dev.cpu().numpy() - want)) <= tol * np.max(np.abs(want))


@pytest.mark.parametrize("nb,periodicity", [((35, 21), (False, True)), ((21, 35), (True, False)),
                                            ((84, 64), (False, True)), ((20, 33), (False, False))])
def test_semi_periodic(nb, periodicity):
    """Odd domains 2n - 1, unpadded forces."""
    import contactmechanics_b200 as cm
    rng = np.random.default_rng(5)
    f = rng.standard_normal(nb)
    sub = cm.SemiPeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), periodicity=periodicity, n_images=3)
    dom = oc.semi_periodic_domain(nb, periodicity)
    kernel = oc.semi_periodic_kernel(nb, (1.0, 1.0), 1.0, periodicity, 3, extended=True)
    area = 1.0 / (nb[0] * nb[1])
    pad = np.zeros(dom)
    pad[:nb[0], :nb[1]] = -f
    want = np.fft.irfft2(np.fft.rfft2(pad) * np.fft.rfft2(kernel), s=dom) / area
    got = sub.evaluate_disp(f, bIncludePadding=True)
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("nb", [(45, 60), (33, 100)])
def test_free_unpadded(nb):
    import contactmechanics_b200 as cm
    f = np.random.default_rng(6).standard_normal(nb)
    dom = (2 * nb[0], 2 * nb[1])
    kernel = oc.love_kernel_extended(nb, (1.0, 1.0), 1.0)
    pad = np.zeros(dom)
    pad[:nb[0], :nb[1]] = -f
    want = np.fft.irfft2(np.fft.rfft2(pad) * np.fft.rfft2(kernel), s=dom) * (nb[0] * nb[1])
    sub = cm.FreeFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    got = sub.evaluate_disp(f)
    assert np.max(np.abs(got - want[:nb[0], :nb[1]])) <= 1e-12 * np.max(np.abs(want))
    assert np.max(np.abs(sub.evaluate_disp(f, bIncludePadding=True) - want)) <= 1e-12 * np.max(np.abs(want))
    assert np.max(np.abs(sub.evaluate_disp(pad * -1) - want)) <= 1e-12 * np.max(np.abs(want))


def test_one_dimension():
    import contactmechanics_b200 as cm
    for n in (2, 3, 45, 77, 1000):
        f = np.random.default_rng(n).standard_normal(n)
        want = oc.PeriodicSubstrate((n,), 1.0, (1.0,)).evaluate_disp(f)
        got = cm.PeriodicFFTElasticHalfSpace((n,), 1.0, (1.0,)).evaluate_disp(f)
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("kind,nb", [("periodic", (64, 64)), ("periodic", (64, 1024)),
                                     ("periodic", (1024, 64)), ("periodic", (512, 512)),
                                     ("free", (32, 32)), ("free", (128, 64)), ("free", (64, 512))])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_one_launch_operator(kind, nb, precision):
    """Small domains with sides 2^k (cm_op_one.cu): repeated calls and a captured
    graph's replays leave its barrier ready for the next."""
    import torch
    import contactmechanics_b200 as cm
    from contactmechanics_b200 import _lib
    tol = 1e-12 if precision == "fp64" else 2e-5
    f = np.random.default_rng(8).standard_normal(nb)
    if kind == "free":
        dom = (2 * nb[0], 2 * nb[1])
        pad = np.zeros(dom)
        pad[:nb[0], :nb[1]] = -f
        want = np.fft.irfft2(np.fft.rfft2(pad) * np.fft.rfft2(oc.love_kernel_extended(nb, (1.0, 1.0), 1.0)),
                             s=dom)[:nb[0], :nb[1]] * (nb[0] * nb[1])
        sub = cm.FreeFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), precision=precision)
    else:
        want = oc.PeriodicSubstrate(nb, 1.0, (1.0, 1.0)).evaluate_disp(f)
        sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0), precision=precision)
    fd = torch.from_numpy(f).cuda().to(torch.float64 if precision == "fp64" else torch.float32)
    n0 = _lib.lib().cm_launch_count()
    outs = [sub.evaluate_disp(fd) for _ in range(3)]
    assert _lib.lib().cm_launch_count() - n0 == 3
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = sub.evaluate_disp(fd)
    for _ in range(3):
        captured.zero_()
        graph.replay()
        outs.append(captured.clone())
    outs.append(sub.evaluate_disp(fd))
    for u in outs:
        assert np.max(np.abs(u.double().cpu().numpy() - want)) <= tol * np.max(np.abs(want))
        assert torch.equal(u, outs[0])


@pytest.mark.parametrize("nb", [(64, 64), (45, 60), (2048, 64)])
def test_input_forms(nb):
    """Transposed, strided, other types, host tensors and arrays give what a
    contiguous CUDA tensor of the operator's type gives."""
    import torch
    import contactmechanics_b200 as cm
    sub = cm.PeriodicFFTElasticHalfSpace(nb, 1.0, (1.0, 1.0))
    f = torch.from_numpy(np.random.default_rng(9).standard_normal(nb)).cuda()
    f = f.float().double()  # values that both types hold
    want = sub.evaluate_disp(f)
    strided = torch.zeros((nb[0], 2 * nb[1]), dtype=f.dtype, device="cuda")
    strided[:, ::2] = f
    for g in (f.t().contiguous().t(), strided[:, ::2], f.float(), f.cpu()):
        assert torch.equal(sub.evaluate_disp(g), want)
    assert np.array_equal(sub.evaluate_disp(f.cpu().numpy()), want.cpu().numpy())
    assert np.array_equal(sub.evaluate_disp(np.asfortranarray(f.cpu().numpy())), want.cpu().numpy())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        again = sub.evaluate_disp(f)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(again, want)
