"""Timed workloads of the framework: what its users run, through its public calls.

A case is a dict of plain values.  ``op`` says which call it makes:

* ``disp`` / ``force``: one application of the Green's-function operator,
  ``substrate.evaluate_disp`` or ``substrate.evaluate_force``, on a field that
  is already on the GPU (the inner call of energy minimisers, of
  displacement post-processing and of a user's own solver loops);
* ``solve``: one contact solve under load control,
  ``constrained_conjugate_gradients``, elastic or with a hardness;
* ``batch``: many independent periodic solves of mixed sizes,
  ``constrained_conjugate_gradients_batch`` (parameter studies).

Sides are those of the test and benchmark configurations (powers of two,
3 * 2^m) and those of measured topographies, which come in any size.
"""
import math

import numpy as np
import torch

import contactmechanics_b200 as cm

YOUNG = 1.0
SIZES = (1.0, 1.0)
IMAGES = 10           # periodic images of a semi-periodic substrate (its default)
HURST, SLOPE = 0.8, 0.1
# pentol as a fraction of the height range: tight enough that a mixed-precision
# solve and an FP64 solve agree far below any physical interest
PENTOL = 1e-11
POW2 = (64, 128, 256, 512, 1024, 2048)
SMOOTH = (96, 192, 384, 768, 1536)
ODD = (75, 91, 105, 117, 135, 165, 195, 231, 275, 315, 375)
BATCH_SIDES = (64, 96, 128, 192, 256, 384, 512)


def listed():
    return [
        # the smallest call: a coarse surface inside a user's own minimiser loop
        dict(name="disp_periodic_64", op="disp", domain="periodic", nx=64, ny=64, precision="fp64"),
        # a measured map that is neither square nor a power of two
        dict(name="disp_periodic_500x300", op="disp", domain="periodic", nx=500, ny=300,
             precision="fp64"),
        # forces of a displacement field on a rectangular 3 * 2^m grid (the
        # gradient of the primal objective)
        dict(name="force_periodic_768x1536", op="force", domain="periodic", nx=768, ny=1536,
             precision="fp64"),
        # the operator benchmark's size in the fast precision
        dict(name="disp_periodic_2048_fp32", op="disp", domain="periodic", nx=2048, ny=2048,
             precision="fp32"),
        # non-periodic surface of the benchmark's size (2048^2 padded domain)
        dict(name="disp_free_1024", op="disp", domain="free", nx=1024, ny=1024, precision="fp64"),
        # the largest periodic grid that is in ordinary use
        dict(name="disp_periodic_4096", op="disp", domain="periodic", nx=4096, ny=4096,
             precision="fp64"),
        # periodic along one axis only: an odd domain of 511 x 256 points
        dict(name="disp_semi_256", op="disp", domain="semi", nx=256, ny=256, precision="fp64"),
        # Hertzian contact of a sphere from a script that holds numpy arrays
        dict(name="solve_hertz_256_host", op="solve", domain="periodic", nx=256, ny=256,
             surface="sphere", pressure=1e-3, hardness=0.0, precision="fp64", host=True),
        # the headline: a rough non-periodic 1024^2 surface in mixed precision
        dict(name="solve_free_1024_mixed", op="solve", domain="free", nx=1024, ny=1024,
             surface="rough", pressure=1e-3, hardness=0.0, precision="mixed", host=False),
        # elastic-plastic contact of a rough periodic surface
        dict(name="solve_plastic_512", op="solve", domain="periodic", nx=512, ny=512,
             surface="rough", pressure=5e-3, hardness=0.05, precision="fp64", host=False),
        # a rough measured map of odd sides on a free domain
        dict(name="solve_free_250x180", op="solve", domain="free", nx=250, ny=180,
             surface="rough", pressure=2e-3, hardness=0.0, precision="fp64", host=False),
        # a parameter study: 64 periodic solves of mixed sizes together
        dict(name="batch_64_mixed", op="batch", count=64, smallest=64, largest=512,
             pressure=1e-3, precision="mixed"),
    ]


def _log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _side(rng, low, high, op):
    """A side between low and high: a power of two, 3 * 2^m, a round number or
    an odd one.  Sides with large prime factors cost the most: one operator
    takes any odd side up to 300, a solve (hundreds of operators) odd sides
    with small factors."""
    want = _log_uniform(rng, low, high)
    kind = rng.choice(("pow2", "pow2", "smooth", "round", "odd"))
    if kind == "round":
        return max(low, 10 * round(want / 10))
    if kind == "odd" and op != "solve":
        return max(low, 2 * int(min(want, 300) / 2) + 1)
    sets = {"pow2": POW2, "smooth": SMOOTH, "odd": ODD}
    from_set = [s for s in sets[kind] if low <= s <= high]
    return min(from_set, key=lambda s: abs(math.log(s / want)))


def draw(rng):
    op = rng.choice(("disp", "disp", "force", "solve", "solve", "batch"))
    if op == "batch":
        return dict(op=op, count=rng.randint(8, 64), smallest=rng.choice((64, 96, 128)),
                    largest=rng.choice((256, 384, 512)), pressure=_log_uniform(rng, 3e-4, 3e-3),
                    precision=rng.choice(("mixed", "fp64")))
    if op == "solve":
        domain = rng.choice(("periodic", "free"))
        top = 1024 if domain == "periodic" else 512
        nx = _side(rng, 64, top, op)
        ny = nx if rng.random() < 0.5 else _side(rng, 64, top, op)
        # spheres are checks against Hertz and plastic solves branch on their
        # contact sets: both are run in FP64
        kind = rng.choice(("rough", "rough", "sphere", "plastic" if domain == "periodic" else "rough"))
        return dict(op=op, domain=domain, nx=nx, ny=ny,
                    surface="sphere" if kind == "sphere" else "rough",
                    pressure=_log_uniform(rng, 3e-4, 5e-3),
                    hardness=0.05 if kind == "plastic" else 0.0,
                    precision=rng.choice(("fp64", "mixed")) if kind == "rough" else "fp64",
                    host=rng.random() < 0.3)
    domain = rng.choice(("periodic", "periodic", "free", "semi")) if op == "disp" else "periodic"
    top = {"periodic": 2048, "free": 1024, "semi": 512}[domain]
    nx = _side(rng, 64, top, op)
    ny = nx if rng.random() < 0.5 else _side(rng, 64, top, op)
    # the force operator amplifies the shortest waves, so it is used in FP64
    return dict(op=op, domain=domain, nx=nx, ny=ny,
                precision=rng.choice(("fp64", "fp32")) if op == "disp" else "fp64")


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rough(nx, ny, seed, device):
    """A self-affine surface (flat spectrum beyond 1/8 of the size, cut off at
    4 points) with rms slope SLOPE, as an FP64 tensor."""
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    noise = torch.fft.rfft2(torch.randn((nx, ny), generator=gen, device=device,
                                        dtype=torch.float64))
    qx = torch.fft.fftfreq(nx, d=1.0 / nx, device=device, dtype=torch.float64).reshape(-1, 1)
    qy = torch.fft.rfftfreq(ny, d=1.0 / ny, device=device, dtype=torch.float64).reshape(1, -1)
    q = torch.sqrt(qx * qx + qy * qy)
    amp = q.clamp(min=8.0) ** (-(1 + HURST))
    amp[q > min(nx, ny) / 4] = 0
    amp[0, 0] = 0
    h = torch.fft.irfft2(amp * noise, s=(nx, ny))
    dx = (torch.roll(h, -1, 0) - h) * nx
    dy = (torch.roll(h, -1, 1) - h) * ny
    return h * (SLOPE / torch.sqrt(torch.mean(dx * dx + dy * dy)))


def _sphere(nx, ny, seed, device):
    """A paraboloid whose radius and centre (off the grid points) vary with the seed."""
    r = np.random.default_rng(seed)
    cx, cy = 0.5 + r.uniform(-0.5, 0.5, 2) / (nx, ny)
    x = ((torch.arange(nx, device=device, dtype=torch.float64) / nx) - cx).reshape(-1, 1)
    y = ((torch.arange(ny, device=device, dtype=torch.float64) / ny) - cy).reshape(1, -1)
    return -(x * x + y * y) / (2 * r.uniform(0.9, 1.1))


def _field(case, seed, device):
    """The operator's input: point forces of contact patches, or a displacement field."""
    s = _rough(case["nx"], case["ny"], seed, device)
    if case["op"] == "disp":
        s = -s.clamp(min=0.0) * (1e-3 / float(s.clamp(min=0.0).sum()))
    return s.to(torch.float32) if case["precision"] == "fp32" else s


def _heights(case, seed, device):
    make = _sphere if case["surface"] == "sphere" else _rough
    return make(case["nx"], case["ny"], seed, device)


def _batch_shapes(case):
    sides = [s for s in BATCH_SIDES if case["smallest"] <= s <= case["largest"]]
    return [(sides[i % len(sides)], sides[(3 * i + 1) % len(sides)]) for i in range(case["count"])]


def _batch_heights(case, seed, device):
    return [_rough(nx, ny, 1000 * seed + i, device)
            for i, (nx, ny) in enumerate(_batch_shapes(case))]


def _substrate(domain, nx, ny, precision="fp64"):
    if domain == "periodic":
        return cm.PeriodicFFTElasticHalfSpace((nx, ny), YOUNG, SIZES, precision=precision)
    if domain == "free":
        return cm.FreeFFTElasticHalfSpace((nx, ny), YOUNG, SIZES, precision=precision)
    return cm.SemiPeriodicFFTElasticHalfSpace((nx, ny), YOUNG, SIZES, n_images=IMAGES,
                                              precision=precision)


def _span(h):
    return float(h.max() - h.min())


def prepare(case, seed):
    if case["op"] in ("disp", "force"):
        sub = _substrate(case["domain"], case["nx"], case["ny"], case["precision"])
        return dict(case=case, substrate=sub, field=_field(case, seed, "cuda"))
    if case["op"] == "solve":
        h = _heights(case, seed, "cuda")
        kw = dict(external_force=case["pressure"], pentol=PENTOL * _span(h),
                  forcetol=1e-12 * case["pressure"], maxiter=20000, precision=case["precision"])
        if case["hardness"]:
            kw["hardness"] = case["hardness"] / (case["nx"] * case["ny"])
        return dict(case=case, substrate=_substrate(case["domain"], case["nx"], case["ny"]),
                    heights=h.cpu().numpy() if case["host"] else h, kw=kw)
    hs = _batch_heights(case, seed, "cuda")
    return dict(case=case, heights=hs,
                substrates=[_substrate("periodic", *h.shape) for h in hs],
                kw=dict(external_force=case["pressure"], pentol=[PENTOL * _span(h) for h in hs],
                        forcetol=1e-12 * case["pressure"], maxiter=20000,
                        precision=case["precision"]))


def _solved(results, names):
    for r in results:
        if not r.success:
            raise RuntimeError(r.message)
    return {k: [r[k] for r in results] for k in names}


def run(state):
    case = state["case"]
    if case["op"] == "disp":
        return state["substrate"].evaluate_disp(state["field"])
    if case["op"] == "force":
        return state["substrate"].evaluate_force(state["field"])
    if case["op"] == "solve":
        r = cm.constrained_conjugate_gradients(state["substrate"], state["heights"], **state["kw"])
        out = _solved([r], ["x", "jac", "active_set"] + (["plastic"] if case["hardness"] else []))
        return {k: v[0] for k, v in out.items()}
    rs = cm.constrained_conjugate_gradients_batch(state["substrates"], state["heights"],
                                                  **state["kw"])
    # the study's fields, gathered into one array each
    return {k: torch.cat([a.reshape(-1) for a in v])
            for k, v in _solved(rs, ("x", "jac", "active_set")).items()}


# ---------------------------------------------------------------------------
# compulsory work
# ---------------------------------------------------------------------------
def _domain(domain, nx, ny):
    return {"periodic": (nx, ny), "free": (2 * nx, 2 * ny), "semi": (2 * nx - 1, ny)}[domain]


def _operator_flops(nxd, nyd):
    # forward and inverse real transform (2.5 N log2 N each) and the multiply
    n = nxd * nyd
    return 5.0 * n * math.log2(n) + n


def _solve_work(domain, nx, ny, hardness):
    """Heights in, displacement, forces and contact set out; two operators and
    about thirty element operations per iteration, for the forty iterations
    that a solve needs at least at these tolerances."""
    nxd, nyd = _domain(domain, nx, ny)
    n, nd = nx * ny, nxd * nyd
    return dict(bytes=8.0 * n + 8.0 * nd + 8.0 * n + nd + (n if hardness else 0)
                + 8.0 * nxd * (nyd // 2 + 1),
                flops=40 * (2 * _operator_flops(nxd, nyd) + 30.0 * n))


def work(case):
    if case["op"] in ("disp", "force"):
        nx, ny = case["nx"], case["ny"]
        nxd, nyd = _domain(case["domain"], nx, ny)
        p = 4 if case["precision"] == "fp32" else 8
        # field in, field out, the Green's table
        return dict(bytes=float(p * (2 * nx * ny + nxd * (nyd // 2 + 1))),
                    flops=_operator_flops(nxd, nyd))
    if case["op"] == "solve":
        return _solve_work(case["domain"], case["nx"], case["ny"], case["hardness"])
    parts = [_solve_work("periodic", nx, ny, 0.0) for nx, ny in _batch_shapes(case)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------
# the same answers in plain torch and numpy
# ---------------------------------------------------------------------------
def _love(x, y, dx, dy):
    """Displacement at (x, y) of a uniformly loaded dx x dy pixel (Johnson, Contact
    Mechanics, p. 54), in extended precision: its terms cancel far from the load."""
    xp, xm, yp, ym = x + dx / 2, x - dx / 2, y + dy / 2, y - dy / 2
    pp, mp = np.sqrt(yp * yp + xp * xp), np.sqrt(ym * ym + xp * xp)
    pm, mm = np.sqrt(yp * yp + xm * xm), np.sqrt(ym * ym + xm * xm)
    v = (xp * np.log((yp + pp) / (ym + mp)) + yp * np.log((xp + pp) / (xm + pm))
         + xm * np.log((ym + mm) / (yp + pm)) + ym * np.log((xm + mm) / (xp + mp)))
    return v / (np.longdouble("3.14159265358979323846264338327950288") * np.longdouble(YOUNG))


def _greens(domain, nx, ny, device):
    """The operator's Green's function on the half spectrum, FP64."""
    nxd, nyd = _domain(domain, nx, ny)
    if domain == "periodic":
        qx = torch.fft.fftfreq(nx, d=1.0 / nx, device=device, dtype=torch.float64).abs()
        qy = torch.fft.rfftfreq(ny, d=1.0 / ny, device=device, dtype=torch.float64)
        k = math.pi * YOUNG * torch.sqrt((qx * qx).reshape(-1, 1) + (qy * qy).reshape(1, -1))
        k[0, 0] = math.pi * YOUNG  # the mean of the longest waves' stiffness along x and y
        return 1.0 / k
    lng = np.longdouble
    dx, dy = lng(1) / lng(nx), lng(1) / lng(ny)
    x = (np.arange(nxd // 2 + 1).astype(lng) * dx).reshape(-1, 1)
    y = (np.arange(nyd // 2 + 1).astype(lng) * dy).reshape(1, -1)
    images = range(-IMAGES, IMAGES + 1) if domain == "semi" else (0,)
    q = sum(_love(x, y + lng(m), dx, dy) for m in images).astype(np.float64)
    i, j = np.arange(nxd), np.arange(nyd)
    kernel = q[np.ix_(np.minimum(i, nxd - i), np.minimum(j, nyd - j))]
    return torch.fft.rfft2(torch.from_numpy(kernel).to(device)).real.contiguous()


def _displace(p, greens, nx, ny, nxd, nyd):
    """Displacements on the domain due to point pressures p on the topography."""
    return torch.fft.irfft2(torch.fft.rfft2(p, s=(nxd, nyd)) * greens, s=(nxd, nyd)) * (nx * ny)


def _exact_solve(h, domain, force, hardness):
    """Frictionless contact with 0 <= p <= hardness and a given total force, by
    conjugate gradients on the points strictly between the bounds (the upper
    one comes down to the hardness over the first iterations)."""
    nx, ny = h.shape
    nxd, nyd = _domain(domain, nx, ny)
    greens = _greens(domain, nx, ny, h.device)
    full = lambda p: _displace(p, greens, nx, ny, nxd, nyd)  # noqa: E731
    p = torch.full_like(h, force / h.numel())
    t, g_old, step = torch.zeros_like(h), 1.0, 0.0
    span = _span(h)
    for it in range(3000):
        cap = hardness * max(1.0, 16.0 * 0.9 ** it)
        p = p.clamp(max=cap)
        u = full(p)
        g = u[:nx, :ny] - h
        c = (p > 0) & (p < cap)
        offset = g[c].mean()
        g = g - offset
        small = float((g * c).abs().max()) < 1e-14 * span
        wrong = ((p == 0) & (g < -1e-14 * span)) | ((p == cap) & (g > 1e-14 * span))
        if small and cap == hardness and not bool(wrong.any()):
            break
        g2 = (g * g * c).sum()
        t = torch.where(c, g + step * (g2 / g_old) * t, torch.zeros_like(g))
        g_old = g2
        r = full(t)[:nx, :ny]
        tau = (g * t).sum() / (r * t).sum()
        p = (p - tau * t).clamp(0.0, cap)
        wrong = ((p == 0) & (g < 0)) | ((p == cap) & (g > 0))
        step = 0.0 if bool(wrong.any()) else 1.0
        p = torch.where(wrong, p - tau * g, p).clamp(0.0, cap)
        flows = p == cap
        rest = force - float(flows.sum()) * cap if math.isfinite(cap) else force
        p = torch.where(flows, p, p * (rest / p[~flows].sum())).clamp(max=cap)
    x = full(p)
    return (x, p) if bool(torch.isfinite(x).all()) else (None, None)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["op"] in ("disp", "force"):
        nx, ny = case["nx"], case["ny"]
        f = _field(case, seed, device).to(torch.float64)
        nxd, nyd = _domain(case["domain"], nx, ny)
        greens = _greens(case["domain"], nx, ny, device)
        if case["op"] == "force":
            return -torch.fft.irfft2(torch.fft.rfft2(f) / greens, s=(nx, ny)) / (nx * ny)
        return _displace(-f, greens, nx, ny, nxd, nyd)[:nx, :ny].contiguous()
    if case["op"] == "solve":
        h = _heights(case, seed, device)
        cap = case["hardness"] / h.numel() if case["hardness"] else math.inf
        x, jac = _exact_solve(h, case["domain"], case["pressure"], cap)
        return None if x is None else dict(x=x, jac=jac, active_set=None)
    solved = [_exact_solve(h, "periodic", case["pressure"], math.inf)
              for h in _batch_heights(case, seed, device)]
    return dict(x=torch.cat([x.reshape(-1) for x, _ in solved]),
                jac=torch.cat([p.reshape(-1) for _, p in solved]), active_set=None)
