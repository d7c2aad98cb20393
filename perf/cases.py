"""Performance cases of the pearl_gpu library: the jobs its users give it, at the sizes they give them.

Every case is one synthetic Fe-C pearlite domain (or a batch of them): lamellar pairs of ferrite and
cementite below a growth front, austenite above it, seeded jitter of the pair widths and of the front.
`front` is the front's height as a share of the domain: a run starts with a few rows of pearlite and a
moving window later holds the front between 0.35 and 0.65.  `layer` is the length (cells) of the
carbon diffusion field that a run has built up ahead of its front, 0 at a run's start.

Kinds:
  step      one accepted step on caller-owned device planes (pearl_gpu_advance_noalloc)
  run       a restarted job: state up from host buffers, `steps` accepted steps, state down
  interval  one output interval of a long run: `steps` accepted steps, moving window check, snapshot,
            frame down to host buffers; each pass goes on from the last one's state
  sweep     a batch of independent small domains, `steps` accepted steps of each
  adjoint   gradient of a final-state misfit with respect to mobility, sigma and D_gamma
  init      initial state on the device: filling commands, interface smoothing, composition
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "fe-c_eutectoid_phase-field_simulation_b200"))

DX = 2e-9
TE_ABC = dict(A=(4724862.6373624019, 100000000.0, 172591.65731409981),
              B=(22964.296428571855, -49968654.66102279, 19450.725112218221),
              C=(-42255.03701292308, 6207741.2462954065, -42053.816371518253),
              ceq=(0.00088690859310575857, 0.25, 0.034458832049305582),
              slopes=((-4.6282639461434345e-06, -0.00031198492411304955), (0.0, 0.00010753713136114516)))


def listed():
    return [
        # the smallest call: a host program that steps a tiny domain itself, one step at a time
        dict(name="step_64x48", kind="step", nx=64, ny=48, front=0.25, layer=0.0, cooling=10.0),
        # one step of a ragged domain near the largest that this entry point takes
        dict(name="step_509x511", kind="step", nx=509, ny=511, front=0.3, layer=3.0, cooling=20.0),
        # the small configuration (4 pairs, 10 K, fixed dt)
        dict(name="run_128x256", kind="run", nx=128, ny=256, front=0.125, layer=0.0, cooling=10.0, steps=24),
        # the reference's start-up check's grid, ragged both ways
        dict(name="run_137x250", kind="run", nx=137, ny=250, front=0.4, layer=4.0, cooling=10.0, steps=24),
        # a usual production domain in its moving window, most of it pearlite
        dict(name="run_512x1024_pearlite", kind="run", nx=512, ny=1024, front=0.6, layer=6.0, cooling=15.0, steps=20),
        # a usual domain of odd size, front in the middle
        dict(name="run_1000x1537", kind="run", nx=1000, ny=1537, front=0.45, layer=6.0, cooling=20.0, steps=20),
        # the large configuration (64 pairs, 20 K, adaptive dt, moving window) at its start
        dict(name="interval_2048x4096", kind="interval", nx=2048, ny=4096, front=0.0078125, layer=0.0, cooling=20.0,
             steps=24),
        # the same, as the moving window holds it later: half pearlite, diffusion field ahead of the front
        dict(name="interval_2048x4096_window", kind="interval", nx=2048, ny=4096, front=0.5, layer=8.0, cooling=20.0,
             steps=20),
        # both mixed-precision forms together, on a domain of the size they are offered for
        dict(name="mixed_1024x2048", kind="run", nx=1024, ny=2048, front=0.4, layer=6.0, cooling=20.0, steps=20,
             precision="mixed"),
        # a parameter sweep: spacings 16..96 cells, heights 64..1024, 5..40 K
        dict(name="sweep_96", kind="sweep", n=96, steps=20),
        # the adjoint configuration's domain and dt, a shorter horizon
        dict(name="adjoint_256x512", kind="adjoint", nx=256, ny=512, front=0.0625, layer=0.0, cooling=15.0, steps=60,
             every=30),
        # initial state of a run from a filling description
        dict(name="init_384x640", kind="init", nx=384, ny=640, front=0.3, cooling=10.0, steps=50),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "run", "interval", "mixed", "sweep", "adjoint", "init"])
    c = dict(kind="run" if kind == "mixed" else kind, front=round(rng.uniform(0.02, 0.62), 4),
             layer=round(rng.choice([0.0, rng.uniform(1.0, 10.0)]), 3), cooling=round(rng.uniform(8.0, 25.0), 3))
    if kind == "step":
        c.update(nx=_log_size(rng, 48, 511), ny=_log_size(rng, 48, 511))
    elif kind in ("run", "mixed"):
        c.update(nx=_log_size(rng, 96, 1400), ny=_log_size(rng, 128, 2048), steps=rng.randint(10, 40))
        if kind == "mixed":
            c["precision"] = rng.choice(["mixed", "mixed_propose", "mixed_solve"])
    elif kind == "interval":
        c.update(nx=_log_size(rng, 1024, 2048), ny=_log_size(rng, 1536, 4000), steps=rng.randint(10, 24))
    elif kind == "sweep":
        c = dict(kind="sweep", n=rng.randint(24, 110), steps=rng.randint(8, 20), draw=rng.randrange(1 << 20))
    elif kind == "adjoint":
        steps = rng.randint(20, 60)
        c.update(nx=_log_size(rng, 96, 256), ny=_log_size(rng, 128, 512), steps=steps, every=rng.randint(10, steps))
    else:
        c = dict(kind="init", front=c["front"], cooling=c["cooling"], nx=_log_size(rng, 128, 800),
                 ny=_log_size(rng, 128, 800), steps=rng.randint(30, 60))
    return c


# ---------------------------------------------------------------- inputs
def _params(nx, ny, cooling, dt, dt_max):
    """Run parameters at `cooling` K below the eutectoid (phase-diagram slopes, fixed curvature)."""
    L = np.longdouble
    A, B, C = (list(TE_ABC[k]) for k in "ABC")
    ce, gA = TE_ABC["ceq"], np.longdouble(TE_ABC["A"][2])
    for p in (0, 1):
        dp, dg = (-L(cooling) * L(s) for s in TE_ABC["slopes"][p])
        pA = L(A[p])
        B[p] = float(L(B[p]) + 2 * (gA * dg - pA * dp))
        C[p] = float(L(C[p]) + pA * dp * (2 * L(ce[p]) + dp) - gA * dg * (2 * L(ce[2]) + dg))
    sigma = 0.5
    return dict(A=A, B=B, C=C, D=[2e-9, 2e-9, 1e-9], Vm=1e-6, epsilon=14e-9, sigma=sigma, triple=10.0,
                tau=[1.72402799784e8, 1.72402799784e8, 7.11828875478e9], dx=DX, dy=DX, dt_max=dt_max,
                dt_min=dt / 1048576.0, max_phase_change=0.04, cg_rtol=1e-11, cg_atol=1e-14, closure_tol=1e-10,
                energy_rtol=1e-11, energy_atol=1e-13 * sigma * max(nx * DX, ny * DX), cg_max=2000, max_retries=24,
                check_energy=1, phase_only=0, mu_reference=2.0 * A[2] * ce[2] + B[2])


def _pairs(nx, pairs, rng, ferrite=0.875):
    raw = (nx / pairs) * (1.0 + rng.uniform(-0.1, 0.1, size=pairs))
    edges = np.rint(np.concatenate([[0.0], np.cumsum(raw)]) * (nx / raw.sum())).astype(int)
    return [(a, max(1, int(round((b - a) * (1.0 - ferrite))))) for a, b in zip(edges[:-1], edges[1:])]


def _fields(nx, ny, front_rows, layer, prm, pairs, rng, ferrite=0.875):
    """phi [ny, nx, 3], carbon, mu [ny, nx]: tanh interfaces 4 cells wide, closed composition."""
    delta = 2.0
    xc = np.arange(nx) + 0.5
    theta = np.zeros(nx)
    for a, t in _pairs(nx, pairs, rng, ferrite):
        for img in (-nx, 0, nx):
            theta += 0.5 * (np.tanh((xc - a - img) / delta) - np.tanh((xc - a - t - img) / delta))
    theta = np.clip(theta, 0.0, 1.0)
    front = front_rows + rng.integers(-1, 2, size=nx)
    ahead = (np.arange(ny) + 0.5)[:, None] - front[None, :]
    P = 0.5 * (1.0 - np.tanh(ahead / delta))
    phi = np.empty((ny, nx, 3))
    phi[..., 0] = (1.0 - theta) * P
    phi[..., 1] = theta * P
    phi[..., 2] = 1.0 - P
    mu = np.full((ny, nx), prm["mu_reference"])
    if layer > 0:
        # carbon pushed ahead of the front: a diffusion tail of length `layer`, alternating with the lamellae
        mu += 60.0 * (0.3 + 0.7 * (theta - theta.mean())) * np.exp(-(np.abs(ahead) / (2.0 * layer)) ** 2)
    chi, c0, _ = _mixture([phi[..., k] for k in range(3)], prm)
    return phi, np.ascontiguousarray(chi * mu + c0), mu


def _scalars(carbon, dt):
    return dict(time=0.0, dt=dt, shift_distance=0.0, initial_carbon=float(carbon.sum()) * DX * DX, carbon_added=0.0,
                carbon_removed=0.0, step=0, shifts=0, rejected=0)


def _single(case, seed):
    """Parameters and host fields of a single-domain case."""
    nx, ny = case["nx"], case["ny"]
    dt = 2e-12 if case["kind"] == "adjoint" else 4e-12
    adaptive = case["kind"] != "adjoint" and not case["cooling"] <= 10.0
    prm = _params(nx, ny, case["cooling"], dt, 2 * dt if adaptive else dt)
    rng = np.random.default_rng([seed, nx, ny])
    pairs = 4 if case["kind"] == "adjoint" else max(1, nx // 32)
    front = min(max(case["front"] * ny, 10.0), ny - 12.0)
    return (prm, dt) + _fields(nx, ny, front, case["layer"], prm, pairs, rng)


def _sweep(case, seed):
    sizes, rng = np.random.default_rng([case["n"], case.get("draw", 0)]), np.random.default_rng([seed, case["n"]])
    out = []
    for _ in range(case["n"]):
        spacing, ny = int(sizes.integers(16, 97)), int(sizes.integers(64, 1025))
        ferrite, cooling = float(rng.uniform(0.85, 0.90)), float(rng.uniform(5.0, 40.0))
        layer = float(rng.choice([0.0, rng.uniform(1.0, 6.0)]))
        front = float(rng.uniform(20.0, max(22.0, 0.6 * ny)))
        nx = 2 * spacing
        prm = _params(nx, ny, cooling, 4e-12, 8e-12)
        out.append((prm, 4e-12) + _fields(nx, ny, front, layer, prm, 2, rng, ferrite))
    return out


def _commands(case, seed):
    """Filling commands: a ferrite slab with cementite lamellae of seeded positions and a cementite disc."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng([seed, nx, ny])
    top = int(case["front"] * ny) + 8
    ops = [("FILLCUBE", [0, 0, 0, 0, nx - 1, top, 0])]
    for a, t in _pairs(nx, max(1, nx // 32), rng):
        ops.append(("FILLCUBE", [1, a, 0, 0, a + t + 1, top + int(rng.integers(-2, 3)), 0]))
    ops.append(("FILLCYLINDER", [1, int(rng.integers(nx // 4, 3 * nx // 4)), top, 0, 0, 9]))
    return ops


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _pin(a):
    p = _pinned(*a.shape)
    p[...] = a
    return p


# ---------------------------------------------------------------- the program's side
def prepare(case, seed):
    import pearl_gpu

    kind = case["kind"]
    if kind == "sweep":
        ws = _sweep(case, seed)
        batch = pearl_gpu.Batch([(p, c.shape[1], c.shape[0]) for p, _, _, c, _ in ws])
        # all instances' frames in three buffers, one after another
        ends = np.cumsum([0] + [c.size for _, _, _, c, _ in ws])
        flat = [_pinned(k * int(ends[-1])) for k in (3, 1, 1)]
        out = [tuple(f[k * a:k * b].reshape(w[2 + j].shape) for j, (f, k) in enumerate(zip(flat, (3, 1, 1))))
               for w, a, b in zip(ws, ends[:-1], ends[1:])]
        return dict(case=case, batch=batch, host=[tuple(map(_pin, f)) for _, _, *f in ws],
                    scalars=[_scalars(c, dt) for _, dt, _, c, _ in ws], flat=flat, out=out)
    nx, ny = case["nx"], case["ny"]
    if kind == "init":
        prm = _params(nx, ny, case["cooling"], 4e-12, 4e-12)
        return dict(case=case, ctx=pearl_gpu.Context(prm, nx, ny), commands=_commands(case, seed),
                    mu=prm["mu_reference"], out=(_pinned(ny, nx, 3), _pinned(ny, nx), _pinned(ny, nx)))
    prm, dt, phi, carbon, mu = _single(case, seed)
    scalars = _scalars(carbon, dt)
    if kind == "step":
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (np.moveaxis(phi, -1, 0), carbon, mu)]
        return dict(case=case, lib=pearl_gpu.library(), params=pearl_gpu.PearlParams.from_dict(prm), scalars=scalars,
                    start=dev, state=[torch.empty_like(t) for t in dev])
    ctx = pearl_gpu.Context(prm, nx, ny)
    if case.get("precision"):
        ctx.set_precision(case["precision"])
    state = dict(case=case, ctx=ctx, scalars=scalars, out=(_pinned(ny, nx, 3), _pinned(ny, nx), _pinned(ny, nx)))
    if kind == "interval":
        ctx.upload(phi, carbon, mu, scalars)
    else:
        state["host"] = tuple(map(_pin, (phi, carbon, mu)))
    if kind == "adjoint":
        # the target: the front of the same lamellae, seeded rows further on
        shift = int(np.random.default_rng([seed, 7]).integers(1, 4))
        state["target"] = np.ascontiguousarray(np.concatenate([phi[:shift, :, 0], phi[:-shift, :, 0]]))
    return state


def run(state):
    import pearl_gpu

    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        for t, s in zip(state["state"], state["start"]):
            t.copy_(s)
        phi, carbon, mu = state["state"]
        s, info = pearl_gpu.PearlScalars.from_dict(state["scalars"]), pearl_gpu.PearlStepInfo()
        rc = state["lib"].pearl_gpu_advance_noalloc(
            ctypes.byref(state["params"]), case["nx"], case["ny"], ctypes.c_void_p(phi.data_ptr()),
            ctypes.c_void_p(carbon.data_ptr()), ctypes.c_void_p(mu.data_ptr()), ctypes.byref(s), 1e300,
            ctypes.byref(info), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(f"step failed: {pearl_gpu.STATUS[rc]}")
        return dict(phi=phi, carbon=carbon, mu=mu, time=s.time, retries=info.retries)
    if kind == "sweep":
        batch = state["batch"]
        for i, (host, s) in enumerate(zip(state["host"], state["scalars"])):
            batch.upload(i, *host, s)
        _, status = batch.run(case["steps"])
        if any(status):
            raise RuntimeError("an instance failed")
        end = [batch.download(i, out)[3] for i, out in enumerate(state["out"])]
        flat = state["flat"]
        return dict(phi=flat[0], carbon=flat[1], mu=flat[2], time=np.array([s.time for s in end]),
                    rejected=np.array([s.rejected for s in end]))
    ctx, out = state["ctx"], state["out"]
    if kind == "init":
        ctx.fill(state["commands"])
        ctx.smooth_interface(case["steps"], case["steps"])
        sum_c0, sum_chi = ctx.mixture_sums()
        total = ctx.init_composition(state["mu"])
        ctx.download(out)
        return dict(phi=out[0], carbon=out[1], mu=out[2], sums=np.array([sum_c0, sum_chi, total]))
    if kind == "interval":
        ctx.run(case["steps"])
        ny = case["ny"]
        ctx.maybe_shift(0.65 * ny * DX, 0.35 * ny * DX, TE_ABC["ceq"][2])
        d = ctx.snapshot()
        s = ctx.download(out)[3]
        return dict(phi=out[0], carbon=out[1], mu=out[2], time=s.time, step=s.step, shifts=s.shifts,
                    diagnostics=np.array([d.c_min, d.c_max, d.mu_min, d.mu_max, d.mass, d.energy]))
    ctx.upload(*state["host"], state["scalars"])
    if kind == "adjoint":
        rep = ctx.adjoint_gradient(case["steps"], case["every"], state["target"])
        ctx.download(out)
        return dict(phi=out[0], carbon=out[1], mu=out[2], objective=rep.objective, gradient=np.array(list(rep.grad)))
    ctx.run(case["steps"])
    s = ctx.download(out)[3]
    return dict(phi=out[0], carbon=out[1], mu=out[2], time=s.time, rejected=s.rejected)


def work(case):
    """State of five fields read and written once per step (each step's size and acceptance hang on all
    cells of the step before), about 300 operations a cell for the proposal, 150 for the energy and
    closure, and 4 conjugate-gradient iterations of 26."""
    # a sweep's instances are 112 x 544 cells on average
    cells = case["n"] * 112 * 544 if case["kind"] == "sweep" else case["nx"] * case["ny"]
    steps = case.get("steps", 1)
    if case["kind"] == "init":
        return dict(bytes=cells * (48.0 * steps + 40.0), flops=cells * 200.0 * steps)
    if case["kind"] == "adjoint":
        return dict(bytes=cells * steps * 240.0, flops=cells * steps * 1500.0)
    return dict(bytes=cells * steps * 80.0, flops=cells * steps * 560.0)


# ---------------------------------------------------------------- 64-bit values, in plain torch
def _mixture(p, prm):
    A, B, D = prm["A"], prm["B"], prm["D"]
    triple = 2.0 * p[0] * p[1] * p[2]
    chi = c0 = K = 0.0
    for k in range(3):
        h = p[k] * p[k] * (3.0 - 2.0 * p[k]) + triple
        x = 1.0 / (2.0 * A[k])
        chi = chi + h * x
        c0 = c0 - h * x * B[k]
        K = K + p[k] * D[k] * x
    return chi, c0, K


def _diff(f, axis):
    """f of the next cell minus f: periodic in x (axis 1), without the wall faces in y (axis 0)."""
    return f.roll(-1, 1) - f if axis == 1 else f[1:] - f[:-1]


def _operator(K, chi, dt, prm):
    wx = 0.5 * (K + K.roll(-1, 1)) / prm["dx"] ** 2
    wy = 0.5 * (K[1:] + K[:-1]) / prm["dy"] ** 2

    def flux(u):  # sum over a cell's faces of w (u_neighbour - u)
        fx, fy = wx * _diff(u, 1), wy * _diff(u, 0)
        out = fx - fx.roll(1, 1)
        out[:-1] += fy
        out[1:] -= fy
        return out

    w = wx + wx.roll(1, 1)
    w[:-1] += wy
    w[1:] += wy
    return (lambda u: chi * u - dt * flux(u)), flux, chi + dt * w


def _cg(apply, diag, rhs, x, tol, most):
    r = rhs - apply(x)
    z = r / diag
    p, rz = z, (r * z).sum()
    for _ in range(most):
        if float((r * r).sum().sqrt()) <= tol:
            break
        Ap = apply(p)
        a = rz / (p * Ap).sum()
        x, r = x + a * p, r - a * Ap
        z = r / diag
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
    return x


class _Solve(torch.autograd.Function):
    """u of A(K, chi) u = rhs, started from x0."""

    @staticmethod
    def forward(ctx, K, chi, rhs, x0, dt, prm, tol):
        A, _, diag = _operator(K, chi, dt, prm)
        u = _cg(A, diag, rhs, x0, tol, prm["cg_max"])
        ctx.save_for_backward(K, chi, u)
        ctx.more = (dt, prm)
        return u

    @staticmethod
    def backward(ctx, g):
        K, chi, u = ctx.saved_tensors
        dt, prm = ctx.more
        A, _, diag = _operator(K, chi, dt, prm)
        lam = _cg(A, diag, g, torch.zeros_like(g), 1e-13 * float(g.norm()), 500)
        with torch.enable_grad():
            k, c = K.detach().requires_grad_(), chi.detach().requires_grad_()
            gK, gc = torch.autograd.grad(-(lam * _operator(k, c, dt, prm)[0](u)).sum(), (k, c))
        return gK, gc, lam, None, None, None, None


def _capillary(p, prm, sigma):
    """Interface part of the phase forces."""
    eps = prm["epsilon"]
    obs, tr = 16.0 * sigma / (math.pi ** 2 * eps), prm["triple"] / eps
    f = [obs * (p[(a + 1) % 3] + p[(a + 2) % 3]) + tr * p[(a + 1) % 3] * p[(a + 2) % 3] for a in range(3)]
    ny = p[0].shape[0]
    for axis, back, d2 in ((1, 1, prm["dx"] ** 2), (1, -1, prm["dx"] ** 2), (0, 1, prm["dy"] ** 2), (0, -1, prm["dy"] ** 2)):
        n = [q.roll(back, axis) for q in p]
        keep = torch.ones(ny, 1, dtype=p[0].dtype, device=p[0].device)
        if axis == 0:
            keep[0 if back == 1 else ny - 1] = 0.0
        for a in range(3):
            for b in range(a + 1, 3):
                w = keep * (2.0 * eps * sigma / d2) * (p[a] * n[b] - n[a] * p[b])
                f[a] = f[a] + w * n[b]
                f[b] = f[b] - w * n[a]
    return f


def _simplex(z):
    s, _ = torch.sort(torch.stack(z), dim=0, descending=True)
    th = s[0] - 1.0
    t2, t3 = (s[0] + s[1] - 1.0) / 2.0, (s[0] + s[1] + s[2] - 1.0) / 3.0
    th = torch.where(s[1] > t2, t2, th)
    th = torch.where(s[2] > t3, t3, th)
    return [torch.clamp(q - th, min=0.0) for q in z]


def _propose(p, mu, dt, prm, M, sigma):
    f = _capillary(p, prm, sigma)
    psi = [prm["C"][k] - 0.25 / prm["A"][k] * (mu - prm["B"][k]) ** 2 for k in range(3)]
    for a in range(3):
        for b in range(2):
            dh = 2.0 * p[(a + 1) % 3] * p[(a + 2) % 3] + (6.0 * p[b] * (1.0 - p[b]) if a == b else 0.0)
            f[a] = f[a] + (psi[b] - psi[2]) * dh / prm["Vm"]
    mean = (f[0] + f[1] + f[2]) / 3.0
    w = [p[0] * p[1], p[0] * p[2], p[1] * p[2]]
    ws = w[0] + w[1] + w[2]
    some = ws > 1e-30
    tau = torch.where(some, sum(x * t for x, t in zip(w, prm["tau"])) / torch.where(some, ws, torch.ones_like(ws)),
                      torch.full_like(ws, min(prm["tau"])))
    s = M * dt / (tau * prm["epsilon"])
    return _simplex([q - s * (x - mean) for q, x in zip(p, f)])


def _energy(p, c, prm):
    chi, c0, _ = _mixture(p, prm)
    icpt = chi * prm["mu_reference"] + c0
    psi = [prm["C"][k] - 0.25 / prm["A"][k] * (prm["mu_reference"] - prm["B"][k]) ** 2 for k in range(3)]
    triple = 2.0 * p[0] * p[1] * p[2]
    e = 0.5 * (c - icpt) ** 2 / chi
    for k in range(2):
        e = e + (p[k] * p[k] * (3.0 - 2.0 * p[k]) + triple) * (psi[k] - psi[2])
    return (e / prm["Vm"]).sum() * prm["dx"] * prm["dy"] + _interface_energy(p, prm)


def _interface_energy(p, prm):
    eps, sigma = prm["epsilon"], prm["sigma"]
    obs, tr = 16.0 * sigma / (math.pi ** 2 * eps), prm["triple"] / eps
    e = (obs * (p[0] * p[1] + p[0] * p[2] + p[1] * p[2]) + tr * p[0] * p[1] * p[2]).sum()
    for a in range(3):
        for b in range(a + 1, 3):
            zx = (p[a] * p[b].roll(-1, 1) - p[a].roll(-1, 1) * p[b]) / prm["dx"]
            zy = (p[a][:-1] * p[b][1:] - p[a][1:] * p[b][:-1]) / prm["dy"]
            e = e + eps * sigma * ((zx * zx).sum() + (zy * zy).sum())
    return e * prm["dx"] * prm["dy"]


def _valid(p, c, mu, prm):
    """Carbon, and each present phase's carbon at mu, within [0, 1]."""
    ok = bool(((c >= -1e-10) & (c <= 1 + 1e-10)).all())
    for k in range(3):
        ck = (mu - prm["B"][k]) / (2.0 * prm["A"][k])
        ok = ok and bool(((p[k] <= 0.01) | ((ck >= -1e-10) & (ck <= 1 + 1e-10))).all())
    return ok


def _advance(p, c, mu, dt0, prm, energy0, M=1.0, sigma=None, grad=False):
    """One accepted step: (p, c, mu, accepted dt, energy, rejected attempts)."""
    dt, rejected = min(dt0, prm["dt_max"]), 0
    while True:
        q = _propose(p, mu, dt, prm, M, prm["sigma"] if sigma is None else sigma)
        if max(float((a - b).detach().abs().max()) for a, b in zip(q, p)) <= prm["max_phase_change"]:
            chi, c0, K = _mixture(q, prm)
            icpt = chi * prm["mu_reference"] + c0
            rhs = c - icpt
            tol = prm["cg_atol"] + prm["cg_rtol"] * float(rhs.detach().norm())
            x0 = (mu - prm["mu_reference"]).detach()
            u = _Solve.apply(K, chi, rhs, x0, dt, prm, tol)
            if grad:
                return q, icpt + chi * u, prm["mu_reference"] + u, dt, energy0, rejected
            cn = c + dt * _operator(K, chi, dt, prm)[1](u)
            mn = prm["mu_reference"] + (cn - icpt) / chi
            e = float(_energy(q, cn, prm))
            if _valid(q, cn, mn, prm) and e <= energy0 + prm["energy_atol"] + prm["energy_rtol"] * abs(energy0):
                return q, cn, mn, dt, e, rejected
        dt, rejected = 0.5 * dt, rejected + 1


def _steps(prm, dt, phi, carbon, mu, steps, dev):
    p = [torch.from_numpy(np.ascontiguousarray(phi[..., k])).to(dev) for k in range(3)]
    c, m = torch.from_numpy(carbon).to(dev), torch.from_numpy(mu).to(dev)
    t, rejected, e = 0.0, 0, float(_energy(p, c, prm))
    for _ in range(steps):
        p, c, m, used, e, rej = _advance(p, c, m, dt, prm, e)
        t, rejected, dt = t + used, rejected + rej, min(1.1 * used, prm["dt_max"])
    return p, c, m, t, rejected, e


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    with torch.no_grad():
        if kind == "init":
            return _exact_init(case, seed, dev)
        if kind == "sweep":
            ends = [_steps(*w, case["steps"], dev) for w in _sweep(case, seed)]
            return dict(phi=torch.cat([torch.stack(e[0], -1).reshape(-1) for e in ends]),
                        carbon=torch.cat([e[1].reshape(-1) for e in ends]), mu=torch.cat([e[2].reshape(-1) for e in ends]),
                        time=np.array([e[3] for e in ends]), rejected=np.array([e[4] for e in ends]))
        prm, dt, phi, carbon, mu = _single(case, seed)
        if kind != "adjoint":
            p, c, m, t, rejected, e = _steps(prm, dt, phi, carbon, mu, case.get("steps", 1), dev)
            out = dict(phi=torch.stack(p, 0 if kind == "step" else -1), carbon=c, mu=m, time=t)
            if kind == "interval":
                out.update(step=case["steps"], shifts=0, diagnostics=np.array(
                    [float(v) for v in (c.min(), c.max(), m.min(), m.max(), c.sum() * DX * DX, e)]))
            else:
                out["retries" if kind == "step" else "rejected"] = rejected
            return out
    shift = int(np.random.default_rng([seed, 7]).integers(1, 4))
    target = torch.from_numpy(np.concatenate([phi[:shift, :, 0], phi[:-shift, :, 0]])).to(dev)
    p = [torch.from_numpy(np.ascontiguousarray(phi[..., k])).to(dev) for k in range(3)]
    c, m = torch.from_numpy(carbon).to(dev), torch.from_numpy(mu).to(dev)
    M, sigma, Dg = (torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)
                    for v in (1.0, prm["sigma"], prm["D"][2]))
    prm = dict(prm, D=[prm["D"][0], prm["D"][1], Dg])
    for _ in range(case["steps"]):
        p, c, m, _, _, _ = _advance(p, c, m, dt, prm, 0.0, M, sigma, grad=True)
    J = ((p[0] - target) ** 2).sum()
    g = torch.autograd.grad(J, (M, sigma, Dg))
    return dict(phi=torch.stack(p, -1).detach(), carbon=c.detach(), mu=m.detach(), objective=float(J.detach()),
                gradient=np.array([float(v) for v in g]))


def _exact_init(case, seed, dev):
    nx, ny = case["nx"], case["ny"]
    prm = _params(nx, ny, case["cooling"], 4e-12, 4e-12)
    x, y = np.arange(nx)[None, :], np.arange(ny)[:, None]
    label = np.full((ny, nx), 2)
    for name, v in _commands(case, seed):
        if name == "FILLCUBE":
            inside = (x >= v[1]) & (x <= v[4]) & (y >= v[2]) & (y <= v[5])
        else:
            inside = (x - v[1]) ** 2 + (y - v[2]) ** 2 <= v[5] ** 2
        label[inside] = v[0]
    p = [torch.from_numpy((label == k).astype(np.float64)).to(dev) for k in range(3)]
    base = 0.12 * DX * DX / (prm["epsilon"] * prm["sigma"])
    before = first = float(_interface_energy(p, prm))
    for _ in range(case["steps"]):
        f = _capillary(p, prm, prm["sigma"])
        mean = (f[0] + f[1] + f[2]) / 3.0
        f = [a - mean for a in f]
        scale = min(base, 0.02 / max(float(a.abs().max()) for a in f))
        while True:
            q = _simplex([a - scale * b for a, b in zip(p, f)])
            e = float(_interface_energy(q, prm))
            if e <= before + 1e-14 * max(1.0, abs(before), abs(first)):
                break
            scale *= 0.5
        p, before = q, e
    chi, c0, _ = _mixture(p, prm)
    mu = torch.full((ny, nx), prm["mu_reference"], dtype=torch.float64, device=dev)
    c = chi * mu + c0
    return dict(phi=torch.stack(p, -1), carbon=c, mu=mu,
                sums=np.array([float(c0.sum()), float(chi.sum()), float(c.sum()) * DX * DX]))
