"""The workloads that performance work on this repository is measured on.

A case is one modelling call as a user's program makes it through
``tide_b200``: a 2-D TM forward run, a forward + gradient evaluation, a
tangent (``linearize(...).jvp``), a Debye-medium gradient, a 3-D Yee forward
run or gradient.  The listed cases span the range the repository's own
workloads cover (96 x 96 with one shot up to 1024 x 2048 with many shots, 128^3
in 3-D, FP32 and BF16 snapshots, device and checkpoint storage, stencils 2 and
4); ``draw`` gives more of the same ranges, stencils 6 and 8 and FP64 among
them.

``exact`` restates the physics in plain torch in 64 bits (CPML Yee stepping,
gradients by autograd through the time loop), independent of the package.
"""

from __future__ import annotations

import math
import pathlib
import sys

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

ROOT = pathlib.Path.cwd()
sys.path.insert(0, str(ROOT / "tide-gpr_b200"))

import tide_b200 as tide  # noqa: E402

EP0 = 8.8541878128e-12
MU0 = 1.2566370614359173e-06
C0 = 1.0 / math.sqrt(EP0 * MU0)
DX = 0.02  # grid spacing (m)
NOISE = 5  # half width of the box smoothing of the model's random part (cells)


def _tm(name, kind, ny, nx, shots, nt, *, pml=20, n_rec=64, stencil=2, dtype="float32",
        storage="device", compression="none", k=1):
    c = dict(kind=kind, ny=ny, nx=nx, shots=shots, nt=nt, pml=pml, n_rec=n_rec, stencil=stencil,
             dtype=dtype, storage=storage, compression=compression, k=k)
    return dict(c, name=name) if name else c


def _em3d(name, kind, nz, ny, nx, shots, nt, *, pml=12, n_rec=64, stencil=2,
          storage="checkpoint", compression="bf16"):
    c = dict(kind=kind, nz=nz, ny=ny, nx=nx, shots=shots, nt=nt, pml=pml, n_rec=n_rec,
             stencil=stencil, dtype="float32", storage=storage, compression=compression, k=1)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the plain single-shot model a user tries first (96 x 96, CPML 10, one receiver)
        _tm("fwd_single_shot", "forward", 96, 96, 1, 300, pml=10, n_rec=1),
        # a small survey simulated from an odd-sized model
        _tm("fwd_survey_ragged", "forward", 301, 487, 6, 600, n_rec=97),
        # synthetic data for the widest models of the served range, many shots at once
        _tm("fwd_survey_large", "forward", 1024, 2048, 16, 200, n_rec=256),
        # one inversion iteration on a small crop, two shots
        _tm("grad_crop", "gradient", 120, 160, 2, 400, n_rec=40),
        # one shot batch of the inversion the benchmark times, shortened in nt
        _tm("grad_batch", "gradient", 512, 1024, 8, 320, n_rec=256),
        # compressed snapshots, every second step imaged, odd sizes
        _tm("grad_bf16_k2", "gradient", 389, 701, 5, 500, n_rec=128, compression="bf16", k=2),
        # a record too long for a stored history: checkpoint and recompute
        _tm("grad_checkpoint", "gradient", 512, 1024, 4, 400, n_rec=256, storage="checkpoint"),
        # fourth-order stencil
        _tm("grad_order4", "gradient", 256, 384, 4, 300, n_rec=96, stencil=4),
        # a Gauss-Newton product: linearise once, apply the Jacobian to a direction
        _tm("jvp", "jvp", 256, 512, 4, 300, n_rec=128),
        # dispersive ground, gradients in eps_inf, sigma, delta_eps and tau
        _tm("grad_debye", "debye", 768, 1536, 4, 96, pml=30, n_rec=256, storage="checkpoint"),
        # 3-D simulation of a box with unequal sides
        _em3d("fwd_3d", "forward3d", 90, 111, 125, 2, 120),
        # 3-D inversion batch on 128^3, BF16 snapshots recomputed per segment
        _em3d("grad_3d", "gradient3d", 128, 128, 128, 4, 64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward"] * 3 + ["gradient"] * 5 + ["jvp", "debye", "forward3d", "gradient3d"])
    if kind in ("forward3d", "gradient3d"):
        nz, ny, nx = (_log(rng, 40, 128) for _ in range(3))
        shots = rng.randint(1, 4)
        return _em3d(None, kind, nz, ny, nx, shots, rng.randint(24, 64), pml=rng.choice([8, 12]),
                     n_rec=rng.randint(1, 64), stencil=rng.choice([2, 2, 2, 4]),
                     storage=rng.choice(["checkpoint", "device"]) if shots < 3 else "checkpoint")
    hi_y, hi_x = {"forward": (1024, 2048), "debye": (768, 1536)}.get(kind, (640, 1280))
    ny, nx = _log(rng, 96, hi_y), _log(rng, 96, hi_x)
    shots = _log(rng, 1, {"forward": 16, "debye": 4, "jvp": 4}.get(kind, 8))
    nt = {"debye": rng.randint(40, 96), "jvp": rng.randint(100, 300)}.get(kind, rng.randint(150, 600))
    stencil = rng.choice([2, 2, 2, 2, 2, 4, 6, 8]) if kind in ("forward", "gradient") else 2
    dtype = rng.choice(["float32"] * 7 + ["float64"]) if kind in ("forward", "gradient") else "float32"
    compression = rng.choice(["none", "none", "bf16"]) if kind == "gradient" and dtype == "float32" else "none"
    storage = rng.choice(["device", "device", "checkpoint"]) if kind == "gradient" else (
        "checkpoint" if kind == "debye" else "device")
    # no dearer than the largest listed case of its kind (cell-steps), nor more than 12 GB of history
    most = {"forward": 7e9, "gradient": 1.6e9, "jvp": 2e8, "debye": 4.5e8}[kind]
    if stencil != 2 or dtype != "float32":
        most /= 6
    cells = (ny + 41) * (nx + 41) * shots
    nt = max(24, min(nt, int(most / cells)))
    return _tm(None, kind, ny, nx, shots, nt, pml=rng.choice([10, 20, 20]), n_rec=rng.randint(1, 256),
               stencil=stencil, dtype=dtype, storage=storage, compression=compression,
               k=rng.choice([1, 1, 1, 2, 3]) if kind == "gradient" else 1)


# ------------------------------------------------------------------ inputs


def _smooth(u, n):
    """Box mean of half width NOISE over the last n axes (edges replicated)."""
    for a in range(n):
        u = u.movedim(u.ndim - 1 - a, -1)
        shape = u.shape
        v = F.pad(u.reshape(1, -1, shape[-1]), (NOISE, NOISE), mode="replicate")
        u = F.avg_pool1d(v, 2 * NOISE + 1, 1).reshape(shape)
        u = u.movedim(-1, u.ndim - 1 - a)
    return u


def _layers(g, shape, lo, hi):
    n = shape[0]
    v = lo + (hi - lo) * torch.rand(6, generator=g, device="cuda", dtype=torch.float64)
    rows = torch.clamp(torch.arange(n, device="cuda") * 6 // n, max=5)
    return v[rows].reshape(-1, *([1] * (len(shape) - 1))).expand(shape)


def _inputs(case, seed):
    """Model, acquisition and source wavelets, on the GPU, in the case's dtype."""
    g = torch.Generator(device="cuda").manual_seed(7919 * int(seed) + 17)
    three = "nz" in case
    shape = (case["nz"], case["ny"], case["nx"]) if three else (case["ny"], case["nx"])
    nd = len(shape)
    dtype = getattr(torch, case["dtype"])
    S, nt = case["shots"], case["nt"]

    def noise(scale):
        return scale * _smooth(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64), nd)

    def field(lo, hi):
        u = _smooth(torch.rand(shape, generator=g, device="cuda", dtype=torch.float64), nd)
        u = (u - u.min()) / (u.max() - u.min())
        return lo + (hi - lo) * u

    d = {}
    if case["kind"] == "debye":
        eps, sig = field(3.0, 10.0), field(0.0, 0.002)
        d["deps"], d["tau"] = field(0.1, 5.0).to(dtype), field(2e-10, 1e-9).to(dtype)
    else:
        eps = (_layers(g, shape, 3.0, 16.0 if three else 25.0) + noise(3.0)).clamp(min=1.5)
        sig = _layers(g, shape, 0.0, 0.005 if three else 0.01) + noise(1e-3).abs()
    d["eps"], d["sig"] = eps.to(dtype), sig.to(dtype)
    d["mu"] = torch.ones(shape, device="cuda", dtype=dtype)
    csum = {2: 1.0, 4: 9 / 8 + 1 / 24, 6: 75 / 64 + 25 / 384 + 3 / 640,
            8: 1225 / 1024 + 245 / 3072 + 49 / 5120 + 5 / 7168}[case["stencil"]]
    vmax = C0 / math.sqrt(float(d["eps"].min()))
    d["dt"] = 0.9 * DX / (math.sqrt(nd) * vmax) / csum
    freq = (500e6 if three else 400e6) * (0.9 + 0.2 * torch.rand(S, generator=g, device="cuda",
                                                                dtype=torch.float64))
    t = torch.arange(nt, device="cuda", dtype=torch.float64) * d["dt"]
    ph = (math.pi * freq[:, None] * (t[None] - 1.0 / freq[:, None])).square()
    d["amp"] = ((1 - 2 * ph) * torch.exp(-ph)).reshape(S, 1, nt).to(dtype)
    # one source a shot along a line near the surface from edge to edge, receivers on the
    # same line (2-D) or above the source (3-D)
    top = min(3 if three else 10, shape[0] // 4)

    def line(n, first, extent):
        i = torch.arange(n, device="cuda")
        return first + i * (extent - 2 * first - 1) // max(1, n - 1)

    jit = torch.randint(0, 3, (S,), generator=g, device="cuda")
    row = torch.full((S,), top, device="cuda")
    if three:
        src = torch.stack([row, line(S, 8, shape[1]) + jit, line(S, 8, shape[2])], -1)
        i = torch.arange(case["n_rec"], device="cuda")
        side = max(1, math.isqrt(case["n_rec"]))
        off = torch.stack([torch.zeros_like(i), i // side * 4, i % side * 3], -1)
        rec = (src[:, None] * torch.tensor([0, 1, 1], device="cuda") + off[None]) % torch.tensor(
            shape, device="cuda")
    else:
        src = torch.stack([row, line(S, 8, shape[1]) + jit], -1)
        i = line(case["n_rec"], 12, shape[1])
        rec = torch.stack([torch.full_like(i, top), i], -1)[None].expand(S, -1, -1)
    d["src"] = src[:, None].contiguous()
    d["rec"] = rec.contiguous()
    if case["kind"] == "jvp":
        d["v_eps"], d["v_sig"] = noise(1.0).to(dtype), noise(1e-3).to(dtype)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    comp = "ez" if "nz" in case else "ey"
    op = tide.Maxwell3D if "nz" in case else tide.MaxwellTM
    storage = tide.StorageOptions(
        mode=tide.StorageMode(case["storage"]),
        compression="bf16" if case["compression"] == "bf16" else False)
    d["op"] = op(
        tide.Discretization(DX, d["dt"], stencil=case["stencil"], boundary=tide.CPML(case["pml"])),
        tide.Experiment(tide.Acquisition(d["src"], d["rec"]), d["amp"], source_component=comp,
                        receiver_component=comp),
        storage=storage, model_gradient_sampling_interval=case["k"])
    d["kind"] = case["kind"]
    if case["kind"] == "jvp":
        d["direction"] = tide.EMDirection(d["v_eps"], d["v_sig"])
    return d


def _state(s):
    return [getattr(s, n) for n in s.__slots__]


def run(d):
    kind, op = d["kind"], d["op"]
    if kind in ("forward", "forward3d"):
        res = op(tide.EMModel(d["eps"], d["sig"], d["mu"]))
        return [res.receiver_data, *_state(res.final_state)]
    if kind == "jvp":
        lin = op.linearize(tide.EMModel(d["eps"], d["sig"], d["mu"]))
        tan = lin.jvp(d["direction"])
        return [lin.primal.receiver_data, tan.receiver_data, *_state(tan.final_state)]
    leaves = [d["eps"].detach().clone().requires_grad_(True), d["sig"].detach().clone().requires_grad_(True)]
    disp = None
    if kind == "debye":
        leaves += [d["deps"].detach().clone().requires_grad_(True), d["tau"].detach().clone().requires_grad_(True)]
        disp = tide.DebyeDispersion(leaves[2], leaves[3])
    r = op(tide.EMModel(leaves[0], leaves[1], d["mu"], disp)).receiver_data
    (0.5 * (r * r).sum()).backward()
    return [r.detach(), *[t.grad for t in leaves]]


# ------------------------------------------------------------------ work, tolerance


def _padded(case):
    return [case[n] + 2 * case["pml"] + case["stencil"] - 1 for n in ("nz", "ny", "nx") if n in case]


def work(case):
    item = 8 if case["dtype"] == "float64" else 4
    three = "nz" in case
    model = math.prod(case[n] for n in ("nz", "ny", "nx") if n in case)
    cells = math.prod(_padded(case)) * case["shots"]
    P = case["stencil"] // 2
    # per cell and step: H and E half steps (differences of P terms, coefficient
    # products), the adjoint half steps, and the two image terms
    fwd = (6 * 2 if three else 4) * (3 * P) + (18 if three else 8)
    adj = fwd + (12 if three else 6)
    per = {"forward": fwd, "forward3d": fwd, "gradient": fwd + adj, "gradient3d": fwd + adj,
           "jvp": 2 * fwd + 4, "debye": fwd + adj + 30}[case["kind"]]
    records = case["nt"] * case["shots"] * (1 + case["n_rec"])
    state = (18 if three else 7) * math.prod(
        case[n] + 2 * case["pml"] for n in ("nz", "ny", "nx") if n in case) * case["shots"]
    io = {"forward": 3 * model + state, "forward3d": 3 * model + state, "gradient": 5 * model,
          "gradient3d": 5 * model, "jvp": 5 * model + state + records, "debye": 9 * model}[case["kind"]]
    return {"bytes": item * (io + records), "flops": per * cells * case["nt"]}


def tolerance(case):
    if case["dtype"] == "float64":
        return {"rel": 1e-11}
    if case["compression"] == "bf16" and case["kind"] in ("gradient", "gradient3d"):
        # snapshots rounded to 8 bits before they are imaged
        return {"rel": 2e-2}
    # the loosest outputs against 64 bits: CPML memories of a strip the wave has hardly
    # reached (1.4e-4); gradients 2e-5
    return {"rel": 2e-4 if case["kind"] in ("forward", "forward3d") else 1e-4}


# ------------------------------------------------------------------ 64-bit restatement

_FD = {2: [1.0], 4: [9 / 8, -1 / 24], 6: [75 / 64, -25 / 384, 3 / 640],
       8: [1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168]}


def _cpml(n, P, width, dt, max_pml, half):
    """(a, b, kappa) of one axis on integer or half points."""
    x = torch.arange(n, device="cuda", dtype=torch.float64) + (0.5 if half else 0.0)
    a, b, k = torch.zeros_like(x), torch.zeros_like(x), torch.ones_like(x)
    if width == 0:
        return a, b, k
    s0 = 5 / (150.0 * math.pi * DX)
    for dist in (P + width - x, x - (n - 1 - (P - 1) - width)):
        frac = (dist / width).clamp(0, 1)
        sig, kap, alp = s0 * frac**4, 1 + 4 * frac**4, 0.008 * (1 - frac) + 0.0008
        bb = torch.exp(-(sig / kap + alp) * dt / EP0)
        aa = sig * (bb - 1) / (kap * (sig + kap * alp) + 1e-9)
        inside = dist >= 0
        a = torch.where(inside, torch.where(sig > 1e-6, aa, 0.0), a)
        b, k = torch.where(inside, bb, b), torch.where(inside, kap, k)
    return a, b, k


class _Grid:
    """Differences on the update domain [P, n - P + 1) of each axis, with their
    CPML memories; arrays are [S, *shape]."""

    def __init__(self, case, dt):
        self.P = case["stencil"] // 2
        self.c = _FD[case["stencil"]]
        self.shape = _padded(case)
        self.nd = len(self.shape)
        self.prof = {}
        for ax, n in enumerate(self.shape):
            for half in (False, True):
                view = [1] * (self.nd + 1)
                view[ax + 1] = n
                p = _cpml(n, self.P, case["pml"], dt, case["pml"] * DX, half)
                self.prof[ax, half] = [v.reshape(view) for v in p]

    def inner(self, t, ax, half):
        """t on the domain, with the last plane of `ax` left out for half points."""
        for a, n in enumerate(self.shape):
            hi = n - self.P + (0 if (half and a == ax) else 1)
            if t.shape[a + 1] > 1:
                t = t.narrow(a + 1, self.P, hi - self.P)
        return t

    def outer(self, t, ax, half):
        pad = []
        for a in reversed(range(self.nd)):
            pad += [self.P, self.P - 1 + (1 if (half and a == ax) else 0)]
        return F.pad(t, pad)

    def diff(self, f, ax, half):
        P, n = self.P, self.shape[ax]
        ln = n - 2 * P + (0 if half else 1)
        for a, m in enumerate(self.shape):
            if a != ax:
                f = f.narrow(a + 1, P, m - 2 * P + 1)
        out = 0.0
        for m, c in enumerate(self.c):
            lo, hi = (P - m, P + m + 1) if half else (P - m - 1, P + m)
            out = out + c * (f.narrow(ax + 1, hi, ln) - f.narrow(ax + 1, lo, ln))
        return out / DX

    def step(self, f, mem, ax, half):
        """CPML difference of f along ax (full array) and its new memory."""
        d = self.diff(f, ax, half)
        a, b, k = (self.inner(v, ax, half) for v in self.prof[ax, half])
        mem = b * mem + a * d
        return self.outer(d / k + mem, ax, half), mem

    def zeros(self, S, ax, half):
        z = torch.zeros((S, *self.shape), device="cuda", dtype=torch.float64)
        return self.inner(z, ax, half).contiguous()

    def crop(self, t):
        for a, n in enumerate(self.shape):
            t = t.narrow(a + 1, self.P, n - 2 * self.P + 1)
        return t


def _replicate(t, pad):
    """Replicate-pad by P + width below and P - 1 + width above on every axis."""
    for a in range(t.ndim):
        n = t.shape[a]
        i = (torch.arange(-pad[0], n + pad[1], device=t.device)).clamp(0, n - 1)
        t = t.index_select(a, i)
    return t


def _coefs(eps, sig, mu, dt):
    u = sig * dt / (2 * eps * EP0)
    return (1 - u) / (1 + u), dt / (eps * EP0) / (1 + u), dt / (mu * MU0)


def _flat(loc, shape, off):
    i = 0
    for a, n in enumerate(shape):
        i = i * n + loc[..., a] + off
    return i


def _add(f, idx, v):
    return f.reshape(f.shape[0], -1).scatter_add(1, idx, v).reshape(f.shape)


def _loop(step, state, nt, grads):
    """Runs step(t, *state) -> (state, r); with gradients in checkpointed segments."""
    seg = max(1, int(math.sqrt(nt)) // 2)

    def part(t0, n, *s):
        rs = []
        for t in range(t0, t0 + n):
            s, r = step(t, *s)
            rs.append(r)
        return (*s, torch.stack(rs))

    out = []
    for t0 in range(0, nt, seg):
        n = min(seg, nt - t0)
        res = checkpoint(part, t0, n, *state, use_reentrant=False) if grads else part(t0, n, *state)
        state, r = res[:-1], res[-1]
        out.append(r)
    return state, torch.cat(out)


def _exact_tm(case, d):
    kind, S, nt = case["kind"], case["shots"], case["nt"]
    G = _Grid(case, d["dt"])
    P, dt = G.P, d["dt"]
    pad = (P + case["pml"], P - 1 + case["pml"])
    leaves = [d["eps"], d["sig"]] + ([d["deps"], d["tau"]] if kind == "debye" else [])
    grads = kind in ("gradient", "debye")
    leaves = [t.double().requires_grad_(grads) for t in leaves]
    eps, sig, mu = (_replicate(t, pad) for t in (leaves[0], leaves[1], d["mu"].double()))
    da = db = dcp = None
    if kind == "debye":
        de, tau = (_replicate(t, pad) for t in leaves[2:])
        da = (2 * tau - dt) / (2 * tau + dt)
        db = EP0 * de * dt / (2 * tau + dt)
        den = eps * EP0 + sig * dt / 2 + db
        ca, cb, cq = (eps * EP0 - sig * dt / 2 - db) / den, dt / den, dt / (mu * MU0)
        dcp = (1 - da) / den
    else:
        ca, cb, cq = _coefs(eps, sig, mu, dt)
    src = _flat(d["src"], G.shape, pad[0])
    rec = _flat(d["rec"], G.shape, pad[0])
    f = d["amp"].double().permute(2, 0, 1) * cb.reshape(-1)[src] * (-1.0 / DX**2)
    dom = torch.zeros((1, *G.shape), device="cuda", dtype=torch.float64)
    dom[:, P:G.shape[0] - P + 1, P:G.shape[1] - P + 1] = 1.0
    if kind == "jvp":
        zp = [pad[0], pad[1]] * 2
        v = [F.pad(d["v_eps"].double(), zp), F.pad(d["v_sig"].double(), zp)]
        (_, _), (dca, dcb) = torch.func.jvp(lambda e, s: _coefs(e, s, mu, dt)[:2], (eps, sig), tuple(v))
        df = d["amp"].double().permute(2, 0, 1) * dcb.reshape(-1)[src] * (-1.0 / DX**2)

    def half_h(ey, hx, hz, mex, mez):
        dz, mez = G.step(ey, mez, 0, True)
        dx, mex = G.step(ey, mex, 1, True)
        return hx - cq * dz, hz + cq * dx, mex, mez

    def curl(hx, hz, mhx, mhz):
        dz, mhz = G.step(hz, mhz, 1, False)
        dy, mhx = G.step(hx, mhx, 0, False)
        return dz - dy, mhx, mhz

    def record(ey):
        return ey.reshape(S, -1).gather(1, rec)

    def step(t, ey, hx, hz, mex, mez, mhx, mhz, *pol):
        hx, hz, mex, mez = half_h(ey, hx, hz, mex, mez)
        c, mhx, mhz = curl(hx, hz, mhx, mhz)
        e = torch.where(dom > 0, ca * ey + cb * c, ey)
        if pol:
            e = e + dom * (dcp * pol[0])
        e = _add(e, src, f[t])
        if pol:
            pol = (torch.where(dom > 0, da * pol[0] + db * (e + ey), pol[0]),)
        return (e, hx, hz, mex, mez, mhx, mhz, *pol), record(e)

    def step_jvp(t, *s):
        (ey, hx, hz, mex, mez, mhx, mhz), (se, sx, sz, pex, pez, phx, phz) = s[:7], s[7:]
        hx, hz, mex, mez = half_h(ey, hx, hz, mex, mez)
        sx, sz, pex, pez = half_h(se, sx, sz, pex, pez)
        c, mhx, mhz = curl(hx, hz, mhx, mhz)
        sc, phx, phz = curl(sx, sz, phx, phz)
        se = torch.where(dom > 0, ca * se + cb * sc + dca * ey + dcb * c, se)
        ey = torch.where(dom > 0, ca * ey + cb * c, ey)
        ey, se = _add(ey, src, f[t]), _add(se, src, df[t])
        return ((ey, hx, hz, mex, mez, mhx, mhz, se, sx, sz, pex, pez, phx, phz),
                torch.stack([record(ey), record(se)]))

    z = [torch.zeros((S, *G.shape), device="cuda", dtype=torch.float64) for _ in range(3)]
    mem = [(1, True), (0, True), (0, False), (1, False)]  # m_Ey_x, m_Ey_z, m_Hx_z, m_Hz_x
    z += [G.zeros(S, *m) for m in mem]
    if kind == "debye":
        z.append(torch.zeros((S, *G.shape), device="cuda", dtype=torch.float64))
    if kind == "jvp":
        z = z + z
    state, r = _loop(step_jvp if kind == "jvp" else step, tuple(z), nt, grads)
    if grads:
        return [r.detach(), *torch.autograd.grad(0.5 * (r * r).sum(), leaves)]
    full = [G.crop(t) for t in state[-7:-4]] + [G.crop(G.outer(t, *m)) for t, m in zip(state[-4:], mem)]
    return [r[:, 0], r[:, 1], *full] if kind == "jvp" else [r, *full]


def _exact_3d(case, d):
    S, nt, grads = case["shots"], case["nt"], case["kind"] == "gradient3d"
    G = _Grid(case, d["dt"])
    P, dt = G.P, d["dt"]
    pad = (P + case["pml"], P - 1 + case["pml"])
    leaves = [t.double().requires_grad_(grads) for t in (d["eps"], d["sig"])]
    eps, sig, mu = (_replicate(t, pad) for t in (*leaves, d["mu"].double()))
    ca, cb, cq = _coefs(eps, sig, mu, dt)
    src, rec = _flat(d["src"], G.shape, pad[0]), _flat(d["rec"], G.shape, pad[0])
    f = d["amp"].double().permute(2, 0, 1) * cb.reshape(-1)[src] * (-1.0 / DX**3)
    dom = torch.zeros((1, *G.shape), device="cuda", dtype=torch.float64)
    dom[:, P:G.shape[0] - P + 1, P:G.shape[1] - P + 1, P:G.shape[2] - P + 1] = 1.0

    # memories in the state's order: field, axis (z, y, x = 0, 1, 2), half points
    mems = [("hz", 1), ("hy", 0), ("hx", 0), ("hz", 2), ("hy", 2), ("hx", 1),
            ("ey", 0), ("ez", 1), ("ez", 2), ("ex", 0), ("ex", 1), ("ey", 2)]
    at = {m: i for i, m in enumerate(mems)}

    def step(t, ex, ey, ez, hx, hy, hz, *m):
        m = list(m)
        F_ = {"ex": ex, "ey": ey, "ez": ez, "hx": hx, "hy": hy, "hz": hz}

        def D(name, ax):
            i = at[name, ax]
            out, m[i] = G.step(F_[name], m[i], ax, name[0] == "e")
            return out

        hx = hx - cq * (D("ey", 0) - D("ez", 1))
        hy = hy - cq * (D("ez", 2) - D("ex", 0))
        hz = hz - cq * (D("ex", 1) - D("ey", 2))
        F_.update(hx=hx, hy=hy, hz=hz)
        cx, cy, cz = D("hy", 0) - D("hz", 1), D("hz", 2) - D("hx", 0), D("hx", 1) - D("hy", 2)
        ex, ey, ez = (torch.where(dom > 0, ca * e + cb * c, e) for e, c in ((ex, cx), (ey, cy), (ez, cz)))
        ez = _add(ez, src, f[t])
        return (ex, ey, ez, hx, hy, hz, *m), ez.reshape(S, -1).gather(1, rec)

    z = [torch.zeros((S, *G.shape), device="cuda", dtype=torch.float64) for _ in range(6)]
    z += [G.zeros(S, ax, n[0] == "e") for n, ax in mems]
    state, r = _loop(step, tuple(z), nt, grads)
    if grads:
        return [r.detach(), *torch.autograd.grad(0.5 * (r * r).sum(), leaves)]
    full = [G.crop(t) for t in state[:6]]
    full += [G.crop(G.outer(t, ax, n[0] == "e")) for t, (n, ax) in zip(state[6:], mems)]
    return [r, *full]


def exact(case, seed):
    d = _inputs(case, seed)
    with torch.set_grad_enabled(case["kind"] in ("gradient", "gradient3d", "debye")):
        out = _exact_3d(case, d) if "nz" in case else _exact_tm(case, d)
    return [t.detach() for t in out]
