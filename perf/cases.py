"""The work that programs built on this library have it do, as timed cases.

Every case is one whole call sequence of a user's program through the public
entry points (``BGK3D``, ``run_loop``, the C-ABI with buffers of the
program's own), from inputs that the program already holds to results in its
hands:

  loop     initial condition, ``run_loop`` (the reference program's time loop:
           boundaries, col_MC, diagnostic every ``icheck`` steps), then the
           populations into the program's pinned buffer
  calls    the same sequence spelled out step by step, as a Fortran or C
           driver calls it
  steps    initial condition, ``run(n)``, one diagnostic record, populations
  fields   what is looked at while a run is under way: the diagnostic record
           with enstrophy, the energy spectrum and the velocity field
  adjoint  loss and gradients of a run with respect to its initial velocity
           and tau
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from bgk3d_hit_b200 import BGK3D, _abi, run_loop

DP = C.POINTER(C.c_double)
STORE = {"fp64": torch.float64, "fp32": torch.float32, "fp16": torch.float16}
ELEM = {"fp64": 8, "fp32": 4, "fp16": 2}


def _case(name, kind, size, precision, steps, *, scheme="two_lattice", tau=0.505, field="hit", k0=4.0, u=0.03,
          icheck=10, les=0.0, ckpt=0, rebuild=False):
    nx, ny, nz = (size,) * 3 if isinstance(size, int) else size
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, scheme=scheme, steps=steps, tau=tau, field=field,
             k0=k0, u=u, icheck=icheck, les=les, ckpt=ckpt, rebuild=rebuild)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small Taylor-Green box on the default diagnostic interval: a
        # program's test run, where launches and read-backs are the cost
        _case("tgv_32_fp64", "loop", 32, "fp64", 100, field="tgv", tau=0.53, u=0.05),
        # a Taylor-Green validation run (64^3, tau = 0.53, 500 steps)
        _case("tgv_64_fp64", "loop", 64, "fp64", 500, field="tgv", tau=0.53, u=0.05),
        # the reference's shipped run (180^3, svisc = 0.0014317, icheck = 85)
        # in its default single-precision build: rows that are no power of two
        _case("tgv_180_fp32", "loop", 180, "fp32", 170, field="tgv", tau=0.5042951, u=0.1, icheck=85),
        # a Fortran driver that calls boundaries, col_MC and diagnostic itself
        _case("calls_128_fp64", "calls", 128, "fp64", 200, icheck=100),
        # decaying turbulence at 256^3 in the three storage forms, the box
        # that the throughput figures are quoted on
        _case("hit_256_fp64", "steps", 256, "fp64", 200),
        _case("hit_256_fp32", "steps", 256, "fp32", 300),
        _case("hit_256_fp16", "steps", 256, "fp16", 300),
        # the in-place scheme, used where memory is short: the largest box
        _case("hit_384_aa_fp16", "steps", 384, "fp16", 200, scheme="aa", k0=8.0, tau=0.503),
        # under-resolved turbulence with the Smagorinsky collision, in place
        _case("les_256_aa_fp32", "steps", 256, "fp32", 200, scheme="aa", les=0.17, tau=0.503),
        # a box of odd sides in the smallest storage form
        _case("hit_odd_fp16", "steps", (201, 163, 117), "fp16", 300, tau=0.51),
        # one look at a running simulation: record, spectrum, velocity field
        _case("fields_256_fp64", "fields", 256, "fp64", 4),
        # gradients of a turbulent run, a checkpoint every 32 steps
        _case("adjoint_128_fp64", "adjoint", 128, "fp64", 128, tau=0.51, ckpt=32),
    ]


# A drawn pass moves at most this many bytes of populations when every step
# reads and writes each of them once (the listed 256^3 FP64 run: 1.02e12).
DRAW_TRAFFIC = 7e11
DRAW_STATE = 3e9


def draw(rng):
    kind = rng.choice(["loop", "loop", "calls", "steps", "steps", "steps", "steps", "fields", "adjoint"])
    precision = rng.choice(["fp64", "fp32", "fp16"] if kind != "adjoint" else ["fp64", "fp32"])
    scheme = rng.choice(["two_lattice", "two_lattice", "aa"]) if kind != "adjoint" else "two_lattice"
    top = 128 if kind == "adjoint" else 320
    while True:
        base = math.exp(rng.uniform(math.log(16), math.log(top)))
        dims = []
        for _ in range(3):
            n = max(12, min(top, round(base * math.exp(rng.uniform(-0.35, 0.35)))))
            form = rng.randrange(3)  # any side, a multiple of 4, a multiple of 32
            dims.append(n if form == 0 else max(12, n // 4 * 4) if form == 1 else max(32, n // 32 * 32))
        if rng.randrange(3) == 0:
            dims = [dims[0]] * 3
        cells = dims[0] * dims[1] * dims[2]
        per = 38 * ELEM[precision] * cells
        if per <= DRAW_STATE:
            break
    most = max(4, min(500, int(DRAW_TRAFFIC / per)))
    steps = round(math.exp(rng.uniform(math.log(max(4, most // 8)), math.log(most))))
    les = rng.choice([0.0, 0.0, 0.17]) if kind != "adjoint" else 0.0
    icheck = min(steps, rng.choice([10, 50, 100]))
    if kind == "fields":
        steps = rng.randint(2, 6)
    if kind == "adjoint":
        steps = min(steps, 128)
    # a coarse box needs the larger viscosity to stay resolved
    side = min(dims)
    taus = [0.56, 0.6] if side < 32 else [0.53, 0.56] if side < 64 else [0.51, 0.53] if side < 128 else [0.505, 0.51]
    return _case(None, kind, tuple(dims), precision, steps, scheme=scheme, tau=rng.choice(taus),
                 field=rng.choice(["hit", "hit", "tgv"]), k0=rng.choice([3.0, 4.0]) if side >= 64 else 2.0,
                 u=rng.choice([0.02, 0.03]),
                 icheck=icheck, les=les, ckpt=rng.choice([4, 11, 16, 32]) if kind == "adjoint" else 0,
                 rebuild=kind == "adjoint" and rng.randrange(2) == 0)


# ------------------------------------------------------------------- inputs
def _wavenumbers(nx, ny, nz, dev):
    f = dict(dtype=torch.float64, device=dev)
    return (torch.fft.rfftfreq(nx, 1.0 / nx, **f).reshape(1, 1, -1),
            torch.fft.fftfreq(ny, 1.0 / ny, **f).reshape(1, -1, 1),
            torch.fft.fftfreq(nz, 1.0 / nz, **f).reshape(-1, 1, 1))


def _velocity(case, seed):
    """(u, v, w) of the case on the GPU: random-phase solenoidal turbulence
    with E(k) ~ k^4 exp(-2 (k/k0)^2), or a Taylor-Green vortex of random phase."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    if case["field"] == "tgv":
        ph = torch.rand(3, generator=gen, dtype=torch.float64, device=dev) * (2 * math.pi)
        ax = [torch.arange(n, dtype=torch.float64, device=dev).add_(0.5).mul_(2 * math.pi / n) for n in (nx, ny, nz)]
        x, y, z = ((a + p).reshape(s) for a, p, s in zip(ax, ph, ((1, 1, -1), (1, -1, 1), (-1, 1, 1))))
        u = case["u"] * torch.sin(x) * torch.cos(y) * torch.cos(z)
        v = -case["u"] * torch.cos(x) * torch.sin(y) * torch.cos(z)
        return u.contiguous(), v.contiguous(), torch.zeros_like(u)
    kx, ky, kz = _wavenumbers(nx, ny, nz, dev)
    k2 = kx * kx + ky * ky + kz * kz
    amp = k2.sqrt()
    amp = amp * torch.exp(-((amp / case["k0"]) ** 2))
    for k, n in ((kx, nx), (ky, ny), (kz, nz)):
        if n % 2 == 0:
            amp = torch.where(k.abs() == n // 2, torch.zeros_like(amp), amp)
    hat = []
    for _ in range(3):
        f = torch.fft.rfftn(torch.randn((nz, ny, nx), generator=gen, dtype=torch.float64, device=dev))
        hat.append(f / f.abs().clamp_min(1e-300) * amp)
    div = (kx * hat[0] + ky * hat[1] + kz * hat[2]) / torch.where(k2 == 0, torch.ones_like(k2), k2)
    out = [torch.fft.irfftn(h - k * div, s=(nz, ny, nx)) for h, k in zip(hat, (kx, ky, kz))]
    rms = math.sqrt(sum(float((x * x).mean()) for x in out) / 3.0)
    return tuple((x * (case["u"] / rms)).contiguous() for x in out)


def _svisc(case):
    return (case["tau"] - 0.5) / 3.0


def prepare(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    vel = _velocity(case, seed)
    box = BGK3D(nx, ny, nz, svisc=_svisc(case), u0=case["u"], precision=case["precision"], scheme=case["scheme"],
                icheck=case["icheck"], les_cs=case["les"])
    s = dict(case=case, box=box)
    pinned = dict(pin_memory=True)
    if case["kind"] == "adjoint":
        target = _velocity(case, seed + 100_003)
        s["host"] = [torch.empty(nz, ny, nx, dtype=torch.float64, **pinned).copy_(a) for a in vel + target]
        s["grad"] = torch.empty(3, nz, ny, nx, dtype=torch.float64, **pinned)
        if case["rebuild"]:
            _abi.check(box._lib.bgk_adjoint_mode(box._h, _abi.BGK_ADJ_REBUILD), "bgk_adjoint_mode")
        return s
    torch.cuda.synchronize()  # the context has a stream of its own
    if case["kind"] == "fields":
        s["velocity"] = torch.empty(3, nz, ny, nx, dtype=torch.float64, **pinned)
        box.init_velocity_device(*vel)
        box.run(case["steps"])
        box.synchronize()
    else:
        s["vel"] = vel
        s["pops"] = torch.empty(19, nz, ny, nx, dtype=STORE[case["precision"]], **pinned)
    return s


def _record(d):
    """A diagnostic record: the mean state, and each of the energies and rates."""
    return {"means": torch.tensor([d["rho_mean"], d["ux_mean"], d["uy_mean"], d["uz_mean"]], dtype=torch.float64),
            "ke_mean": d["ke_mean"], "tke_norm": d["tke_norm"], "diss": d["diss"], "eps_strain": d["eps_strain"],
            "enstrophy": d["enstrophy"], "itime": d["itime"], "nonfinite": d["nonfinite"]}


def _records(recs):
    rs = [_record(d) for d in recs]
    out = {k: torch.tensor([r[k] for r in rs]) for k in ("itime", "nonfinite")}
    out.update({k: torch.tensor([r[k] for r in rs], dtype=torch.float64)
                for k in ("ke_mean", "tke_norm", "diss", "eps_strain", "enstrophy")})
    out["means"] = torch.stack([r["means"] for r in rs]) if rs else torch.zeros(0, 4, dtype=torch.float64)
    return out


def run(state):
    case, box = state["case"], state["box"]
    lib, kind, steps = box._lib, case["kind"], case["steps"]
    if kind == "adjoint":
        loss, gtau = C.c_double(), C.c_double()
        ptr = [C.cast(a.data_ptr(), DP) for a in state["host"]]
        _abi.check(lib.bgk_adjoint(box._h, *ptr, steps, case["ckpt"], C.byref(loss),
                                   C.cast(state["grad"].data_ptr(), DP), C.byref(gtau)), "bgk_adjoint")
        return {"loss": loss.value, "grad_u0": state["grad"], "grad_tau": gtau.value}
    if kind == "fields":
        rec = box.diagnostic(0)
        ek = box.spectrum()
        ptr = [C.cast(a.data_ptr(), DP) for a in state["velocity"]]
        _abi.check(lib.bgk_get_velocity(box._h, *ptr), "bgk_get_velocity")
        return {"record": _records([rec]), "spectrum": ek, "velocity": state["velocity"]}
    box.init_velocity_device(*state["vel"])
    if kind == "loop":
        recs = run_loop(box, steps)
    elif kind == "calls":
        recs = []
        for it in range(1, steps + 1):
            box.boundaries(it)
            box.col_MC(it)
            d = box.diagnostic(it)
            if d is not None:
                recs.append(d)
    else:
        box.run(steps)
        recs = [box.diagnostic(0)]
    _abi.check(lib.bgk_get_populations(box._h, state["pops"].data_ptr()), "bgk_get_populations")
    return {"records": _records(recs), "populations": state["pops"]}


def work(case):
    """Inputs read once, results written once; a collision is about 230
    operations (300 with the Smagorinsky closure), a record about 400 a cell,
    an adjoint step about twice a collision."""
    cells = case["nx"] * case["ny"] * case["nz"]
    es, steps = ELEM[case["precision"]], case["steps"]
    pops = 19 * cells * es
    if case["kind"] == "adjoint":
        return {"bytes": 9 * 8 * cells, "flops": cells * steps * (230 + 460)}
    if case["kind"] == "fields":
        n = cells
        return {"bytes": pops + 24 * cells, "flops": cells * 400 + 3 * 2.5 * n * math.log2(n)}
    nrec = 1 if case["kind"] == "steps" else steps // case["icheck"]
    return {"bytes": 24 * cells + pops, "flops": cells * (steps * (300 if case["les"] else 230) + nrec * 400)}


# ------------------------------------- the same in plain torch, in 64 bits
CX = (1, 1, 1, 1, 1, 0, 0, 0, 0, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0)
CY = (-1, 0, 1, 0, 0, 0, 1, 1, 1, -1, 0, 1, 0, 0, 0, -1, -1, -1, 0)
CZ = (0, -1, 0, 1, 0, 1, 1, 0, -1, 0, -1, 0, 1, 0, -1, -1, 0, 1, 0)
W = tuple(1 / 3 if n == 0 else 1 / 18 if n == 1 else 1 / 36
          for n in (abs(a) + abs(b) + abs(c) for a, b, c in zip(CX, CY, CZ)))


def _dot(c, v):
    out = None
    for s, x in zip(c, v):
        if s:
            out = (x if s > 0 else -x) if out is None else (out + x if s > 0 else out - x)
    return out


def _moments(f):
    rho = 1.0 + f.sum(0)
    js = [_dot([c[q] for q in range(19)], f) for c in (CX, CY, CZ)]
    return rho, [j / rho for j in js]


def _eq(q, rho, u, usq):
    """Equilibrium deviation f_eq - w of population q."""
    cu = _dot((CX[q], CY[q], CZ[q]), u)
    p = -usq if cu is None else 3.0 * cu + 4.5 * cu * cu - usq
    return W[q] * ((rho - 1.0) + rho * p)


def _pull(f):
    return torch.stack([torch.roll(f[q], (CZ[q], CY[q], CX[q]), (0, 1, 2)) for q in range(19)])


def _stress(g, rho, u, usq):
    """Non-equilibrium second moments (xx, yy, zz, xy, xz, yz)."""
    P = [torch.zeros_like(rho) for _ in range(6)]
    for q in range(18):
        n = g[q] - _eq(q, rho, u, usq)
        for i, s in enumerate((CX[q] * CX[q], CY[q] * CY[q], CZ[q] * CZ[q], CX[q] * CY[q], CX[q] * CZ[q],
                               CY[q] * CZ[q])):
            if s:
                P[i] += s * n
    return P[0] ** 2 + P[1] ** 2 + P[2] ** 2 + 2.0 * (P[3] ** 2 + P[4] ** 2 + P[5] ** 2)


def _usq(u):
    return 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])


def _step(f, omega, les):
    g = _pull(f)
    rho, u = _moments(g)
    usq = _usq(u)
    if les:
        ts = 0.5 / omega + torch.sqrt(18.0 * les * les * _stress(g, rho, u, usq).sqrt() + (1.0 / omega) ** 2) / 2.0
        omega = 1.0 / ts
    for q in range(19):
        g[q] += omega * (_eq(q, rho, u, usq) - g[q])
    return g


def _initial(vel):
    one = torch.ones_like(vel[0])
    usq = _usq(vel)
    return torch.stack([_eq(q, one, vel, usq) for q in range(19)])


def _exact_record(f, case, itime, omega):
    n = f[0].numel()
    rho, u = _moments(f)
    g = _pull(f)
    rp, up = _moments(g)
    P = _stress(g, rp, up, _usq(up))
    nu = _svisc(case)
    d = [[0.5 * (torch.roll(u[a], -1, ax) - torch.roll(u[a], 1, ax)) for ax in (2, 1, 0)] for a in range(3)]
    w = (d[2][1] - d[1][2], d[0][2] - d[2][0], d[1][0] - d[0][1])
    return {"rho_mean": float(rho.mean()), "ux_mean": float(u[0].mean()), "uy_mean": float(u[1].mean()),
            "uz_mean": float(u[2].mean()), "ke_mean": float(_usq(u).mean()) / 3.0,
            "tke_norm": float(_usq(up).sum()) / 3.0 / n / case["u"] ** 2, "diss": float((2.0 * nu * P).sum()),
            "eps_strain": float((2.0 * nu * 9.0 * omega * omega / (4.0 * rp * rp) * P).mean()),
            "enstrophy": 0.5 * float((w[0] ** 2 + w[1] ** 2 + w[2] ** 2).mean()), "itime": itime, "nonfinite": 0}


def _exact_spectrum(f, case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nb = max(nx, ny, nz) // 2 + 1
    kx, ky, kz = _wavenumbers(nx, ny, nz, f.device)
    shell = torch.floor(torch.sqrt(kx.abs() ** 2 + ky ** 2 + kz ** 2) + 0.5).long().reshape(-1)
    weight = torch.full_like(kx, 2.0)
    weight[..., 0] = 1.0
    if nx % 2 == 0:
        weight[..., -1] = 1.0
    out = torch.zeros(int(shell.max()) + 1, dtype=torch.float64, device=f.device)
    for c in _moments(f)[1]:
        e = torch.fft.rfftn(c).abs() ** 2 * weight * (0.5 / float(nx * ny * nz) ** 2)
        out += torch.bincount(shell, e.reshape(-1), minlength=out.numel())
    return out[:nb].cpu().numpy()


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    vel = torch.stack(_velocity(case, seed)).requires_grad_(True)
    target = _velocity(case, seed + 100_003)
    tau = torch.tensor(case["tau"], dtype=torch.float64, device=vel.device, requires_grad=True)

    def step(f, t):
        g = _pull(f)
        rho, u = _moments(g)
        usq = _usq(u)
        return torch.stack([g[q] + (_eq(q, rho, u, usq) - g[q]) / t for q in range(19)])

    f = _initial(list(vel))
    for _ in range(case["steps"]):
        f = checkpoint(step, f, tau, use_reentrant=False)
    u = _moments(f)[1]
    loss = sum(((a - b) ** 2).sum() for a, b in zip(u, target)) * 0.5 / f[0].numel()
    loss.backward()
    return {"loss": float(loss), "grad_u0": vel.grad.detach(), "grad_tau": float(tau.grad)}


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        f = _initial(_velocity(case, seed))
        scale = 1.0
        if case["precision"] == "fp16":  # the power of two that the context picks for the initial condition
            scale = 2.0 ** math.floor(math.log2(65504.0 / (4.0 * float(f.abs().max()))))
        omega, kind = 1.0 / case["tau"], case["kind"]
        recs = []
        for it in range(1, case["steps"] + 1):
            f = _step(f, omega, case["les"])
            if kind in ("loop", "calls") and it % case["icheck"] == 0:
                recs.append(_exact_record(f, case, it, omega))
        if kind in ("steps", "fields"):
            recs.append(_exact_record(f, case, 0, omega))
        if kind == "fields":
            return {"record": _records(recs), "spectrum": _exact_spectrum(f, case),
                    "velocity": torch.stack(_moments(f)[1])}
        f *= scale
        return {"records": _records(recs), "populations": f}
