"""What users of this library have it do, as cases that can be timed and
compared: time steps of one resident regional domain through
``orctm_b200.api.Instance`` (the hot path alone, the whole step, the hot path
fed from host arrays every step), the hot path's routines called one by one as
the reference's driver calls them, and the scratch-free tracer diffusion on
caller-owned device arrays.

Sizes are those of the workloads in ``orctm_b200/configs.py``: the 512 x 1 x 60
internal-wave slice (c1), the 256 x 256 x 60 tidal box (c2), the
1024 x 1024 x 80 region (c3), and the uneven members of the ensemble and of the
served stream (c4, c5: 96-768 x 96-768 x 40-100).  Grids come from the package's own
grid builder; states are made on the GPU from the seed with the same statistics
as the package's generators (tanh thermocline, filtered-noise ridges with about
15 % land, velocities of some tenths of a metre per second, w from continuity
with a vertical Courant number of at most 0.5).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from orctm_b200 import _lib, configs, grid
from orctm_b200.api import Instance

# Residual target of the Poisson solve, as in the tests of whole steps: with the
# default 1e-10 the pressure is determined to only 7 or 8 digits after some
# steps, and a comparison of two solvers would see nothing but where each stops.
RTOL = 1e-13
MAXIT = 5000


def listed():
    """The cases.  ``kind``: "hot" = ``steps`` hot-path steps on the resident
    state and the download of what an output writer takes; "full" = the same
    with the whole model step; "host" = the drop-in use, where the host model
    hands over the fields and takes the results back every step, copies
    overlapping the kernels (with ``tides``, the step starts with the
    open-boundary forcing and sponges, as the reference's driver does); "routines" = the driver's advection and diffusion calls one by
    one; "octdiff" = orctm_octdiff_noalloc on device arrays."""
    return [
        # the vertical slice: few columns, hundreds of Krylov iterations, bound by latency
        {"name": "slice_hot", "kind": "hot", "config": "c1", "nx": 512, "ny": 1, "nz": 60, "solver": "fp64", "steps": 4},
        # the slice's production run: whole model steps, linear equation of state
        {"name": "slice_full", "kind": "full", "config": "c1", "nx": 640, "ny": 1, "nz": 50, "solver": "fp64", "steps": 4},
        # the smallest ensemble members, ragged in every direction
        {"name": "member_small", "kind": "hot", "config": "c4", "nx": 97, "ny": 131, "nz": 41, "solver": "fp64", "steps": 4},
        # the tidal box, both solver forms
        {"name": "box_hot", "kind": "hot", "config": "c2", "nx": 256, "ny": 256, "nz": 60, "solver": "fp64", "steps": 4},
        {"name": "box_refined", "kind": "hot", "config": "c2", "nx": 256, "ny": 256, "nz": 60, "solver": "fp32_refined", "steps": 4},
        # the box's whole model step (closed: open sides are unstable at this time step)
        {"name": "box_full", "kind": "full", "config": "c2", "nx": 240, "ny": 272, "nz": 60, "solver": "fp64", "steps": 3},
        # the drop-in: fields from and to page-locked host arrays every step
        {"name": "box_host", "kind": "host", "config": "c2", "nx": 256, "ny": 256, "nz": 60, "solver": "fp64", "steps": 1, "tides": True},
        # an ordinary, odd-sized ensemble member
        {"name": "member_odd", "kind": "hot", "config": "c4", "nx": 413, "ny": 311, "nz": 83, "solver": "fp64", "steps": 3},
        # a host model that calls the stencil routines itself, without the solve
        {"name": "member_routines", "kind": "routines", "config": "c4", "nx": 301, "ny": 403, "nz": 67, "solver": "fp64", "steps": 4},
        # a large served request, mixed-precision solver
        {"name": "large_refined", "kind": "hot", "config": "c5", "nx": 640, "ny": 576, "nz": 80, "solver": "fp32_refined", "steps": 3},
        # the headline region
        {"name": "region_hot", "kind": "hot", "config": "c3", "nx": 1024, "ny": 1024, "nz": 80, "solver": "fp64", "steps": 4},
        # tracer diffusion under another runtime's device memory (no allocation)
        {"name": "octdiff_device", "kind": "octdiff", "config": "c4", "nx": 150, "ny": 137, "nz": 90, "solver": "", "steps": 1},
    ]


def draw(rng):
    """One more case of the same ranges."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["hot", "hot", "hot", "full", "host", "routines", "octdiff"])
    solver = rng.choice(["fp64", "fp64", "fp32_refined"])
    slice_ = kind in ("hot", "full") and rng.random() < 0.3
    if slice_:
        return {"kind": kind, "config": "c1", "nx": spread(96, 1000), "ny": 1, "nz": rng.randint(40, 100),
                "solver": solver, "steps": rng.randint(2, 4)}
    if kind == "octdiff":
        return {"kind": kind, "config": "c4", "nx": rng.randint(48, 150), "ny": rng.randint(48, 130), "nz": rng.randint(30, 100),
                "solver": "", "steps": 1}
    hi = {"hot": 800, "full": 420, "host": 420, "routines": 520}[kind]
    config = rng.choice(["c2", "c4", "c5"] if kind != "hot" else ["c2", "c3", "c4", "c5"])
    case = {"kind": kind, "config": config, "nx": spread(96, hi), "ny": spread(96, hi), "nz": rng.randint(40, 80),
            "solver": solver, "steps": 1 if kind == "host" else rng.randint(2, 4)}
    if kind == "host":
        case["tides"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs --
def _smooth2d(shape, sigma, gen):
    """Gaussian-filtered white noise over (rows j, columns i), scaled to 1."""
    a = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(shape[0], device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.fftfreq(shape[1], device="cuda", dtype=torch.float64)[None, :]
    h = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (kx ** 2 + ky ** 2))
    a = torch.fft.ifft2(torch.fft.fft2(a) * h).real
    return a / a.abs().max().clamp_min(1e-30)


def _device(a):
    """A Fortran-ordered host array as a device tensor with reversed axes."""
    return torch.from_numpy(a.T).cuda()


def _grid(case, seed):
    """The instance's geometry (host arrays): bathymetry, metrics, BELEG + BODEN."""
    over = {"nx": case["nx"], "ny": case["ny"], "nz": case["nz"], "closed": case["kind"] == "full"}
    inst = configs.raw_instance(case["config"], seed=seed, **over)
    depto, geo = grid.build_grid(inst["ie"], inst["je"], inst["ke"], inst["dt"], inst["dzw"], inst["depto_raw"],
                                 inst["dlxp"], inst["dlyp"], inst["dlxu"], inst["dlyu"], inst["dlxv"], inst["dlyv"])
    inst["depto"] = depto
    inst.update(geo)
    return inst


def _state(inst, seed):
    """The initial state on the device, each field with its axes reversed
    (levels, j, i), the transpose of the Fortran layout."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    ie, je, ke, dt = inst["ie"], inst["je"], inst["ke"], inst["dt"]
    f64 = {"device": "cuda", "dtype": torch.float64}
    dduo, ddue, ddpo = _device(inst["dduo"]), _device(inst["ddue"]), _device(inst["ddpo"])
    dx = float(inst["dlxp"][0, 0])
    wet = (ddpo > 0).to(torch.float64)
    z = -torch.from_numpy(inst["tiestu"][:ke].copy()).cuda()

    def noise(shape, amp):
        return torch.randn(shape, generator=gen, **f64).mul_(amp)

    lev = torch.linspace(0.0, math.pi, ke, **f64)[:, None, None]
    slice_ = inst["ny"] == 1

    def currents(amp, sigma, white):
        """A barotropic and a first baroclinic pattern and some white noise."""
        u = noise((ke, je, ie + 1), white)
        v = noise((ke, je + 1, ie), white)
        for prof in (0.6 + 0.0 * lev, 0.4 * torch.cos(lev)):
            if slice_:
                line = _smooth2d((1, ie + 1), sigma, gen)
                u += amp * prof * line[None]
            else:
                u += amp * prof * _smooth2d((je, ie + 1), sigma, gen)[None]
                v += amp * prof * _smooth2d((je + 1, ie), sigma, gen)[None]
        u *= dduo > 0
        v *= ddue > 0
        if slice_:
            v.zero_()
        return u, v

    def continuity(u, v):
        fu, fv = u * dduo, v * ddue
        div = ((fu[:, :, :-1] - fu[:, :, 1:]) + (fv[:, 1:, :] - fv[:, :-1, :])) * wet / dx
        w = torch.zeros((ke + 1, je, ie), **f64)
        w[:ke] = div.flip(0).cumsum(0).flip(0)
        return w

    u, v = currents(0.25, 6.0, 0.02)
    w = continuity(u, v)
    thin = torch.where(ddpo > 0, ddpo, torch.full((), math.inf, **f64))
    lim = torch.cat([thin[:1], torch.minimum(thin[:-1], thin[1:])])
    cz = float((w[:ke].abs() * dt / lim).max())
    if cz > configs.VERTICAL_CFL:
        for a in (u, v, w):
            a *= configs.VERTICAL_CFL / cz
    # the state one step before differs by a hydrostatic increment, which
    # drives the right-hand side of the pressure solve
    du, dv = currents(1e-3, 4.0, 0.0)
    u1, v1 = u - du, v - dv
    w1 = continuity(u1, v1)

    eta = torch.zeros(ie, **f64)
    if inst["name"] == "c1":
        x = (torch.arange(ie, **f64) - 0.5) * dx
        eta = -30.0 / torch.cosh((x - 2000.0) / 500.0) ** 2
    # thermocline over a weakly stratified deep layer, so that the convective
    # switches of the whole step do not hang on the last digit
    tho = 15.0 + 5.0 * torch.tanh((z[:, None, None] + 50.0 - eta[None, None, :]) / 10.0) + 1e-3 * z[:, None, None]
    tho = tho.expand(ke, je, ie) + noise((ke, je, ie), 1e-4)
    sao = 35.0 - 1e-4 * z[:, None, None]
    tracers = [tho, sao.expand(ke, je, ie).contiguous()]
    if inst["ntracers"] >= 3:
        tracers.append(torch.rand((ke, je, ie), generator=gen, **f64))
    zo = noise((je, ie), 0.2) * wet[0]

    def mixing(deep, top):
        k = torch.arange(ke + 1, **f64)[:, None, None]
        a = (deep + top * torch.exp(-k / 5.0)) * (0.9 + 0.2 * torch.rand((ke + 1, je, ie), generator=gen, **f64))
        a[:ke] *= wet
        a[0] = 0.0
        return a

    dvo, avo = mixing(2e-5, 1e-3), mixing(2e-4, 5e-3)
    dvo[ke] = 0.0
    st = {"uoo": u, "voe": v, "wno": w, "uko": u, "vke": v, "wo": w, "uoo1": u1, "voe1": v1, "wno1": w1,
          "zo": zo, "dvo": dvo, "avo": avo}
    st.update({f"tracer{n}": t for n, t in enumerate(tracers)})
    return st


def _host(shape):
    """A page-locked host array in Fortran order."""
    return torch.empty(tuple(reversed(shape)), dtype=torch.float64, pin_memory=True).numpy().T


def _to_host(t):
    a = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    a.copy_(t)
    return a.numpy().T


def _forcing(gpu, inst, st):
    """What the whole step reads besides the state: equation of state and
    surface forcing, Coriolis inputs, barotropic constants and wind."""
    surface = [np.asfortranarray(st[f"tracer{n}"][0].cpu().numpy().T) for n in range(2)]
    top = dict(inst, tracers=[s[:, :, None] for s in surface])
    gpu.set_thermo(**configs.make_thermo(top))
    cor = configs.make_coriolis(inst)
    gpu.set_coriolis(cor["ftwou"], cor["ftwov"], cor["gila"], cor["giph"], cor["omega"])
    gpu.set_barotropic(*grid.uv_depths(inst["depto"]), configs.barotropic_minvalue(inst))
    gpu.ocwind(**configs.make_wind(inst))


def _tides(gpu, inst, st):
    """Tidal constants, sponges and T/S climatology of the open sides."""
    gpu.set_obc(configs.make_obc(inst))
    whole = dict(inst, tracers=[st[f"tracer{n}"].cpu().numpy().T for n in range(2)])
    for n in range(2):
        gpu.set_obc_ts(n, configs.make_obc_ts(whole, n))


def _prepare_octdiff(inst, st):
    dev = {k: _device(inst[k]).contiguous() for k in ("ddpo", "weto", "di", "dzw", "dlxp", "dlyp", "dlxu", "dlyu", "dlxv", "dlyv")}
    dev.update(dvo=st["dvo"].contiguous(), zo=st["zo"].contiguous(), tracer_in=st["tracer0"].contiguous(),
               tracer_out=torch.empty_like(st["tracer0"]))
    a = _lib.NoAllocArgs(ie=inst["ie"], je=inst["je"], ke=inst["ke"], dt=inst["dt"], almzer=inst["almzer"],
                     aulapts=inst["aulapts"], ah00=inst["ah00"])
    for k, t in dev.items():
        setattr(a, k, t.data_ptr())
    a.stream = torch.cuda.current_stream().cuda_stream
    return {"kind": "octdiff", "lib": _lib.load(), "args": a, "arrays": dev}


def prepare(case, seed):
    inst = _grid(case, seed)
    st = _state(inst, seed)
    if case["kind"] == "octdiff":
        return _prepare_octdiff(inst, st)
    gpu = Instance(inst)
    gpu.set_solver(case["solver"], rtol=RTOL, maxit=MAXIT)
    if case["kind"] == "full":
        _forcing(gpu, inst, st)
    if case.get("tides"):
        _tides(gpu, inst, st)
    fields = {k: _to_host(t) for k, t in st.items()}
    for k, a in fields.items():
        gpu.upload(k, a)
    outputs = ["uoo", "voe", "wno", "pnh"] + [f"tracer{n}" for n in range(gpu.ntr)]
    if case["kind"] == "full":
        outputs.append("zo")
    if case["kind"] == "routines":
        outputs.remove("pnh")
    out = {k: _host(gpu.shape(k)) for k in outputs}
    state = {"kind": case["kind"], "gpu": gpu, "steps": case["steps"], "out": out, "step": 0, "ntr": gpu.ntr, "tides": bool(case.get("tides"))}
    if case["kind"] == "host":
        # the fields the rest of the host model changes between two steps
        state["in"] = fields
        fields["pnh"] = _host(gpu.shape("pnh"))
        fields["pnh"][...] = 0.0
        gpu.set_step_outputs(out)
    return state


# -------------------------------------------------------------------- pass --
def run(state):
    kind = state["kind"]
    if kind == "octdiff":
        _lib.check(state["lib"].orctm_octdiff_noalloc(C.byref(state["args"])))
        return {"tracer0": state["arrays"]["tracer_out"]}
    gpu, out = state["gpu"], state["out"]
    for _ in range(state["steps"]):
        state["step"] += 1
        if kind == "hot":
            gpu.step_hotpath()
        elif kind == "full":
            gpu.step_full(state["step"], check_contra=False)
        elif kind == "host":
            for name, a in state["in"].items():
                gpu.upload_async(name, a)
            if state["tides"]:
                gpu.obc_ts()
                gpu.obc_eta(state["step"])
                gpu.obc_uv(state["step"])
                gpu.octimf()
            gpu.step_hotpath()
            gpu.wait_copies()
        else:
            gpu.ocuad()
            gpu.ocvad()
            gpu.ocwad()
            for n in range(state["ntr"]):
                gpu.ocadpo(n)
            gpu.octdiff()
            gpu.octimf()
            gpu.ocvisc()
    if kind != "host":
        for name, a in out.items():
            gpu.download(name, a)
    return out


def work(case):
    """Per step: every field that enters it read once and every field that
    leaves it written once (FP64; fields that are only renamed count nothing),
    and some hundred operations per cell for each advected or diffused field.
    Krylov iterations are not counted: how many there are is the solver's own."""
    n = 2 if case["config"] == "c1" else 3
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "octdiff":
        return {"bytes": 8.0 * 3 * cells, "flops": 60.0 * cells}
    reads, writes, flops = {"hot": (12 + n, 4 + n, 300.0 * (4 + n)), "host": (12 + n, 4 + n, 300.0 * (4 + n)),
                            "full": (12 + n, 8 + n, 300.0 * (8 + n)), "routines": (8 + n, 3 + n, 300.0 * (3 + n))}[case["kind"]]
    return {"bytes": 8.0 * (reads + writes) * cells * case["steps"], "flops": flops * cells * case["steps"]}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Tracer diffusion in plain 64-bit torch; whole steps have no short
    restatement."""
    if case["kind"] != "octdiff":
        return None
    inst = _grid(case, seed)
    st = _state(inst, seed)
    g = {k: _device(inst[k]) for k in ("ddpo", "weto", "di", "dzw", "dlxp", "dlyp", "dlxu", "dlyu", "dlxv", "dlyv")}
    dt, eps, aul, ke = inst["dt"], inst["almzer"], inst["aulapts"], inst["ke"]
    x, dvo = st["tracer0"].clone(), st["dvo"]
    inner = (slice(1, -1), slice(1, -1))
    thick = g["ddpo"].clone()
    thick[0] += st["zo"]
    thick = (thick + eps)[(slice(None),) + inner]
    wet = g["weto"]
    # implicit vertical diffusion: lower a, upper c, diagonal 1 - a - c
    a = -dt * dvo[:ke][(slice(None),) + inner] * wet[(slice(None),) + inner] * g["di"][:ke, None, None] / thick
    c = -dt * dvo[1:][(slice(None),) + inner] * g["di"][1:, None, None] / thick
    d = 1.0 - a - c
    r = x[(slice(None),) + inner].clone()
    for k in range(1, ke):
        m = a[k] / d[k - 1]
        d[k] -= m * c[k - 1]
        r[k] -= m * r[k - 1]
    r[ke - 1] /= d[ke - 1]
    for k in range(ke - 2, -1, -1):
        r[k] = (r[k] - c[k] * r[k + 1]) / d[k]
    x[(slice(None),) + inner] = r
    # explicit biharmonic part: fluxes of the Laplacian
    mid, we, ea = (slice(None), slice(1, -1), slice(1, -1)), (slice(None), slice(1, -1), slice(0, -2)), (slice(None), slice(1, -1), slice(2, None))
    no, so = (slice(None), slice(0, -2), slice(1, -1)), (slice(None), slice(2, None), slice(1, -1))
    xw, xe = g["dlxu"][1:-1, 1:-2], g["dlxu"][1:-1, 2:-1]
    yn, ys = g["dlyv"][1:-2, 1:-1], g["dlyv"][2:-1, 1:-1]
    dxp, dyp = g["dlxp"][inner], g["dlyp"][inner]
    lap = torch.zeros_like(x)
    lap[mid] = wet[mid] * ((wet[we] * (x[we] - x[mid]) / xw + wet[ea] * (x[ea] - x[mid]) / xe) / dxp
                           + (wet[no] * (x[no] - x[mid]) / yn + wet[so] * (x[so] - x[mid]) / ys) / dyp)
    bw, be = aul * xw ** 3 * g["dlyu"][1:-1, 1:-2], aul * xe ** 3 * g["dlyu"][1:-1, 2:-1]
    bn, bs = aul * yn ** 3 * g["dlxv"][1:-2, 1:-1], aul * ys ** 3 * g["dlxv"][2:-1, 1:-1]
    flux = (wet[we] * bw * (lap[we] - lap[mid]) + wet[ea] * be * (lap[ea] - lap[mid])
            + wet[no] * bn * (lap[no] - lap[mid]) + wet[so] * bs * (lap[so] - lap[mid]))
    x[mid] -= wet[mid] * g["dzw"][:, None, None] * flux / (thick * dxp * dyp)
    return {"tracer0": x}
