"""Column solves shared by the threads of a block against 80-bit arithmetic: their
rounding errors are those of the plain elimination in FP64.  The rms over some
1e5 cells is good to a few per mille, so 1.005 times the plain elimination's is
the limit (a solve that multiplies by reciprocals of the pivots has 1.02)."""
import ctypes as C

import numpy as np
import pytest

from orctm_b200 import _lib, configs, grid
from orctm_b200.api import Instance

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _thomas(a, b, c, x):
    """x(K) of a(K) x(K-1) + b(K) x(K) + c(K) x(K+1) = x(K) along the last axis."""
    n = x.shape[2]
    b, x = b.copy(), x.copy()
    for k in range(1, n):
        m = a[..., k] / b[..., k - 1]
        b[..., k] = b[..., k] - c[..., k - 1] * a[..., k] / b[..., k - 1]
        x[..., k] = x[..., k] - m * x[..., k - 1]
    x[..., n - 1] = x[..., n - 1] / b[..., n - 1]
    for k in range(n - 2, -1, -1):
        x[..., k] = (x[..., k] - c[..., k] * x[..., k + 1]) / b[..., k]
    return x


def _rms(got, exact, wet):
    e = (got.astype(LD) - exact)[wet]
    return float(np.sqrt((e * e).mean()))


def _tracer(inst, st, t):
    """OCTDIFF's vertical part in type t, interior columns."""
    f = lambda v: np.asarray(v).astype(t)
    ke, dt = inst["ke"], t(inst["dt"])
    th = f(inst["ddpo"]).copy()
    th[:, :, 0] = th[:, :, 0] + f(st["zo"])
    th = th + t(inst["almzer"])
    dvo, di = f(st["dvo"]), f(inst["di"])
    a = -dt * dvo[:, :, :ke] * f(inst["weto"]) * di[:ke] / th
    c = -dt * dvo[:, :, 1:] * di[1:] / th
    return _thomas(a, 1 - a - c, c, f(st["tracers"][0]))[1:-1, 1:-1]


def _w(inst, st, t):
    """OCVISC for w without its biharmonic part in type t, levels 2..KE of interior
    columns: the solve, and the cell volume and its reciprocal of ocvisc.f90:673-688."""
    f = lambda v: np.asarray(v).astype(t)
    ke, dt = inst["ke"], t(inst["dt"])
    wet, th, avo, di = f(inst["weto"]), f(inst["ddpo"]), f(st["avo"]), f(inst["di"])
    dn = 2 * t(inst["almzer"]) + th[:, :, :-1] + th[:, :, 1:]
    up = t(.5) * (avo[:, :, :ke - 1] + avo[:, :, 1:ke]) * wet[:, :, :-1]
    lo = t(.5) * (avo[:, :, 2:ke + 1] + avo[:, :, 1:ke]) * wet[:, :, 1:]
    lo[:, :, -1] = 0
    a = -2 * dt * up * wet[:, :, 1:] * di[:ke - 1] / dn
    c = -2 * dt * lo * wet[:, :, 1:] * di[1:ke] / dn
    x = _thomas(a, 1 - a - c, c, f(st["wno"])[:, :, 1:ke] * wet[:, :, 1:])
    area = (f(inst["dlxp"]) * f(inst["dlyp"]))[:, :, None]
    dz = np.where(th > 0, th, t(1))[:, :, 1:]
    return ((1 / area) / dz * (area * dz * x))[1:-1, 1:-1]


SIZES = [(60, 50, 40), (60, 50, 60), (50, 50, 80), (50, 41, 100), (40, 40, 150), (30, 30, 300)]


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_w_solve_rounds_as_the_plain_elimination(nx, ny, nz):
    inst = configs.make_instance("c2", builder=grid.build_grid, nx=nx, ny=ny, nz=nz)
    inst["aulapuv"] = 0.0
    st = configs.copy_state(inst)
    with Instance(inst) as gpu:
        gpu.upload_state(st)
        gpu.ocvisc()
        got = gpu.download("wno")[1:-1, 1:-1, 1:nz]
    wet = inst["weto"][1:-1, 1:-1, 1:] > 0
    exact = _w(inst, st, LD)
    assert _rms(got, exact, wet) <= 1.005 * _rms(_w(inst, st, np.float64), exact, wet)


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_scratch_free_solve_rounds_as_the_plain_elimination(nx, ny, nz):
    import torch

    inst = configs.make_instance("c2", builder=grid.build_grid, nx=nx, ny=ny, nz=nz)
    st = configs.copy_state(inst)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(np.ravel(a, order="F"))).cuda()

    keep = {k: dev(inst[k]) for k in ("ddpo", "weto", "di", "dzw", "dlxp", "dlyp", "dlxu", "dlyu", "dlxv", "dlyv")}
    keep.update(dvo=dev(st["dvo"]), zo=dev(st["zo"]), tracer_in=dev(st["tracers"][0]))
    keep["tracer_out"] = torch.empty_like(keep["tracer_in"])
    a = _lib.NoAllocArgs(ie=inst["ie"], je=inst["je"], ke=inst["ke"], dt=inst["dt"], almzer=inst["almzer"],
                         aulapts=0.0, ah00=inst["ah00"])
    for k, t in keep.items():
        setattr(a, k, t.data_ptr())
    a.stream = torch.cuda.current_stream().cuda_stream
    lib = _lib.load()
    lib.orctm_octdiff_noalloc.argtypes = [C.POINTER(_lib.NoAllocArgs)]
    assert lib.orctm_octdiff_noalloc(C.byref(a)) == 0
    got = keep["tracer_out"].cpu().numpy().reshape(inst["weto"].shape, order="F")[1:-1, 1:-1]
    wet = inst["weto"][1:-1, 1:-1] > 0
    exact = _tracer(inst, st, LD)
    assert _rms(got, exact, wet) <= 1.005 * _rms(_tracer(inst, st, np.float64), exact, wet)
