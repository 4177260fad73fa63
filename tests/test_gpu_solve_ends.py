"""The conjugate-gradient loop of the pressure solve: its two forms (one kernel on
small grids; separate kernels, which profiling selects) give the same values, and how
it ends when it cannot go on."""
import numpy as np
import pytest

from orctm_b200 import _lib
from orctm_b200 import configs as C
from orctm_b200 import grid
from orctm_b200.api import Instance

pytestmark = pytest.mark.gpu


def test_breakdown_keeps_the_last_full_step():
    """Right-hand side so small that p.q underflows while r.r does not (a
    millimetre of spacing makes the diagonal some 1e7): the loop breaks down after
    hundreds of iterations.  The pressure is then the last full step's: finite, and
    the same bits from both forms of the loop."""
    inst = C.make_instance("c2", builder=grid.build_grid, nx=40, ny=20, nz=24, dx=1e-3)
    got = []
    for prof in (False, True):
        gpu = Instance(inst)
        st = C.copy_state(inst)
        for k in ("uoo", "voe", "wno", "uoo1", "voe1", "wno1", "pnh", "zo"):
            st[k] = np.zeros_like(st[k])
        st["uoo"] = np.asfortranarray(1e-159 * C.rng(3).standard_normal(st["uoo"].shape) * (inst["dduo"] > 0))
        gpu.upload_state(st)
        gpu.set_solver("fp64", rtol=1e-12, maxit=3000)
        gpu.set_profiling(prof)
        stats = gpu.ocvtot_nh()
        assert stats["converged"] == 0 and 0 < stats["iterations"] < 3000, stats
        got.append(gpu.download("pnh"))
        gpu.close()
    assert np.isfinite(got[0]).all() and np.abs(got[0]).max() > 0
    assert np.array_equal(got[0], got[1])


# (cycles, profiling): at once at the first staged copy, with a form's own
# kernels after it; and one cycle, which a barrier of the one-kernel loop cannot keep
@pytest.mark.parametrize("mode", ["fp64", "fp32_refined"])
@pytest.mark.parametrize("nx,ny,nz", [(45, 21, 50), (34, 34, 105)])
@pytest.mark.parametrize("cycles,prof", [(0, False), (0, True), (1, False)])
def test_a_wait_that_gives_up_is_an_error_and_no_more(nx, ny, nz, cycles, prof, mode):
    """A limit that waits cannot keep: the solve returns ORCTM_E_CUDA and leaves
    the fields alone; with the usual limit the same handle then solves as another
    does."""
    if cycles and nz > 104:
        pytest.skip("columns too long for the one-kernel loop")
    inst = C.make_instance("c2", builder=grid.build_grid, nx=nx, ny=ny, nz=nz)
    want, gpu = Instance(inst), Instance(inst)
    for g in (want, gpu):
        g.upload_state(C.copy_state(inst))
        g.set_solver(mode, rtol=1e-12, maxit=20000)
    gpu.set_profiling(prof)
    before = {k: gpu.download(k) for k in ("uoo", "voe", "wno", "pnh")}
    _lib.check(gpu.lib.orctm_set_wait_cycles(gpu.h, cycles), gpu.h)
    with pytest.raises(_lib.OrctmError) as e:
        gpu.ocvtot_nh()
    assert e.value.status == _lib.ORCTM_E_CUDA and "timed out" in str(e.value)
    for k, a in before.items():
        assert np.array_equal(gpu.download(k), a), k
    _lib.check(gpu.lib.orctm_set_wait_cycles(gpu.h, 2000000000), gpu.h)
    assert gpu.ocvtot_nh()["converged"] == 1 and want.ocvtot_nh()["converged"] == 1
    for k in before:
        assert np.array_equal(gpu.download(k), want.download(k)), k
    assert gpu.lib.orctm_set_wait_cycles(gpu.h, -1) == gpu.lib.orctm_set_wait_cycles(gpu.h, 1 << 40) == _lib.ORCTM_E_ARG
    want.close()
    gpu.close()


@pytest.mark.parametrize("mode", ["fp64", "fp32_refined"])
@pytest.mark.parametrize("nz", [40, 41, 64, 80, 81, 89, 104])
def test_both_forms_of_the_loop_agree_for_every_split_of_a_column(nz, mode):
    """5, 6, 8, 10, 11 and 13 levels a thread (and the most of each): the same
    pressure bits and iterations from one kernel and from separate ones."""
    inst = C.make_instance("c2", builder=grid.build_grid, nx=45, ny=21, nz=nz)
    got = []
    for prof in (False, True):
        gpu = Instance(inst)
        gpu.upload_state(C.copy_state(inst))
        gpu.set_solver(mode, rtol=1e-12, maxit=20000)
        gpu.set_profiling(prof)
        stats = gpu.ocvtot_nh()
        assert stats["converged"] == 1
        got.append((stats["iterations"], stats["outer_iterations"], gpu.download("pnh")))
        gpu.close()
    assert got[0][:2] == got[1][:2]
    assert np.array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("nx,ny,nz,coarse", [(45, 21, 50, False), (34, 34, 105, True)])
def test_profile_tells_the_kernels_of_an_iteration_apart(nx, ny, nz, coarse):
    """Red, black and column kernel as often as each other, the coarse correction once
    more where there is one, and one record before and one after each correction."""
    inst = C.make_instance("c2", builder=grid.build_grid, nx=nx, ny=ny, nz=nz)
    gpu = Instance(inst)
    gpu.upload_state(C.copy_state(inst))
    gpu.set_solver("fp64", rtol=1e-12, maxit=20000)
    gpu.set_profiling(True)
    stats = gpu.ocvtot_nh()
    n = {k: v["launches"] for k, v in gpu.profile().items()}
    gpu.close()
    assert n["pcg_red"] == n["pcg_spmv"] == n["pcg_col"] >= stats["iterations"] > 0
    assert n["pcg_coarse"] == (n["pcg_red"] + stats["outer_iterations"] if coarse else 0)
    assert n["pcg_ends"] == 2 * stats["outer_iterations"]
    assert n["resid"] == stats["outer_iterations"] + 1
