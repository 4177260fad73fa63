"""How the conjugate-gradient loop of the pressure solve ends when it cannot go
on, in its two forms (one kernel on small grids; separate kernels, which
profiling selects)."""
import numpy as np
import pytest

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
