"""Sizes at which the kernels' splits change, against the oracle: the first and
last column length of every split of a column over threads, planes one row or
column around a tile's edge, grids on either side of the change to another kernel, the
shortest and longest columns a handle accepts, fields larger than the upload's
staging buffer.  Where a routine has a test of its own, that test is called with
these sizes (and its tolerance: bit for bit, or 1e-12)."""
import numpy as np
import pytest

import oracle as O
import test_gpu_baroclinic
import test_gpu_parity
import test_zz_no_alloc
from orctm_b200 import configs as C
from orctm_b200 import grid
from orctm_b200.api import Instance

pytestmark = pytest.mark.gpu


def _make(name, nx, ny, nz, **over):
    return C.make_instance(name, builder=grid.build_grid, nx=nx, ny=ny, nz=nz, **over)


# Poisson: columns of every split (8, 16, 32 threads; both tile widths); up to
# 104 levels these planes go through the one-kernel loop, 130 x 240 and longer columns
# through separate kernels with the coarse space: planes of one and two tiles of 34
# (500 m spacing) and 46 columns (1852 m), and without it (20 km)
POISSON = ([("c2", 18, 5, 40), ("c2", 20, 6, 41), ("c2", 33, 7, 48), ("c2", 34, 9, 49), ("c2", 17, 30, 64),
            ("c2", 40, 11, 65), ("c2", 31, 12, 80), ("c2", 35, 8, 81), ("c2", 36, 9, 88), ("c2", 19, 10, 89),
            ("c2", 20, 9, 104), ("c2", 9, 4, 2), ("c1", 130, 1, 60)],
           [("c2", 34, 34, 105), ("c2", 35, 33, 106), ("c2", 69, 12, 160), ("c2", 30, 35, 161),
            ("c2", 14, 8, 320), ("c1", 70, 1, 110), ("c2", 46, 47, 105, 1852.0), ("c2", 12, 9, 120, 2e4),
            ("c2", 130, 240, 41)])


@pytest.mark.parametrize("mode", ["fp64", "fp32_refined"])
@pytest.mark.parametrize("size", POISSON[0] + POISSON[1], ids=lambda s: "-".join(map(str, s)))
def test_poisson_residual_by_the_oracles_matrix(size, mode):
    """||b - A x|| with the oracle's matrix and right-hand side: the target 1e-12
    plus the rounding of this evaluation, nine operations a row."""
    name, nx, ny, nz, *dx = size
    inst = _make(name, nx, ny, nz, **({"dx": dx[0]} if dx else {}))
    orc, gpu, st = test_gpu_parity._pair(inst)
    b = orc.nh_rhs(st["uoo"], st["uoo1"], st["voe"], st["voe1"], st["wno"], st["wno1"], st["zo"])
    A = orc.matrix()
    gpu.set_solver(mode, rtol=1e-12, maxit=20000)
    stats = gpu.ocvtot_nh()
    assert stats["converged"] == 1 and stats["relres"] <= 1e-12, stats
    x = gpu.download("pnh")[1:-1, 1:-1, :].reshape(-1, order="F")
    rounding = 9 * np.finfo(np.float64).eps * np.linalg.norm(abs(A) @ abs(x) + abs(b))
    assert np.linalg.norm(b - A @ x) <= 1e-12 * np.linalg.norm(b) + rounding
    gpu.close()


@pytest.mark.parametrize("mode", ["fp64", "fp32_refined"])
def test_poisson_one_kernel_equals_separate_kernels(mode):
    """With profiling on the loop runs as separate kernels: the same values and
    the same order of sums as the one kernel of small grids."""
    inst = _make("c2", 45, 21, 50)
    got = []
    for prof in (False, True):
        _, gpu, _ = test_gpu_parity._pair(inst)
        gpu.set_solver(mode, rtol=1e-12, maxit=20000)
        gpu.set_profiling(prof)
        stats = gpu.ocvtot_nh()
        got.append((gpu.download("pnh"), stats["iterations"]))
        gpu.close()
    assert got[0][1] == got[1][1]
    assert np.array_equal(got[0][0], got[1][0])


# advection marches tiles of 28 cells and chunks of 8 levels; viscosity chunks of 8;
# column solves change their split at 48, 64, 80, 96, 112 and 160 levels
STENCIL = [("c2", 26, 27, 8), ("c2", 27, 3, 9), ("c2", 29, 30, 7), ("c2", 55, 5, 17), ("c2", 8, 4, 2), ("c2", 12, 9, 48),
           ("c2", 9, 8, 49), ("c2", 8, 9, 65), ("c2", 7, 8, 80), ("c2", 30, 4, 97), ("c2", 7, 6, 113), ("c2", 6, 7, 161),
           ("c2", 5, 4, 320), ("c1", 57, 1, 33)]


@pytest.mark.parametrize("size", STENCIL, ids=lambda s: "-".join(map(str, s)))
def test_stencils_at_tile_edges(size):
    case = ("edge", _make(*size))
    for routine in ("ocuad", "ocvad", "ocwad"):
        test_gpu_parity.test_momentum_advection(case, routine)
    test_gpu_parity.test_tracer_advection(case)
    test_gpu_parity.test_tracer_advection_all_equals_one_by_one(case)
    test_gpu_parity.test_tracer_diffusion(case)
    test_gpu_parity.test_momentum_diffusion(case)


@pytest.mark.parametrize("size", [s for s in STENCIL if s[3] >= 7], ids=lambda s: "-".join(map(str, s)))
def test_octdiff_noalloc_at_split_edges(size, monkeypatch):
    monkeypatch.setattr(test_zz_no_alloc, "instance", lambda case: _make(*size))
    test_zz_no_alloc.test_octdiff_noalloc_matches_handle_path_and_oracle("edge", False)


# OCMODMOM takes tiles of 26 points from (0, 0) and chunks of 8 levels, OCCLIT 32
# columns from i = 0, its shared memory takes the opt-in from 95 levels on
@pytest.mark.parametrize("name,over", [("c2", dict(nx=23, ny=24, nz=8)), ("c2", dict(nx=24, ny=23, nz=9)),
                                       ("c2", dict(nx=49, ny=4, nz=16)), ("c2", dict(nx=29, ny=49, nz=7)),
                                       ("c2", dict(nx=30, ny=5, nz=96)), ("c2", dict(nx=31, ny=5, nz=97)), ("c2", dict(nx=28, ny=5, nz=94)),
                                       ("c2", dict(nx=8, ny=6, nz=320)), ("c1", dict(nx=50, nz=17))])
def test_baroclinic_at_tile_edges(name, over):
    test_gpu_baroclinic.test_octher_ocmodmom_occlit_bit_identical(name, over, 0, False)


# TRONEU: one block up to 3072 points, tiles of 22 points and 8 sweeps a launch up to 148
# tiles, 38 points and 4 sweeps beyond; counts of sweeps that do not divide
@pytest.mark.parametrize("nx,ny,niter", [(46, 62, 7), (46, 63, 1), (64, 64, 8), (65, 42, 9), (20, 200, 33),
                                         (262, 262, 17), (264, 263, 5), (300, 290, 13)])
def test_troneu_bit_identical_at_tile_edges(nx, ny, niter):
    inst = _make("c2", nx, ny, 3)
    orc = O.Oracle(inst)
    bt = C.make_barotropic(inst)
    b = dict(O.BARO_DEFAULTS, sorpar=1.7, niter=niter)
    deuto, deute, _, _ = orc.deut(inst["depto"], C.barotropic_minvalue(inst))
    b1o, z1o = orc.troneu(b, *orc.itprep(b, deuto, deute), bt["u1o"], bt["v1e"], bt["uzo"], bt["vze"])
    gpu = Instance(inst)
    gpu.upload_state(C.copy_state(inst))
    gpu.set_barotropic(deuto, deute, C.barotropic_minvalue(inst), sorpar=b["sorpar"], niter=niter)
    gpu.troneu(bt["u1o"], bt["v1e"], bt["uzo"], bt["vze"])
    assert np.array_equal(gpu.download_barotropic("b1o"), b1o)
    assert np.array_equal(gpu.download_barotropic("z1o"), z1o)
    gpu.close()


def test_planes_of_more_rows_than_a_grid_has_in_y(monkeypatch):
    """66 000 rows: launches that take rows one by one count them in x."""
    tall = _make("c2", 2, 66000, 7, dx=2e4)  # within the scratch-free entry's cells
    monkeypatch.setattr(test_zz_no_alloc, "instance", lambda case: tall)
    test_zz_no_alloc.test_octdiff_noalloc_matches_handle_path_and_oracle("edge", False)
    test_gpu_parity.test_momentum_diffusion(("edge", tall))
    test_gpu_baroclinic.test_octher_ocmodmom_occlit_bit_identical("c2", dict(nx=2, ny=66000, nz=7, dx=2e4), 0, False)
    test_poisson_residual_by_the_oracles_matrix(("c2", 2, 66000, 7, 2e4), "fp64")


def test_copies_of_fields_larger_than_the_staging_buffer():
    """A field of 80 MB in several stagings, at every staggering, there and back."""
    inst = _make("c2", 401, 307, 80)
    gpu = Instance(inst)
    g = C.rng(7)
    for k in ("uoo", "voe", "wno", "pnh", "zo"):
        a = np.asfortranarray(g.standard_normal(gpu.shape(k)))
        gpu.upload(k, a)
        assert np.array_equal(gpu.download(k), a), k
    gpu.close()
