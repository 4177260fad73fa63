"""Infinities and NaN go through a routine as through the reference's
expressions, where a mask is a factor 0 (0 times NaN is NaN): the same cells are
non-finite as the oracle's, and the others hold its values.  One value at a time,
in open water, at the bottom and below it, at the coast, on the shore and
inland, so that cells without outflow, local extrema and masked faces are next to it."""
import numpy as np
import pytest

import oracle as O
from orctm_b200 import configs as C
from orctm_b200 import grid
from orctm_b200.api import Instance

pytestmark = pytest.mark.gpu

ROUTINES = {"ocuad": ("uoo", "uko", "vke", "wo"), "ocvad": ("voe", "uko", "vke", "wo"),
            "ocwad": ("wno", "uko", "vke", "wo", "zo"), "ocadpo": ("tracer0", "uko", "vke", "wo", "zo"),
            "octdiff": ("tracer0", "dvo", "zo"), "ocvisc": ("uoo", "voe", "wno", "avo")}


@pytest.fixture(scope="module")
def inst():
    return C.make_instance("c4", builder=grid.build_grid, nx=50, ny=41, nz=31)


def places(inst):
    """Points (i, j, K - 1) by what surrounds them."""
    kb = (inst["weto"] > 0).sum(axis=2)
    ke = inst["ke"]
    inner = np.zeros_like(kb, bool)
    inner[2:-2, 2:-2] = True
    around = [np.roll(kb, s, a) for s in (1, -1) for a in (0, 1)]
    least, most = np.minimum.reduce(around), np.maximum.reduce(around)
    kinds = {"deep": ((kb >= 6) & (least >= 6), lambda b: 3), "surface": ((kb >= 6) & (least >= 6), lambda b: 0),
             "bottom": ((kb >= 4) & (kb < ke - 2), lambda b: b - 1), "below": ((kb >= 4) & (kb < ke - 3), lambda b: b + 1),
             "coast": ((kb >= 4) & (least == 0), lambda b: 1), "shore": ((kb == 0) & (most > 3), lambda b: 1),
             "step": ((kb >= 4) & (least < kb - 2) & (least > 0), lambda b: b - 1)}
    out = {}
    for name, (mask, level) in kinds.items():
        q = np.argwhere(mask & inner)
        i, j = q[len(q) // 2]
        out[name] = (i, j, level(kb[i, j]))
    return out


def _oracle(orc, routine, st):
    a = [st[k] for k in ("uko", "vke", "wo")]
    if routine in ("ocuad", "ocvad"):
        f = {"ocuad": "uoo", "ocvad": "voe"}[routine]
        getattr(orc, routine)(st[f], *a)
        return {f: st[f]}
    if routine == "ocwad":
        orc.ocwad(st["wno"], *a, st["zo"])
        return {"wno": st["wno"]}
    if routine == "ocadpo":
        orc.ocadpo(st["tracers"][0], *a, st["zo"])
        return {"tracer0": st["tracers"][0]}
    if routine == "octdiff":
        orc.octdiff(st["tracers"], st["dvo"], st["zo"])
        return {"tracer0": st["tracers"][0]}
    orc.ocvisc(*(st[k] for k in ("uoo", "voe", "wno", "uko", "vke", "avo")))
    return {k: st[k] for k in ("uoo", "voe", "wno")}


# (an infinity in a column solve is no case: the kernels' quotient by refinement gives
# NaN where IEEE division gives an infinity, and the two part ways from there)
@pytest.mark.parametrize("routine,value", [(r, v) for r in sorted(ROUTINES) for v in (np.nan, np.inf)
                                           if np.isnan(v) or r not in ("octdiff", "ocvisc")])
def test_nonfinite_values_spread_as_in_the_oracle(inst, routine, value):
    orc = O.Oracle(inst)
    gpu = Instance(inst)
    for place, (i, j, k) in places(inst).items():
        for field in ROUTINES[routine]:
            st = C.copy_state(inst)
            a = st["tracers"][0] if field == "tracer0" else st[field]
            a[(i, j) if a.ndim == 2 else (i, j, k)] = value
            gpu.upload_state(st)
            gpu.ocadpo(0) if routine == "ocadpo" else getattr(gpu, routine)()
            with np.errstate(all="ignore"):
                want = _oracle(orc, routine, st)
            for f, w in want.items():
                got = gpu.download(f)
                what = (place, field, f)
                fin = np.isfinite(w)
                assert np.array_equal(np.isfinite(got), fin), what
                assert np.abs(got[fin] - w[fin]).max() <= 1e-12 * np.abs(w[fin]).max(), what
    gpu.close()
