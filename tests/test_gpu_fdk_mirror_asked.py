"""The mirrored FDK back-projector asked for (sgb_plan_set_mirror), against the FP64 oracle and the unmirrored one.

A plan takes it where it is predicted to be faster, which volumes as small as an oracle allows often are not;
these are the cases of the tests of the plan's own choice, and volumes thinner than a run of voxels.  Bars: those
of every FDK parity test (form_bars); the two kernels take the same taps and agree to FP32 rounding of the
weights, or to the quads' own bar."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S
from test_gpu_fdk_mirror import CASES, G

pytestmark = pytest.mark.gpu

THIN = {
    "thin": (dict(na=24), (40, 36, 3), (0.5, 0.5, 0.5), (0, 0, 0)),
    "thin odd": (dict(na=25), (40, 36, 5), (0.5, 0.5, 1.0), (0, 0, 0)),
    "thin short": (dict(na=21, orbit=200.0), (36, 36, 9), (0.5, 0.5, 1.0), (0, 0, 0)),
    "thin past the detector": (dict(na=24), (36, 36, 9), (0.5, 0.5, 4.0), (0, 0, 0)),
}
# voxels that share their geometry in FP32: view slots (four with X, Y and XY, two) times z and -z where they pair
IMAGES = {"even": 4, "odd": 4, "short": 2, "start off axis": 4, "offset z": 2, "quarter row and bin": 2, "thin": 4,
          "thin odd": 4, "thin short": 2}


def _plan(kind, name, storage):
    change, dims, deltas, offsets = (CASES | THIN)[name]
    g = dict(dict(kind=kind, offset_s=0.0, offset_t=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, **G), **change)
    ig = dict(dims=dims, deltas=deltas, offsets=tuple(float(o) for o in offsets))
    return g, ig, S.plan_fbp(C.to_geom(g), C.to_image(ig), storage=storage)


def _check(kind, name, storage):
    g, ig, plan = _plan(kind, name, storage)
    proj = O.ellipsoid_proj(g, C.ELL3).astype(np.float32)
    ref = O.fdk(g, ig, proj)
    rmse, maxrel = C.form_bars(storage, g["na"])
    recs = []
    for mirror in (False, True):
        plan.set_mirror(mirror)
        images = plan.info()["images"]
        assert images > 1 if mirror else images == 1
        rec = S.fdk(plan, proj)
        assert O.rel_rmse(rec, ref) < rmse
        assert np.abs(rec - ref).max() <= maxrel * np.abs(ref).max()
        recs.append(rec)
    assert O.rel_rmse(recs[1], recs[0]) < rmse
    if storage == "f32" and name in IMAGES:
        assert images == IMAGES[name]


@pytest.mark.parametrize("kind", ["flat", "arc"])
@pytest.mark.parametrize("name", list(CASES) + list(THIN))
def test_f32(cuda, kind, name):
    _check(kind, name, "f32")


@pytest.mark.parametrize("kind", ["flat", "arc"])
@pytest.mark.parametrize("name", ["even", "even odd sides", "odd", "odd long z", "long z", "edges inside", "reversed", "thin",
                                  "thin odd", "thin past the detector"])
def test_f16(cuda, kind, name):
    _check(kind, name, "f16")


def test_scans_without_symmetry_refuse(cuda):
    g, ig, plan = _plan("flat", "offset z", "f32")
    rg = C.to_geom(dict(g, na=25, orbit=333.0))  # no whole turn, and no plane of symmetry in z
    plan = S.plan_fbp(rg, C.to_image(ig))
    with pytest.raises(Exception, match="symmetry"):
        plan.set_mirror(True)


def test_choice(cuda):
    """A thin volume from a short scan, whose runs would be mostly padding, stays with the other kernel; the same
    scan's thicker volume does not."""
    rg = S.CtFanFlat(ns=333, nt=48, ds=1.0, dt=1.0, na=181, orbit=215.0, dsd=528.0, dod=200.0)
    d = 0.45
    assert S.plan_fbp(rg, S.ImageGeom((256, 256, 8), (d, d, 2 * d))).info()["images"] == 1
    assert S.plan_fbp(rg, S.ImageGeom((256, 256, 64), (d, d, d / 2))).info()["images"] == 2
