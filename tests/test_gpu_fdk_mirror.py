"""FDK of scans with mirror symmetry (csrc/sgb_fdk_mirror_kernel.cuh) against the FP64 oracle.

Each case is a combination of what decides the kernel's slots, run length and row forms: which
reflections the orbit has (even, odd and short view counts, starts on and off the axes, reversed and
repeated turns), odd and even axes, unequal sides, spacings of either sign, detector offsets that do
and do not allow the reflection in z, voxels below and above one detector row apart, runs longer than
the volume, and detector edges inside the volume.  Bars: those of every FDK parity test (form_bars)."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu

G = dict(ns=48, nt=40, ds=1.0, dt=1.0, dsd=300.0, dod=100.0)
CASES = {
    # name: (geometry changes, image dims, deltas, offsets)
    "even": (dict(na=24), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "even odd sides": (dict(na=24), (21, 17, 15), (0.75, 0.75, 0.75), (0, 0, 0)),
    "odd": (dict(na=25), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "odd odd sides": (dict(na=25), (19, 19, 13), (0.75, 0.75, 0.75), (0, 0, 0)),
    "long z": (dict(na=24), (18, 18, 37), (0.75, 0.75, 0.375), (0, 0, 0)),
    "odd long z": (dict(na=25), (18, 18, 70), (0.75, 0.75, 0.25), (0, 0, 0)),
    "one plane": (dict(na=24), (18, 18, 1), (0.75, 0.75, 0.75), (0, 0, 0)),
    "start 90": (dict(na=24, orbit_start=90.0), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "start half step": (dict(na=24, orbit_start=7.5), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "start off axis": (dict(na=24, orbit_start=11.0), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "reversed": (dict(na=24, orbit=-360.0), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "two turns": (dict(na=34, orbit=720.0), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "short": (dict(na=21, orbit=200.0), (20, 18, 15), (0.75, 0.75, 0.75), (0, 0, 0)),
    "short long z": (dict(na=21, orbit=200.0), (20, 18, 67), (0.75, 0.75, 0.25), (0, 0, 0)),
    "offset x": (dict(na=24), (20, 18, 14), (0.75, 0.75, 0.75), (0.5, 0, 0)),
    "offset z": (dict(na=25), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 1.5)),
    "half row": (dict(na=25, offset_t=0.5), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "quarter row and bin": (dict(na=25, offset_t=0.25, offset_s=0.25), (20, 18, 14), (0.75, 0.75, 0.75), (0, 0, 0)),
    "negative spacings": (dict(na=25), (20, 18, 14), (-0.75, 0.75, -0.75), (0, 0, 0)),
    "rows apart": (dict(na=25), (20, 18, 12), (0.75, 0.75, 1.0), (0, 0, 0)),
    "rows far apart": (dict(na=24), (20, 18, 9), (0.75, 0.75, 2.25), (0, 0, 0)),
    "edges inside": (dict(na=24), (34, 30, 30), (1.25, 1.25, 1.25), (0, 0, 0)),
    "edges inside odd": (dict(na=25), (34, 30, 30), (1.25, 1.25, 1.25), (0, 0, 0)),
}


def _run(kind, name, storage, mask=False, passes=None):
    change, dims, deltas, offsets = CASES[name]
    g = dict(dict(kind=kind, offset_s=0.0, offset_t=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, **G), **change)
    ig = dict(dims=dims, deltas=deltas, offsets=tuple(float(o) for o in offsets))
    m = C.cyl_mask(ig, 5.0) if mask else None
    proj = O.ellipsoid_proj(g, C.ELL3).astype(np.float32)
    plan = S.plan_fbp(C.to_geom(g), C.to_image(ig, m), storage=storage)
    if passes:
        plan.set_view_passes(passes)
    ref = O.fdk(g, dict(ig, mask=m), proj)
    rec = S.fdk(plan, proj)
    rmse, maxrel = C.form_bars(storage, g["na"])
    assert O.rel_rmse(rec, ref) < rmse
    assert np.abs(rec - ref).max() <= maxrel * np.abs(ref).max()
    return rec


@pytest.mark.parametrize("kind", ["flat", "arc"])
@pytest.mark.parametrize("name", list(CASES))
def test_f32(cuda, kind, name):
    _run(kind, name, "f32")


@pytest.mark.parametrize("kind", ["flat", "arc"])
@pytest.mark.parametrize("name", ["even", "even odd sides", "odd", "odd long z", "long z", "edges inside", "reversed"])
def test_f16(cuda, kind, name):
    _run(kind, name, "f16")


@pytest.mark.parametrize("name", ["even odd sides", "odd odd sides"])
def test_masked_and_split_over_launches(cuda, name):
    a = _run("flat", name, "f32", mask=True)
    b = _run("flat", name, "f32", mask=True, passes=3)
    assert O.rel_rmse(a, b) < 1e-6  # the same taps summed in another order
