"""Every launch of the 2D back-projector (csrc/sgb_back2_kernel.cuh) against the FP64 oracle: pixels with
their images under the scan's symmetry (four by quarter turns or by reflections, two), slices in fours, and
neither, each alone and with the views split over a cluster.  The plan chooses between them by predicted
time, so each is asked for here, on images too small for the choice to take it; at sizes where it does, the
choice itself is held to.  Scans, images and bar (1e-5, FP32 arithmetic on smooth data inside the field of
view) are those of the tests of the plan's own choice."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S
from test_gpu_back2_symmetry import FAN, IMAGES, PAR, SCANS

pytestmark = pytest.mark.gpu

# images per pixel that a scan's symmetry gives a square and a wide image, full turns
SLOTS = {"quarter turns": (4, 4), "even": (4, 4), "odd": (2, 2), "start 90": (2, 2), "half step": (4, 4), "off axis": (2, 2),
         "off axis odd": (1, 1), "quarter bin": (2, 2), "quarter bin odd": (1, 1), "quarter bin turns": (4, 2)}


def _sino(g, ig, slices):
    rng = np.random.default_rng(g["na"] * 7 + ig["dims"][1] + slices)
    s = np.arange(g["nb"])[None, None, :]
    sino = np.zeros((slices, g["na"], g["nb"]))
    for _ in range(4):
        c = rng.uniform(20, 50, (slices, g["na"], 1))
        sino += rng.uniform(0.2, 1, (slices, g["na"], 1)) * np.exp(-((s - c) / 8) ** 2)
    return sino.astype(np.float32)


def _check(g, image, form, split, slices=1, images=None, mask=None):
    ig = dict(dims=image[0], deltas=image[1])
    m = C.cyl_mask(ig, mask) if mask else None
    plan = S.plan_fbp(C.to_geom(g), C.to_image(ig, m))
    plan.set_back_form(form, split)
    f = plan.back_form(slices)
    assert f["slices"] == (4 if form == "fours" else 1)
    assert f["images"] == (images if form == "symmetric" else 1) and (not split or f["split"] == split)
    sino = _sino(g, ig, slices)
    rec = S.fbp(plan, sino)
    for i in range(slices):
        assert O.rel_rmse(rec[i], O.fbp(g, dict(ig, mask=m), sino[i])) < 1e-5, i


@pytest.mark.parametrize("split", [1, 3])
@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan", [s for s in SCANS if max(SLOTS[s]) > 1])
@pytest.mark.parametrize("kind", ["arc", "flat", "par"])
def test_symmetric(cuda, kind, scan, image, split):
    g = dict(FAN if kind != "par" else dict(PAR, orbit=360.0), kind=kind) | SCANS[scan]
    _check(g, IMAGES[image], "symmetric", split, images=SLOTS[scan][image == "wide"], mask=None if split == 1 else 11.0)


@pytest.mark.parametrize("orbit", [180.0, -180.0])
@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan, images", [("quarter turns", 4), ("even", 4), ("odd", 4), ("start 90", 4), ("off axis", 4),
                                          ("off axis odd", 2)])
def test_symmetric_half_turn(cuda, scan, images, image, orbit):
    g = dict(PAR, kind="par") | SCANS[scan] | dict(orbit=orbit)
    if scan == "off axis" and image == "wide":
        images = 2
    _check(g, IMAGES[image], "symmetric", 2, images=images)


@pytest.mark.parametrize("slices", [1, 4, 6])
@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("image", ["square odd", "wide"])
@pytest.mark.parametrize("kind", ["arc", "flat", "par"])
def test_fours_and_plain(cuda, kind, image, split, slices):
    g = dict(FAN if kind != "par" else PAR, kind=kind) | SCANS["even"]
    _check(g, IMAGES[image], "fours", split, slices)
    _check(g, IMAGES[image], "plain", split, slices)


def test_choice_at_larger_sizes(cuda):
    """512 x 512 from 720 views of an arc: images of a pixel for one slice, fours for a stack of eight."""
    g = dict(kind="arc", nb=788, d=1.0, offset=0.0, na=720, orbit=360.0, orbit_start=0.0, source_offset=0.0, dsd=1200.0,
             dod=400.0)
    plan = S.plan_fbp(C.to_geom(g), S.ImageGeom((512, 512), (0.9, 0.9)))
    assert plan.back_form(1)["images"] == 4 and plan.back_form(8)["slices"] == 4
