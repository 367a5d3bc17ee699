"""2D FBP plans whose pixels share their geometry (csrc/sgb_back2_kernel.cuh): the images of a pixel
under the scan's symmetry, and the slices of a stack, against the FP64 oracle.

Each case decides the slots: quarter turns (square images, 90 degrees a whole number of views),
reflections in both axes or one, half turns, none; full, half (parallel beams) and repeated turns;
odd and even sides; spacings of either sign; detectors that reversed bins do and do not fit.  Slices
1 (no sharing), 2 and 5 (a full and a ragged group of four).  Images lie inside the field of view;
the bar is the 1e-5 of every FP32 parity test on smooth data."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu

FAN = dict(nb=72, d=1.0, offset=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, dsd=300.0, dod=100.0)
PAR = dict(nb=72, d=1.0, offset=0.0, orbit=180.0, orbit_start=0.0)
IMAGES = {
    "square": ((40, 40), (0.7, 0.7)),
    "square odd": ((41, 41), (0.7, 0.7)),
    "square, y down": ((40, 40), (0.7, -0.7)),
    "wide": ((50, 37), (0.6, 0.6)),
}
SCANS = {
    "quarter turns": dict(na=40),
    "even": dict(na=42),
    "odd": dict(na=41),
    "start 90": dict(na=41, orbit_start=90.0),
    "half step": dict(na=42, orbit_start=180.0 / 42),
    "off axis": dict(na=42, orbit_start=11.0),
    "off axis odd": dict(na=41, orbit_start=11.0),
    "quarter bin": dict(na=42, offset=0.25),
    "quarter bin odd": dict(na=41, offset=0.25),
    "quarter bin turns": dict(na=40, offset=1.25),
}


def _check(g, image, slices):
    dims, deltas = image
    ig = dict(dims=dims, deltas=deltas)
    # sums of Gaussian bumps along each row: smooth, nothing symmetric about them
    rng = np.random.default_rng(g["na"] * 7 + dims[1])
    s = np.arange(g["nb"])[None, None, :]
    sino = np.zeros((slices, g["na"], g["nb"]))
    for _ in range(4):
        c = rng.uniform(20, 50, (slices, g["na"], 1))
        sino += rng.uniform(0.2, 1, (slices, g["na"], 1)) * np.exp(-((s - c) / 8) ** 2)
    sino = sino.astype(np.float32)
    rec = S.fbp(S.plan_fbp(C.to_geom(g), C.to_image(ig)), sino if slices > 1 else sino[0])
    for i in range(slices):
        assert O.rel_rmse(rec[i] if slices > 1 else rec, O.fbp(g, ig, sino[i])) < 1e-5, i


@pytest.mark.parametrize("slices", [1, 2, 5])
@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan", list(SCANS))
def test_fan(cuda, scan, image, slices):
    kind = "arc" if (len(scan) + slices) % 2 else "flat"
    _check(dict(FAN, kind=kind) | SCANS[scan], IMAGES[image], slices)


@pytest.mark.parametrize("slices", [1, 5])
@pytest.mark.parametrize("orbit", [180.0, -180.0, 360.0])
@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan", list(SCANS))
def test_par(cuda, scan, image, orbit, slices):
    _check(dict(PAR, kind="par") | SCANS[scan] | dict(orbit=orbit), IMAGES[image], slices)


def test_fan_source_offset_and_two_turns(cuda):
    _check(dict(FAN, kind="flat") | dict(na=40, source_offset=1.5), IMAGES["square"], 1)
    _check(dict(FAN, kind="arc") | dict(na=34, orbit=720.0), IMAGES["wide"], 2)
