"""The separable-footprint pair has one matrix (csrc/sgb_sf.cu): every element is the same FP32 number in both
directions, whichever views and pixels share its evaluation.  The projection of a single pixel gives a row of
elements with nothing added to them, the back-projection of a single bin a column."""
import numpy as np
import pytest

import cases as C
import sinograms as S

pytestmark = pytest.mark.gpu

FAN = dict(nb=26, d=1.0, offset=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, dsd=140.0, dod=50.0)
PAR = dict(nb=26, d=1.0, offset=0.0, orbit=180.0, orbit_start=0.0)
SCANS = {"quarter turns": dict(na=12), "even": dict(na=14), "odd": dict(na=13), "start 90": dict(na=13, orbit_start=90.0),
         "off axis": dict(na=14, orbit_start=11.0), "off axis turns": dict(na=12, orbit_start=11.0),
         "quarter bin": dict(na=14, offset=0.25), "quarter bin turns": dict(na=12, offset=0.25),
         "none": dict(na=13, orbit_start=11.0)}
IMAGES = {"square": ((14, 14), (0.9, 0.9)), "odd, y down": ((13, 13), (0.9, -0.9)), "wide": ((16, 11), (0.8, 0.8))}


@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan", list(SCANS))
@pytest.mark.parametrize("kind, orbit", [("par", 180.0), ("par", -180.0), ("par", 360.0), ("arc", 360.0), ("flat", 360.0)])
def test_whole_matrix(cuda, kind, orbit, scan, image):
    import torch
    g = dict(PAR if kind == "par" else FAN, kind=kind) | SCANS[scan] | dict(orbit=orbit)
    (nx, ny), deltas = IMAGES[image]
    plan = S.SFPlan(C.to_geom(g), S.ImageGeom((nx, ny), deltas))
    pixels = torch.eye(nx * ny, device="cuda").reshape(-1, ny, nx)
    bins = torch.eye(g["na"] * g["nb"], device="cuda").reshape(-1, g["na"], g["nb"])
    fwd = torch.stack([plan.project(p).flatten() for p in pixels])
    back = torch.stack([plan.backproject(b).flatten() for b in bins])
    assert (fwd != 0).sum() > nx * ny * g["na"]
    assert torch.equal(fwd, back.T)


@pytest.mark.parametrize("kind", ["arc", "flat", "par"])
def test_elements_of_a_large_scan(cuda, kind):
    """888 bins: 1 bit of a bin coordinate is 3e-5 bins there."""
    import torch
    kw = dict(nb=888, na=90, d=1.0239, orbit=360.0)
    rg = S.SinoPar(**kw) if kind == "par" else (S.SinoFanArc if kind == "arc" else S.SinoFanFlat)(dsd=949.075, dod=408.075, **kw)
    plan = S.SFPlan(rg, S.ImageGeom((512, 512), (0.9766, 0.9766)))
    rng = np.random.default_rng(5)
    for _ in range(6):
        x, y = (int(v) for v in rng.integers(0, 512, 2))
        img = torch.zeros((512, 512), device="cuda")
        img[y, x] = 1
        p = plan.project(img)
        hits = p.nonzero()
        for a, k in hits[torch.as_tensor(rng.integers(0, len(hits), 30), device="cuda")].tolist():
            sino = torch.zeros((90, 888), device="cuda")
            sino[a, k] = 1
            assert plan.backproject(sino)[y, x] == p[a, k], (a, k)
