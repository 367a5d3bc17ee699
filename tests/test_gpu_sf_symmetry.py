"""Separable-footprint plans whose views share elements under the scan's symmetry (csrc/sgb_sf.cu):
both directions against the FP64 oracle and each other.  The cases decide the slots (reflections,
quarter turns, half turns, none; half-turn parallel scans; views that are their own images), odd and
even sides, masks, and image sizes with and without a split of the views.  Bars: those of the other
SF tests, 1e-5 relative RMSE against FP64 and 2e-6 for the adjoint."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu

FAN = dict(nb=56, d=1.0, offset=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, dsd=300.0, dod=100.0)
PAR = dict(nb=56, d=1.0, offset=0.0, orbit=180.0, orbit_start=0.0)
IMAGES = {"square": ((30, 30), (0.9, 0.9)), "odd": ((31, 31), (0.9, 0.9)), "wide": ((37, 24), (0.8, -0.9)),
          "larger": ((70, 66), (0.4, 0.4))}
SCANS = {"quarter turns": dict(na=20), "even": dict(na=22), "odd": dict(na=21), "start 90": dict(na=21, orbit_start=90.0),
         "off axis": dict(na=22, orbit_start=11.0), "quarter bin": dict(na=20, offset=0.25),
         "quarter bin even": dict(na=22, offset=0.25), "none": dict(na=21, orbit_start=11.0)}


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("image", list(IMAGES))
@pytest.mark.parametrize("scan", list(SCANS))
@pytest.mark.parametrize("kind", ["par", "arc", "flat"])
def test_pair(cuda, kind, scan, image, masked):
    g = dict(PAR if kind == "par" else FAN, kind=kind) | SCANS[scan]
    dims, deltas = IMAGES[image]
    ig = dict(dims=dims, deltas=deltas, offsets=(0.0, 0.0))
    m = C.cyl_mask(ig, 11.0) if masked else None
    rng = np.random.default_rng(len(scan) * 31 + dims[0])
    img = rng.random((dims[1], dims[0])).astype(np.float32)
    sino = rng.random((g["na"], g["nb"])).astype(np.float32)
    plan = S.SFPlan(C.to_geom(g), C.to_image(ig, m))
    p, b = plan.project(img), plan.backproject(sino)
    assert O.rel_rmse(p, O.sf_project(g, dict(ig, mask=m), img)) < 1e-5
    assert O.rel_rmse(b, O.sf_back(g, dict(ig, mask=m), sino)) < 1e-5
    fwd, adj = float((p.astype(np.float64) * sino).sum()), float((b.astype(np.float64) * img).sum())
    assert abs(fwd - adj) < 2e-6 * abs(fwd)
    assert np.array_equal(p, plan.project(img)) and np.array_equal(b, plan.backproject(sino))
