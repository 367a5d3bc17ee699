"""The one-shot SF calls set up what one direction reads, in one block (csrc/sgb_sf.cu): device allocations and
frees are most of what a small call takes.  Their results are a plan's."""
import numpy as np
import pytest

import cases as C
import sinograms as S
from sinograms import _lib

pytestmark = pytest.mark.gpu

PAR = dict(kind="par", nb=101, na=61, d=1.0, offset=0.0, orbit=180.0, orbit_start=0.0)
FAN = dict(kind="arc", nb=101, na=60, d=1.0, offset=0.0, orbit=360.0, orbit_start=0.0, source_offset=0.0, dsd=400.0, dod=150.0)
SCANS = {"par": PAR, "par 11": dict(PAR, orbit_start=11.0), "arc": FAN, "arc 11": dict(FAN, orbit_start=11.0, na=61),
         "flat quarter bin": dict(FAN, kind="flat", offset=0.25), "one view": dict(PAR, na=1), "one bin": dict(PAR, nb=1)}


@pytest.mark.parametrize("shape", [(64, 64), (61, 37), (1, 1)])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("scan", list(SCANS))
def test_allocations_and_results(cuda, scan, masked, shape):
    import torch
    g = SCANS[scan]
    nx, ny = shape
    mask = np.hypot(*np.meshgrid(np.arange(nx) - nx / 2 + 0.5, np.arange(ny) - ny / 2 + 0.5)) < max(nx, ny) / 2.5
    rg, ig = C.to_geom(g), S.ImageGeom(shape, (0.9, 0.9), mask=mask if masked else None)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand((ny, nx), device="cuda", generator=gen)
    y = torch.rand((g["na"], g["nb"]), device="cuda", generator=gen)
    plan = S.SFPlan(rg, ig)
    before = _lib.device_alloc_count()
    back = S.backproject_sf(rg, ig, y)
    assert _lib.device_alloc_count() - before == 1
    before = _lib.device_alloc_count()
    fwd = S.project_sf(rg, ig, x)
    assert _lib.device_alloc_count() - before <= 2  # the tables; the rows of a split sum
    assert torch.equal(back, plan.backproject(y))
    # the same elements, none negative; a plan may add them up in other groups of lines.  At most 64 lines with
    # 8 pixels each that reach a bin, and 2^-24 of the sum for each addition, in both
    want = plan.project(x)
    assert torch.all((fwd - want).abs() <= 2 * 64 * 8 * 2.0 ** -24 * want.abs())
