"""Pixels that lie exactly on the detector's first or last bin (2D, csrc/sgb_back2_kernel.cuh).

The reference takes a tap for 1 <= bb < nb (back-par.jl:307, back-fan.jl:328).  Pixels that share their bin
with the images of a pixel under the scan's symmetry see it from the other end where the image's bins run
the other way, so an exact tie decides differently for them.  With as many pixels as bins of the same size,
parallel views along an axis put the image's first and last columns and rows there; sinograms are smooth
and not zero at their ends.  Pixels of r <= n/2 are held to the 1e-5 of the other tests: the corners outside
see the detector's ends in other views too, where the FP32 position decides."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S
from sinograms import learned

pytestmark = pytest.mark.gpu


def _rows(na, nb, seed):
    rng = np.random.default_rng(seed)
    s, v = np.arange(nb)[None, :] / nb, np.arange(na)[:, None] / na
    rows = 3 + sum(rng.uniform(0.2, 1) * np.cos(2 * np.pi * (k * s + rng.uniform()) + 2 * np.pi * rng.integers(1, 4) * v)
                   for k in rng.uniform(0.3, 2.5, 5))
    return rows.astype(np.float32)


@pytest.mark.parametrize("form", ["plain", "symmetric", "fours"])
@pytest.mark.parametrize("dims, na, orbit", [((96, 96), 60, 180.0), ((96, 96), 60, 360.0), ((96, 96), 62, 180.0),
                                            ((96, 96), 62, 360.0), ((96, 64), 60, 360.0), ((97, 97), 60, 180.0),
                                            ((96, 96), 61, 360.0), ((64, 96), 61, 180.0), ((320, 320), 180, 180.0)])
@pytest.mark.parametrize("split", [0, 2])
def test_parallel_ties(cuda, dims, na, orbit, form, split):
    g = dict(kind="par", nb=max(dims), d=1.0, offset=0.0, na=na, orbit=orbit, orbit_start=0.0)
    ig = dict(dims=dims, deltas=(1.0, 1.0))
    plan = S.plan_fbp(C.to_geom(g), C.to_image(ig))
    plan.set_back_form(form, split)
    if form == "symmetric":
        assert plan.back_form()["images"] > 1
    rows = _rows(na, g["nb"], na)
    rec = learned.fbp_backproject(plan, rows)  # the plan's back-projection alone
    ref = O.fbp_back(g, ig, rows)
    x, y = O.image_axes(ig)
    disk = np.hypot(x[None, :], y[:, None]) <= max(dims) / 2
    assert O.rel_rmse(rec[disk], ref[disk]) < 1e-5
    scale = np.abs(ref[disk]).max()
    assert np.abs(rec - ref)[disk].max() < 1e-4 * scale
