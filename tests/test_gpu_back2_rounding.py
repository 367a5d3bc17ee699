"""The 2D back-projector adds a tap to a pixel's sum with one rounding (csrc/sgb_back2_kernel.cuh).

A rounding of a sum of size v has an rms error of 2.53e-8 v (half a unit in the last place, uniform, over
mantissas spread logarithmically: 2^-23 / sqrt(12) * sqrt(3 / (8 ln 2))).  Over n positive taps of one size the
sum grows linearly and the roundings add up to 2.53e-8 sqrt(n / 3) of it: 5.06e-7 for 1200 views in one
thread block.  Two roundings a tap make that 7.2e-7.  The bar is 1.2 times the former; the rows are smooth,
so that the taps' own errors (a bin coordinate's 2^-16) stay below 1e-8."""
import math

import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S
from sinograms import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form, slices", [("plain", 1), ("symmetric", 1), ("fours", 4)])
@pytest.mark.parametrize("dims", [(64, 64), (64, 48)])  # quarter turns, reflections
def test_one_rounding_per_tap(cuda, dims, form, slices):
    na, nb = 1200, 128
    g = dict(kind="par", nb=nb, d=1.0, offset=0.0, na=na, orbit=360.0, orbit_start=0.0)
    ig = dict(dims=dims, deltas=(0.6, 0.6))
    s, v = np.arange(nb) / nb, np.arange(na)[:, None] / na
    rows = (2 + 0.5 * np.cos(2 * np.pi * (0.7 * s + v))).astype(np.float32)
    plan = S.plan_fbp(C.to_geom(g), C.to_image(ig))
    plan.set_back_form(form, 1)
    rec = learned.fbp_backproject(plan, np.stack([rows] * slices))
    assert O.rel_rmse(rec[-1], O.fbp_back(g, ig, rows)) < 1.2 * 2.53e-8 * math.sqrt(na / 3)
