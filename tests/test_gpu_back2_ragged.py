"""2D back-projection of images whose last tile row holds few pixels: a tile's rows past the image
take part in the kernel's loops and must stay inside the tile's staged detector segment.  Pixels of
about 4 bins put the image's centre row, some 300 bins away, outside it."""
import math

import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["flat", "arc", "par"])
@pytest.mark.parametrize("n", [33, 65, 97])
def test_ragged_image_equals_the_whole_tiles_around_it(cuda, kind, n):
    """The n x n image is the first n rows and columns of one of whole 32 x 32 tiles whose pixels lie
    at the same coordinates, for an orbit without symmetry (views of an odd scan that starts off the
    axes), so that no pixel takes its geometry from another.  Each pixel's taps are the same in both; only the order of the views'
    FP32 sum can differ (the view split follows the tile count): na * 2^-24 = 8e-6 bounds it, and 1e-6
    is its size for independent roundings."""
    g = dict(kind=kind, nb=951, d=1.0, offset=0.0, na=131, orbit=360.0, orbit_start=11.0)
    if kind != "par":
        g.update(source_offset=0.0, dsd=1093.3, dod=394.3)
    m = (n + 31) // 32 * 32
    dx = 1.9 * (270.0 if kind != "par" else 470.0) / math.hypot(m, m)
    off = (n - m) / 2  # pixel i at dx (i - (n - 1) / 2) in both
    rows = np.random.default_rng(n).standard_normal((131, 951)).cumsum(1).astype(np.float32)
    rg = C.to_geom(g)
    rec = S.fbp(S.plan_fbp(rg, S.ImageGeom((n, n), (dx, dx))), rows)
    whole = S.fbp(S.plan_fbp(rg, S.ImageGeom((m, m), (dx, dx), (off, off))), rows)
    assert O.rel_rmse(rec, whole[:n, :n]) < 1e-6
