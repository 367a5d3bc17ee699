"""Distance-driven pair (csrc/sgb_bdd.cu) where its kernels' splits can go wrong, against the FP64
oracle: bins from 0.3 to 6 pixels wide (no, one and several whole pixels inside a bin, and both sides
of the line between the direct and the prefix projector); bin counts about the 31-bin groups, a
warp's four groups and a CTA's 32; image sides about the 31-pixel groups, a warp's nine, and the
staged rows' pitch; tables too large for two stages.  Bar: 1e-5 relative RMSE, that of the other
distance-driven tests; a mapped boundary's FP32 position is good to 2^-24 nPix pixels, 3e-5 of a
pixel at the largest side here, under bins or pixels of at least 0.3."""
import numpy as np
import pytest

import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu

DSD, DS0 = 949.0, 541.0


def check(npix, ndet, na, arc, span, forward=True, side=200.0):
    # `span`: the detector's width over the image's, both at the centre
    psize = side / npix
    dsize = span * side / ndet * DSD / DS0
    angle = np.linspace(0, 2 * np.pi, na, endpoint=False)
    geo = S.BddGeo(DSD, DS0, psize, dsize, npix, ndet, angle, **(dict(arc=True) if arc else {}))
    ogeo = O.bdd_geo(DSD, DS0, psize, dsize, npix, ndet, angle, arc=arc)
    rng = np.random.default_rng(npix + 7 * ndet + na)
    x = rng.random((npix, npix), dtype=np.float32)
    y = rng.random((ndet, na), dtype=np.float32)
    if forward:
        assert O.rel_rmse(S.project_bdd(x, geo), O.project_bdd(x, ogeo)) < 1e-5
    assert O.rel_rmse(S.backproject_bdd(y, geo), O.backproject_bdd(y, ogeo)) < 1e-5


@pytest.mark.parametrize("arc", [False, True])
@pytest.mark.parametrize("step", [0.3, 0.97, 1.04, 1.9, 2.1, 3.2, 5.9, 6.1])
def test_bin_widths(cuda, step, arc):
    ndet = round(1.3 * 62 / step)
    check(62, ndet, 9, arc, step * ndet / 62)


@pytest.mark.parametrize("npix,ndet", [(1, 4), (3, 12), (4, 16), (9, 31), (9, 32), (31, 124), (35, 125), (36, 125),
                                       (60, 249), (250, 993), (279, 64), (280, 300), (560, 90), (64, 1), (64, 2)])
def test_sizes(cuda, npix, ndet):
    check(npix, ndet, 8, False, 1.3)


@pytest.mark.parametrize("ndet", [33, 1025, 2050])
def test_prefix_projector_splits(cuda, ndet):
    check(62, ndet, 4, False, 7 * ndet / 62, side=2.0)  # bins of 7 pixels under a small image


def test_large_tables(cuda):
    check(40, 7100, 3, True, 1.2, forward=False)  # the projector refuses this many bins
