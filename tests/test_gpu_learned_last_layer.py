"""The learned filter's loss and gradients at row lengths about the last layer's tiles (csrc/sgb_learned.cu,
conv_fwd_c1: 128 positions to a warp, 512 to a CTA, 16-byte copies where the rows allow them) and through its
data gradient, against the FP64 oracle with the same BF16 weights.  Bars: those of the other tests of these
passes, 1e-5 on the loss and 1e-4 on the gradients; neither pass's order of summation changes with the tile."""
import numpy as np
import pytest

import learned_oracle as LO
from sinograms import learned as LF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [9, 127, 128, 132, 511, 512, 516, 1025, 1540])
def test_row_lengths(cuda, L):
    rng = np.random.default_rng(L)
    p = (0.2 * rng.standard_normal(LO.nparams())).astype(np.float32)
    z = rng.standard_normal((3, L)).astype(np.float32)
    t = rng.standard_normal((3, L)).astype(np.float32)
    loss, g = LF.LearnedFilter(scale=0.9, params=p).loss_grad(z, t)
    lo, go = LO.loss_grad(p.astype(np.float64), z, t, 0.9, bf16_weights=True)
    assert loss == pytest.approx(lo, rel=1e-5)
    assert np.linalg.norm(g - go) / np.linalg.norm(go) < 1e-4
