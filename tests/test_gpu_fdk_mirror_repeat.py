"""The mirrored FDK back-projector's stages (csrc/sgb_fdk_mirror_kernel.cuh) are complete when they are
published: two lanes write a stage's record (the columns s and -s), one arrives for both.  A warp that read
the columns of the stage's previous view would take other samples, so a call's result would vary with the
warps' timing.  The sums have a fixed order: repeated calls must agree in every bit, and with the oracle."""
import numpy as np
import pytest

import cases as C
import oracle as O
import sinograms as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na", [120, 121])  # four view slots; two (reflection in x), with z and -z in FP32
@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("kind", ["flat", "arc"])
def test_repeated_calls_agree(cuda, kind, storage, na):
    g = dict(kind=kind, ns=80, nt=48, ds=1.0, dt=1.0, dsd=300.0, dod=100.0, offset_s=0.25, offset_t=0.0, orbit=360.0,
             orbit_start=0.0, source_offset=0.0, na=na)
    ig = dict(dims=(48, 44, 20), deltas=(0.75, 0.75, 0.75), offsets=(0.0, 0.0, 0.0))
    proj = O.ellipsoid_proj(g, C.ELL3).astype(np.float32)
    plan = S.plan_fbp(C.to_geom(g), C.to_image(ig), storage=storage)
    plan.set_mirror(True)
    first = S.fdk(plan, proj)
    assert O.rel_rmse(first, O.fdk(g, ig, proj)) < C.form_bars(storage, na)[0]
    for _ in range(30):
        assert np.array_equal(S.fdk(plan, proj), first)
