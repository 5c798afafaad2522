"""The refined form's closest hits where binary32 leaves their order open: triangles that coincide or lie
a few units in the last place above one another, and slivers whose binary32 distances have no useful
bound, against the oracle's refined bake, which tests every candidate in binary64."""
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["refined", "bounce_refined"])
@pytest.mark.parametrize("lift", [0.0, 1e-6, 3e-5])
def test_open_orders_follow_binary64(lift, form):
    inp, opts = scenes.precision_stress(grid=24, chunks=2, boxes=6, decals=500, slivers=120, lights=5, sky_samples=16,
                                        bounce_samples=32, decal_lift=lift, area_samples=16, density=3.0)
    for light in inp.lights:
        light.illumination = dl.SINGLE_BOUNCE
        light.bounce = dl.BakeBounce(samples=32)
    opts.photon_cube_resolution = 48
    mode = oracle.REFINED if form == "refined" else oracle.REFINED_BOUNCE
    want = oracle.bake_ex(inp, opts, mode=mode, eps=dl.DEFAULT_REFINE_EPSILON)["scene"]
    assert_same(dl.bake(inp, opts, form=form), want)
