"""No warp vote takes its lanes from __activemask(): read inside divergent code it names whichever lanes happen to be
together, and a *_sync operation waits for every lane it names. The gather, whose traversal did so, against the
oracle where a warp holds lanes with and without rays."""
import glob
import os
import re

import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_collective_takes_its_mask_from_the_active_lanes():
    sources = glob.glob(os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc", "*"))
    assert len(sources) >= 8
    for path in sources:
        with open(path) as f:
            code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        assert not re.search(r"_sync\s*\(\s*__activemask\b", code), path
        assert not re.search(r"=\s*__activemask\s*\(", code), path  # nor through a variable


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [0, 1, 2, 8, 32])
@pytest.mark.parametrize("form", ["batched", "bounce_refined"])
def test_lanes_with_and_without_rays_match_the_oracle(form, lanes):
    # warps that hold texels out of a light's reach, lights of different sample counts, and suns in
    # index order and in a net's order beside local lights
    inp, opts = scenes.outdoor(grid=17, chunks=2, boxes=6, point_lights=4, density=2.0, sun_samples=16, sky_samples=16,
                               bounce_samples=20)
    local = [light for light in inp.lights if light.shape.kind not in (dl.SUN, dl.SKY)]
    sun = next(light for light in inp.lights if light.shape.kind == dl.SUN)
    for light, samples, radius in zip(local, (2, 3, 33, 7), (30.0, 3.0, 12.0, 60.0)):
        light.illumination, light.bounce, light.radius = dl.SINGLE_BOUNCE, dl.BakeBounce(samples=samples), radius
    opts.photon_cube_resolution = 16
    for bounce in (20, 96):
        sun.bounce = dl.BakeBounce(samples=bounce)
        case = dl.BakeInput(inp.meshes, [sun] + local)
        want = (oracle.bake(case, opts)[0] if form == "batched" else
                oracle.bake_ex(case, opts, mode=oracle.REFINED_BOUNCE, eps=dl.DEFAULT_REFINE_EPSILON)["scene"])
        assert_same(dl.bake(case, opts, form=form, sample_lanes=lanes), want)
