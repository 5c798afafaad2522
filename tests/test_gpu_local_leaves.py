"""Local bounce gathers hold a ray's first leaf back (occluded_postponed): trees from a root that is one leaf to
several levels, opaque and alpha-tested, one lane a texel to a whole warp, in both triangle tests, against the
oracle word for word."""
import numpy as np
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


def _scene(faces, cells, alpha):
    meshes = [scenes.atlas_mesh(1, scenes.box_parts((0, 0, 0), (4, 3, 4), outward=False, faces=faces, cells=cells),
                                (0.8, 0.6, 0.4))]
    if alpha:
        screen = scenes.atlas_mesh(2, scenes.box_parts((1.5, 0.5, 1.2), (1.6, 2.0, 2.8), faces=(0,)), (0.5, 0.5, 0.5))
        screen.uv0 = screen.uv1.copy()
        screen.alpha = dl.AlphaTexture(2, 2, np.array([[255] * 4, [255, 255, 255, 0]] * 2, np.uint8).reshape(-1))
        meshes.append(screen)
    lights = [dl.BakeLight(id=7 + i, position=(1.0 + i, 1.5, 2.1), radius=6.0, illumination=dl.SINGLE_BOUNCE,
                           bounce=dl.BakeBounce(samples=33), transparency=dl.TRANSPARENCY_ENABLED) for i in range(2)]
    return dl.BakeInput(meshes, lights), dl.BakeOptions(pixel_density=3.0, photon_cube_resolution=16)


@pytest.mark.parametrize("form", ["batched", "bounce_refined"])
@pytest.mark.parametrize("alpha", [False, True])
@pytest.mark.parametrize("faces,cells", [((2,), 1), ((2, 3), 1), ((0, 1, 2, 3, 4, 5), 1), ((0, 1, 2, 3, 4, 5), 5)])
def test_few_and_many_leaves_match_the_oracle(faces, cells, alpha, form):
    inp, opts = _scene(faces, cells, alpha)
    mode = oracle.REFINED_BOUNCE if form == "bounce_refined" else None
    want = oracle.bake(inp, opts)[0] if mode is None else oracle.bake_ex(
        inp, opts, mode=mode, eps=dl.DEFAULT_REFINE_EPSILON)["scene"]
    for lanes, blocks in ((0, 0), (1, 6), (32, 8), (2, 9), (4, 10)):
        assert_same(dl.bake(inp, opts, form=form, sample_lanes=lanes, gather_min_blocks=blocks), want)


def test_local_lights_alone_match_the_oracle():
    # points, panels and tubes: rays that return to the nodes after each leaf, for every register budget
    inp, opts = scenes.soft_rooms(rooms=1, boxes_per_room=6, lights=6)
    opts.pixel_density = 6.0
    want, _, _ = oracle.bake(inp, opts)
    for blocks in (0, 7, 8, 9, 10, 12):
        assert_same(dl.bake(inp, opts, min_blocks=blocks), want)


def test_the_queues_two_kernels_match_the_oracle():
    # a sky alone, a sky with sun, points and panels behind it, and those alone, for every register budget
    inp, opts = scenes.outdoor(grid=17, chunks=2, boxes=5, point_lights=2, sky_samples=24, bounce_samples=20)
    opts.pixel_density = 2.0
    skies = [light for light in inp.lights if light.shape.kind == dl.SKY]
    others = [light for light in inp.lights if light.shape.kind != dl.SKY]
    assert skies and others
    for lights in (skies, skies + others, others):
        case = dl.BakeInput(inp.meshes, lights)
        want, _, _ = oracle.bake(case, opts)
        for blocks in (0, 7, 8, 9, 10, 12):
            assert_same(dl.bake(case, opts, min_blocks=blocks), want)
        for blocks in (6, 8, 9, 10):
            assert_same(dl.bake(case, opts, gather_min_blocks=blocks), want)
