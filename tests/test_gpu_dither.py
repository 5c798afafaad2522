"""Dithered bounce packing (6, 5 and 4 bits): whole rounds, ragged last rounds and crops from a few
texels to thousands, white and colored, against the oracle's sequential packer word for word."""
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("colored", [False, True])
@pytest.mark.parametrize("bits,density", [(6, 3.0), (5, 9.0), (4, 20.0), (6, 13.0)])
def test_dithered_words_match_the_oracle(bits, density, colored):
    inp, opts = scenes.small_room(lights=2)
    for k, light in enumerate(inp.lights):
        light.illumination = dl.SINGLE_BOUNCE
        light.bounce = dl.BakeBounce(samples=8, intensity=1.5 if k else 0.02)  # lit, and mostly below the draw
    opts.pixel_density, opts.bounce_compression, opts.colored_bounce = density, bits, colored
    opts.photon_cube_resolution = 32
    for k, mesh in enumerate(inp.meshes):
        mesh.albedo = (0.9, 0.4, 0.05 * (k + 1))
    want, _, _ = oracle.bake(inp, opts)
    assert_same(dl.bake(inp, opts), want)
