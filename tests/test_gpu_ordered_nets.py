"""Sample counts that are no powers of two in the coherent order of the next larger net (ordered_net):
at and around the share where the order is taken, below and above its limits, for every group
size, against the oracle word for word (a sky's open count and a sun bounce's ordered sum)."""
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sky,bounce", [(9, 19), (10, 20), (11, 33), (19, 40), (20, 39), (100, 45), (200, 96), (257, 161),
                                        (321, 160), (64, 257), (40, 256)])
def test_counts_between_powers_of_two_match_the_oracle(sky, bounce):
    inp, opts = scenes.outdoor(grid=25, chunks=2, boxes=8, point_lights=1, sky_samples=sky, bounce_samples=bounce)
    opts.pixel_density = 2.0
    want, _, _ = oracle.bake(inp, opts)
    for lanes in (0, 1, 8, 32):
        assert_same(dl.bake(inp, opts, sample_lanes=lanes), want)
    # under a device-memory cap such counts gather without the order's scratch
    assert_same(dl.bake(inp, opts, max_device_mib=4096), want)
