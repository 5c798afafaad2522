"""A bound on the persistent blocks per SM: the queue's two kernels then run one after the other, with the
bytes of the side-by-side form."""
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes
from oracle import oracle

from .test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["batched", "refined"])
def test_a_bounded_bake_matches_the_oracle(form):
    inp, opts = scenes.outdoor(grid=33, chunks=2, boxes=10, point_lights=3, density=2.0, sky_samples=24, sun_samples=16,
                               bounce_samples=20)
    want = (oracle.bake(inp, opts)[0] if form == "batched" else
            oracle.bake_ex(inp, opts, mode=oracle.REFINED, eps=dl.DEFAULT_REFINE_EPSILON)["scene"])
    for bound in (0, 1, 3):
        report = dl._abi.DlBakeReport()
        assert_same(dl.bake(inp, opts, form=form, blocks_per_sm=bound, report=report), want)
        if bound:
            assert report.tuned_blocks_per_sm <= bound and report.tuned_gather_blocks_per_sm <= bound
