"""What the timing trials keep for later bakes of a scene is the register budget alone: sample lanes and the sun
gather's buffer follow from each bake's own sample counts and memory cap, whatever was baked before."""
import pytest

import dynlight_gb300 as dl
from dynlight_gb300 import scenes

pytestmark = pytest.mark.gpu


def _bake(boxes, sky, bounce, **config):
    # a scene of its own for each test (`boxes`): over a million queue items and 256 K gather items: both stages time their budgets
    inp, opts = scenes.outdoor(grid=193, chunks=2, boxes=boxes, point_lights=2, sky_samples=sky, bounce_samples=bounce,
                               sun_samples=16)
    report = dl._abi.DlBakeReport()
    baked = dl.bake(inp, opts, report=report, **config)
    assert report.work_items >= 1 << 20 and report.bounce_items >= 1 << 18
    return baked, report


@pytest.mark.parametrize("boxes,first,then", [(150, (32, 16), (256, 128)), (152, (256, 128), (32, 16))])
def test_sample_counts_set_the_shape_whatever_came_before(boxes, first, then):
    _, rule = _bake(boxes, *then, no_autotune=1)
    _bake(boxes, *first)
    for _ in range(2):  # trials, then the kept budget
        baked, report = _bake(boxes, *then)
        assert report.tuned_sample_lanes == rule.tuned_sample_lanes
        assert report.tuned_gather_lanes == rule.tuned_gather_lanes
        # the buffer of 128 samples for every lane group is some 100 MB; the budgets tried differ by a tenth of it
        assert abs(report.device_bytes - rule.device_bytes) < 40 << 20
    assert report.tune_trials == 0


def test_a_capped_bake_takes_no_buffer_from_an_uncapped_one():
    # 96 samples gather from a buffer of 128 without a cap, in index order without a buffer under one
    want, free = _bake(154, 16, 96)
    _, alone = _bake(154, 16, 96, no_autotune=1, max_device_mib=1 << 16)
    assert alone.device_bytes < free.device_bytes - (60 << 20)
    cap = (alone.device_bytes >> 20) + 24  # slack for scan and trial scratch
    for _ in range(2):
        baked, report = _bake(154, 16, 96, max_device_mib=cap)
        assert baked.words_equal(want) and baked.stats == want.stats
        assert report.device_bytes <= alone.device_bytes + (24 << 20)
    again, report = _bake(154, 16, 96)  # and the other way round
    assert again.words_equal(want) and report.device_bytes > alone.device_bytes + (60 << 20)
