"""The non-allocating bounce filter's tiles (32 x 8 texels, halo 4): windows of one texel, at and
across tile edges, thin in either direction and placed at the map's corners, against the oracle's
BounceMap (dilation and blur of bounce_map.rs:67-112) bit for bit, which restates the same binary32
operations in the same order."""
import ctypes as C

import numpy as np
import pytest

import dynlight_gb300 as dl
from oracle import oracle
from oracle.oracle import ptr

pytestmark = pytest.mark.gpu

# window corner (x0, y0) and size inside a 200-texel map; a BounceMap's window is its texels' rectangle
# grown by 4 and clipped to the map, so a window narrower than 9 texels touches the map's edge
WINDOWS = [(0, 0, 5, 5), (0, 0, 32, 8), (0, 0, 33, 9), (195, 0, 5, 40), (0, 192, 200, 8), (3, 7, 31, 9), (17, 11, 64, 16),
           (101, 50, 65, 17), (0, 0, 200, 200), (135, 183, 65, 17)]


@pytest.mark.parametrize("x0,y0,w,h", WINDOWS)
def test_tiles_match_the_oracle(x0, y0, w, h):
    torch = pytest.importorskip("torch")
    lib, size = dl.load_library(), 200
    rng = np.random.default_rng(x0 * 7 + y0 * 5 + w * 3 + h)
    grow = lambda lo, n: (lo if lo == 0 else lo + 4, lo + n - 1 if lo + n == size else lo + n - 5)  # noqa: E731
    (ax, bx), (ay, by) = grow(x0, w), grow(y0, h)
    n = max(1, w * h // 6)
    xs, ys = rng.integers(ax, bx + 1, n), rng.integers(ay, by + 1, n)
    vals = rng.random((n, 3), dtype=np.float32) * (rng.random((n, 1)) > 0.2)
    tex = np.ascontiguousarray(np.concatenate([np.stack([xs, ys], 1), vals], 1).astype(np.float32))
    want, win = np.zeros(w * h * 3, np.float32), (C.c_uint32 * 4)()
    oracle.lib().oracle_bounce_map(size, (C.c_uint32 * 4)(ax, ay, bx, by), ptr(tex), n, ptr(want), win)
    assert list(win) == [x0, y0, x0 + w - 1, y0 + h - 1]
    pre = np.zeros((h, w, 3), np.float32)
    for (x, y), v in zip(zip(xs, ys), tex[:, 2:]):
        pre[y - y0, x - x0] = v
    src = torch.from_numpy(pre.reshape(-1)).cuda()
    out = torch.full((w * h * 3,), float("nan"), dtype=torch.float32, device="cuda")
    status = lib.dl_filter_bounce_window_noalloc(C.c_void_p(src.data_ptr()), C.c_void_p(out.data_ptr()), w, h, x0, y0,
                                                 size, None)
    assert status == 0, lib.dl_last_error()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
