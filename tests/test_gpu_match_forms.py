"""The matching kernel's forms give the oracle's lists: one lane per reference
block or several (chosen by how many blocks a launch has), two-entry or full
temporal lists (ps_num), and every strip width a search range selects."""
import numpy as np
import pytest

from gpu_util import graph_run

pytestmark = pytest.mark.gpu


def window(h, w, radius, kind, seed):
    from bm3dcuda import synthetic as S
    frames, _ = S.texture_clip(2 * radius + 1, h, w, seed=seed)
    if kind == "ties":  # 3-level steps without noise: most distances tie exactly
        frames = (np.round(frames * 4) / 4).astype(np.float32)
    return frames[None]


# warps of 4 x 8 blocks per launch choose the form
SIZES = [
    (8, 8, 8),        # one block
    (41, 67, 8),      # clamped last blocks, a few warps
    (120, 97, 2),     # 96 warps: 8 lanes per block
    (100, 90, 1),     # 252: 4 lanes
    (100, 260, 1),    # 768: one lane, 200 registers
    (163, 203, 1),    # 980
    (390, 420, 1),    # 4944: one lane, 168 registers
]


@pytest.mark.parametrize("kind", ["texture", "ties"])
@pytest.mark.parametrize("radius,ps_num", [(0, 2), (1, 1), (2, 2), (1, 3), (1, 8)])
@pytest.mark.parametrize("h,w,step", SIZES)
def test_lists_of_every_form(cuda, engine_lib, oracle, h, w, step, radius, ps_num, kind):
    win = window(h, w, radius, kind, seed=h + radius)
    kw = dict(sigma=8.0, block_step=step, bm_range=4, radius=radius, ps_num=ps_num, ps_range=2)
    _, got = graph_run(win, return_matches=True, **kw)
    _, want = oracle.port_bm3d(win, return_matches=True, **kw)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("step", [8, 5, 4, 3])
@pytest.mark.parametrize("bm_range,ps_range", [(3, 3), (7, 4), (9, 5), (5, 8), (12, 6), (17, 1)])
def test_lists_of_every_strip_width(cuda, engine_lib, oracle, bm_range, ps_range, step):
    win = window(70, 91, 1, "texture", seed=bm_range)
    kw = dict(sigma=8.0, block_step=step, bm_range=bm_range, radius=1, ps_num=2, ps_range=ps_range)
    _, got = graph_run(win, return_matches=True, **kw)
    _, want = oracle.port_bm3d(win, return_matches=True, **kw)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("metric", [1, 2, 3, 4])
@pytest.mark.parametrize("h,w,step,bm_range,radius,ps_num,ps_range", [
    (8, 8, 8, 9, 0, 2, 4),       # one block
    (41, 67, 8, 9, 1, 2, 4),     # strips of 10: 19 and 9 columns
    (40, 52, 5, 3, 1, 3, 3),     # strips of 8: 7 columns
    (163, 203, 1, 4, 0, 2, 4),   # one lane per block
])
def test_lists_of_other_distances(cuda, engine_lib, oracle, metric, h, w, step, bm_range, radius,
                                  ps_num, ps_range):
    win = window(h, w, radius, "texture", seed=metric)
    kw = dict(sigma=8.0, block_step=step, bm_range=bm_range, radius=radius, ps_num=ps_num,
              ps_range=ps_range, bm_error=metric)
    _, got = graph_run(win, return_matches=True, **kw)
    _, want = oracle.port_bm3d(win, return_matches=True, **kw)
    np.testing.assert_array_equal(got, want)
