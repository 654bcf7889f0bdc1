"""The run-time-compiled plugin's distances in every form of the search (strips of
4, 8 and 10, two-entry and full temporal lists, one or four lanes per block, two or
three CTAs per SM): the lists are the oracle's."""
import numpy as np
import pytest

from gpu_util import graph_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [1, 2, 3, 4])
@pytest.mark.parametrize("w,h,step,bm_range,radius,ps_num,ps_range", [
    (67, 41, 8, 1, 0, 2, 4),     # strips of 4, four lanes
    (150, 140, 2, 2, 0, 2, 4),   # strips of 8
    (330, 300, 1, 1, 0, 2, 4),   # strips of 4, three CTAs per SM
    (330, 300, 1, 4, 0, 2, 4),   # strips of 10, three CTAs per SM
    (60, 51, 4, 5, 1, 2, 1),     # strips of 4
    (60, 51, 4, 3, 1, 2, 3),     # strips of 8
    (60, 51, 4, 9, 1, 4, 4),     # full lists: strips of 10
    (60, 51, 5, 4, 1, 8, 1),     # strips of 4
    (60, 51, 5, 3, 2, 3, 3),     # strips of 8
    (330, 230, 2, 5, 1, 2, 1),   # one lane, two-entry lists: strips of 4
    (330, 230, 2, 5, 1, 1, 1),   # strips of 8
])
def test_lists(cuda, engine_lib, oracle, metric, w, h, step, bm_range, radius, ps_num, ps_range):
    from bm3dcuda import synthetic as S
    win = S.texture_clip(2 * radius + 1, h, w, seed=metric)[0][None]
    kw = dict(sigma=8.0, block_step=step, bm_range=bm_range, radius=radius, ps_num=ps_num,
              ps_range=ps_range, bm_error=metric)
    _, got = graph_run(win, return_matches=True, **kw)
    _, want = oracle.port_bm3d(win, return_matches=True, **kw)
    np.testing.assert_array_equal(got, want)
