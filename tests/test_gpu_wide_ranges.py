"""Search ranges near the limit of what is accepted, in launches small enough to
ask for several lanes per reference block: the lists are the oracle's."""
import numpy as np
import pytest

from gpu_util import graph_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,block_step,bm_range,radius,ps_range,metric", [
    (480, 400, 6, 96, 0, 4, 0),    # 180 warps: the four-lane tile does not fit
    (250, 200, 3, 95, 1, 6, 0),    # 189
    (180, 150, 2, 93, 2, 6, 0),    # 198
    (117, 83, 2, 93, 2, 6, 0),     # 8 lanes, at the smallest row pitch
    (117, 83, 2, 93, 2, 6, 1),     # SAD
    (117, 83, 3, 101, 0, 4, 0),    # the largest range of its step
    (117, 83, 8, 88, 0, 4, 0),
])
def test_lists_near_the_limit(cuda, engine_lib, oracle, w, h, block_step, bm_range, radius,
                              ps_range, metric):
    from bm3dcuda import synthetic as S
    frames, _ = S.texture_clip(2 * radius + 1, h, w, seed=block_step)
    kw = dict(sigma=8.0, block_step=block_step, bm_range=bm_range, radius=radius, ps_num=2,
              ps_range=ps_range, bm_error=metric)
    _, got = graph_run(frames[None], return_matches=True, **kw)
    _, want = oracle.port_bm3d(frames[None], return_matches=True, **kw)
    np.testing.assert_array_equal(got, want)
