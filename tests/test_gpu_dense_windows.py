"""Windows on both sides of the lines where the hard-threshold scatter leaves the boxes
for the load/store pipe (a block at every pixel; launches that save a wave by it): the
accumulators are the oracle's bit for bit (pre-rounded sums with room for 64 patches
times 8)."""
import numpy as np
import pytest

from gpu_util import graph_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tx", [0, 2])
@pytest.mark.parametrize("w,h,final", [(8, 8, False), (41, 37, False), (895, 17, False),
                                       (896, 17, False), (41, 37, True)])
def test_accumulators(cuda, engine_lib, oracle, w, h, final, tx):
    from bm3dcuda import synthetic as S
    noisy, clean = S.texture_clip(1, h, w, seed=w)
    win, ref = noisy[None], clean[None].astype(np.float32) if final else None
    kw = dict(sigma=7.0, radius=0, block_step=1, bm_range=2, extractor_exp=10, transform_2d=tx,
              transform_1d=tx)
    got = graph_run(win, ref, **kw)
    want = oracle.port_bm3d(win, ref, return_acc=True, **kw)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("w,h", [(227, 293), (245, 272), (227, 389), (242, 365)])
def test_waves_of_other_transforms(cuda, engine_lib, oracle, w, h):
    """444, 445, 592 and 593 CTAs; three planes."""
    from bm3dcuda import synthetic as S
    win = S.chroma_clip(1, h, w, seed=w)[0].transpose(1, 0, 2, 3).copy()
    kw = dict(sigma=[7.0, 4.0, 4.0], radius=0, block_step=3, bm_range=2, extractor_exp=8,
              chroma=True, transform_2d=2, transform_1d=1)
    got = graph_run(win, **kw)
    want = oracle.port_bm3d(win, return_acc=True, **kw)
    np.testing.assert_array_equal(got, want)
