"""The scatter by TMA reductions (clip path, aggregated output) at the widths
where its 12-column boxes meet the plane's edges, against the oracle bit for
bit (pre-rounded sums); the reciprocal it shares with the Wiener shrinkage."""
import ctypes

import numpy as np
import pytest

from gpu_util import aggregate, graph_run
from test_gpu_parity import port_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("final", [False, True])
@pytest.mark.parametrize("radius", [0, 1])
@pytest.mark.parametrize("h,w", [(8, 8), (9, 11), (17, 32), (40, 33), (31, 64), (24, 97)])
def test_box_edges(cuda, engine_lib, oracle, h, w, radius, final):
    from bm3dcuda import BM3Dv2, Clip
    from bm3dcuda import synthetic as S
    noisy, clean = S.texture_clip(3, h, w, seed=w + h)
    ref = clean if final else None
    # every column phase of the boxes: block_step 3
    kw = dict(sigma=7.0, radius=radius, block_step=3, bm_range=5, extractor_exp=6)
    got = BM3Dv2(Clip.from_array(noisy), ref=Clip.from_array(clean) if final else None,
                 **kw).to_array()
    if radius:
        want = port_clip(oracle, noisy[:, None], ref[:, None] if final else None, **kw)[:, 0]
    else:
        # the oracle's spatial aggregation multiplies by a reciprocal, as the
        # reference's does; here the IEEE quotient of the accumulators, which
        # the window path scatters without TMA (equal to the oracle's bit for bit)
        want = np.stack([aggregate(graph_run(noisy[n][None, None],
                                             clean[n][None, None] if final else None, **kw))[0]
                         for n in range(3)])
    np.testing.assert_array_equal(got, want)


def test_reciprocal_is_correctly_rounded(cuda, engine_lib):
    bad, first = ctypes.c_ulonglong(), ctypes.c_uint()
    assert engine_lib.bm3d_b200_selftest_reciprocal(0x00800000, 0x7E800000, ctypes.byref(bad),
                                                    ctypes.byref(first)) == 0
    assert bad.value == 0, hex(first.value)


@pytest.mark.parametrize("final", [False, True])
@pytest.mark.parametrize("radius,planes", [(0, 1), (1, 1), (1, 3)])
@pytest.mark.parametrize("h,w", [(8, 8), (9, 11), (17, 32), (40, 33), (24, 97)])
def test_weight_boxes_of_a_window(cuda, engine_lib, oracle, h, w, radius, planes, final):
    """Single windows add a weight to every pixel: both slabs of every slot."""
    from bm3dcuda import synthetic as S
    tw = 2 * radius + 1
    noisy, clean = S.chroma_clip(tw, h, w, seed=w + h)
    win = noisy[:, :planes].transpose(1, 0, 2, 3).copy()
    ref = clean[:, :planes].astype(np.float32).transpose(1, 0, 2, 3).copy() if final else None
    kw = dict(sigma=[7.0, 4.0, 4.0], radius=radius, block_step=3, bm_range=5, extractor_exp=6,
              chroma=planes == 3)
    got = graph_run(win, ref, **kw)
    want = oracle.port_bm3d(win, ref, return_acc=True, **kw)
    np.testing.assert_array_equal(got, want)
