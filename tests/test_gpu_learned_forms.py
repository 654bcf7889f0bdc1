"""The learned matcher's forms (general lists; short lists from 1000 warps of 4 x 8
blocks on, with cells ranked row by row or across row ends): lists and fallback flags
are the C oracle's."""
import numpy as np
import pytest

from oracle import proposer_ref as P
from test_gpu_learned import _frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bs,radius,ps_num,ps_range,cells", [
    (203, 181, 1, 1, 2, 4, (2, 2)),    # 1078 warps: short lists, row by row
    (203, 181, 1, 1, 1, 1, (4, 3)),    # narrow windows
    (203, 181, 1, 1, 3, 4, (2, 2)),    # ps_num 3: general
    (203, 181, 1, 0, 2, 4, (8, 1)),    # radius 0: general
    (903, 906, 5, 1, 2, 4, (2, 2)),    # 45 x 23 warps: across row ends, 5 columns
    (903, 906, 5, 1, 2, 6, (3, 4)),    # 7 columns
    (903, 906, 5, 1, 1, 5, (1, 8)),    # 6 columns
    (903, 906, 5, 1, 2, 3, (2, 2)),    # 4 columns: row by row
    (61, 47, 5, 2, 2, 5, (2, 2)),      # a small launch: general
])
def test_lists(cuda, oracle, engine_lib, w, h, bs, radius, ps_num, ps_range, cells):
    from bm3dcuda import synthetic as S
    from bm3dcuda.learned import Proposer, learned_match
    rng = np.random.default_rng(ps_range)
    prop = Proposer()
    try:
        prop.set_params((P.init_params(8.0) + rng.normal(0, 0.02, P.NPARAMS)).astype(np.float32))
        win, _ = S.texture_clip(2 * radius + 1, h, w, seed=ps_range)
        d_f = _frames(cuda, win)
        prop.calibrate(d_f, w, h)
        emb = prop.embed(d_f, w, h)
        kw = dict(block_step=bs, bm_range=5, radius=radius, ps_num=ps_num, ps_range=ps_range,
                  cells_spatial=cells[0], cells_temporal=cells[1], fallback_ssd=0.04)
        got, gfell = learned_match(prop, win, embeddings=emb, **kw)
        want, wfell = oracle.port_learned_match(win, emb.cpu().numpy(), **kw)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(gfell, wfell)
    finally:
        prop.close()
