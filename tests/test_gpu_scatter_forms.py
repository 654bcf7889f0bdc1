"""The scatter by reductions of the load/store pipe, which takes every layout that
the boxes cannot: row strides that are no multiple of 4, buffers off a 16-byte
boundary, raw stacks whose planes do not line up, accumulators of more than 2^20
frames. Pre-rounded sums, so equality is bit for bit. Also the aggregations that
go pixel by pixel there."""
import ctypes

import numpy as np
import pytest

from test_gpu_batch import params

pytestmark = pytest.mark.gpu


def window_run(L, window, ref, stride, offset, *, sigma, block_step, bm_range, radius,
               extractor_exp, chroma, tx=(0, 0)):
    """One window whose buffers have `stride` floats a row and start `offset` floats
    after an aligned address: [planes][2r+1][2][H][W], and the words of the
    accumulators outside the planes."""
    import torch
    from bm3dcuda import _lib
    npl, tw, h, w = window.shape
    final = ref is not None
    halves = [ref, window] if final else [window]
    host = np.zeros((len(halves), npl, tw, h, stride), np.float32)
    for i, half in enumerate(halves):
        host[i, ..., :w] = half
    d_src = torch.zeros(host.size + offset, device="cuda")
    d_src[offset:] = torch.from_numpy(host.reshape(-1)).cuda()
    n = npl * tw * 2 * h * stride
    d_res = torch.full((offset + n + 64,), 3.0, device="cuda")
    s = [L.bm3d_b200_scale_sigma(v, int(final)) for v in sigma]
    handle = ctypes.c_void_p()
    _lib.check(L.bm3d_b200_graph_create_rtc(
        ctypes.byref(handle), d_res.data_ptr() + 4 * offset, d_src.data_ptr() + 4 * offset, None, w,
        h, stride, s[0], block_step, bm_range, radius, 2, 4, int(chroma), s[1], s[2], int(final),
        float(2 ** extractor_exp), 0, *tx))
    try:
        _lib.check(L.bm3d_b200_graph_launch_device(handle, None))
        torch.cuda.synchronize()
    finally:
        L.bm3d_b200_graph_destroy(handle)
    res = d_res.cpu().numpy()
    acc = res[offset:offset + n].reshape(npl, tw, 2, h, stride)
    return acc[..., :w], np.concatenate([res[:offset] - 3, res[offset + n:] - 3,
                                         acc[..., w:].reshape(-1)])


@pytest.mark.parametrize("tx", [(0, 0), (2, 1)])
@pytest.mark.parametrize("final", [False, True])
@pytest.mark.parametrize("radius,planes", [(0, 1), (1, 1), (1, 3)])
@pytest.mark.parametrize("h,w,pad,offset", [(8, 8, 1, 0), (17, 32, 0, 1), (40, 33, 0, 0),
                                            (24, 96, 2, 3), (9, 12, 0, 2)])
def test_window_layouts(cuda, engine_lib, oracle, h, w, pad, offset, radius, planes, final, tx):
    from bm3dcuda import synthetic as S
    noisy, clean = S.chroma_clip(2 * radius + 1, h, w, seed=w + h)
    win = noisy[:, :planes].transpose(1, 0, 2, 3).copy()
    ref = clean[:, :planes].astype(np.float32).transpose(1, 0, 2, 3).copy() if final else None
    kw = dict(sigma=[7.0, 4.0, 4.0], radius=radius, block_step=3, bm_range=5, extractor_exp=6,
              chroma=planes == 3)
    got, outside = window_run(engine_lib, win, ref, w + pad, offset, tx=tx, **kw)
    want = oracle.port_bm3d(win, ref, return_acc=True, transform_2d=tx[0], transform_1d=tx[1], **kw)
    np.testing.assert_array_equal(got, want)
    assert not outside.any()


@pytest.mark.parametrize("final", [False, True])
@pytest.mark.parametrize("h,w", [(8, 8), (9, 11), (17, 32), (40, 33), (31, 64), (24, 97)])
def test_spatial_clip_against_the_oracle(cuda, engine_lib, oracle, h, w, final):
    """Radius 0: the IEEE quotient of the oracle's accumulators."""
    from bm3dcuda import BM3Dv2, Clip
    from bm3dcuda import synthetic as S
    noisy, clean = S.texture_clip(3, h, w, seed=w + h)
    kw = dict(sigma=7.0, radius=0, block_step=3, bm_range=5, extractor_exp=6)
    got = BM3Dv2(Clip.from_array(noisy), ref=Clip.from_array(clean) if final else None,
                 **kw).to_array()
    for n in range(3):
        acc = oracle.port_bm3d(noisy[n][None, None], clean[n][None, None].astype(np.float32)
                               if final else None, return_acc=True, **kw)[0, 0]
        np.testing.assert_array_equal(got[n], (acc[0] / acc[1]).astype(np.float32))


@pytest.mark.parametrize("final", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_raw_planes_that_do_not_line_up(cuda, engine_lib, precision, final):
    """4:2:0 of an odd height: no plane's pairs line up with the others', so the raw
    stacks go without boxes. Each plane equals the same plane as a clip of its own."""
    import torch
    from bm3dcuda import _lib
    from bm3dcuda import synthetic as S
    L, w, h, n, stride = engine_lib, 70, 37, 3, 96
    p = params(L, 1, 5, 6.0)
    for i in range(3):
        p.sigma[i], p.block_step[i], p.bm_range[i] = 6.0, 5, 4

    def run(width, height, planes, ss, src, ref):
        c = ctypes.c_void_p()
        _lib.check(L.bm3d_b200_clip_create(ctypes.byref(c), width, height, planes, ss, ss, n,
                                           ctypes.byref(p), 0))
        try:
            _lib.check(L.bm3d_b200_clip_set_precision(c, precision))
            dst = torch.zeros((n, L.bm3d_b200_clip_raw_frame_floats(c)), device="cuda")
            _lib.check(L.bm3d_b200_clip_run(c, src.data_ptr(), ref.data_ptr() if final else None,
                                            dst.data_ptr(), _lib.DST_RAW, None))
            torch.cuda.synchronize()
            return dst
        finally:
            L.bm3d_b200_clip_destroy(c)

    sizes = [(w, h), (w // 2, h // 2), (w // 2, h // 2)]
    sources = []
    for i, (pw, ph) in enumerate(sizes):
        pair = []
        for half in S.texture_clip(n, ph, pw, seed=40 + i):
            host = np.zeros((n, ph, stride), np.float32)
            host[:, :, :pw] = half
            pair.append(torch.from_numpy(host).cuda())
        sources.append(pair)
    whole = [torch.cat([s[k].reshape(n, -1) for s in sources], 1).contiguous() for k in (0, 1)]
    got = run(w, h, 3, 1, whole[0], whole[1])
    at = 0
    for (pw, ph), pair in zip(sizes, sources):
        own = (pw + 31) // 32 * 32
        alone = run(pw, ph, 1, 0, *[s[:, :, :own].contiguous() for s in pair])
        rows = 2 * 3 * ph
        part = got[:, at:at + rows * stride].reshape(n, rows, stride)
        assert torch.equal(part[..., :pw], alone.reshape(n, rows, own)[..., :pw])
        assert not part[..., pw:].any()
        at += rows * stride


def test_batch_of_more_frames_than_boxes_count(cuda, engine_lib):
    """2^20 frames of 8 x 8: the batch kernels without boxes, beside a small clip."""
    import torch
    from bm3dcuda import _lib
    from bm3dcuda import synthetic as S
    L = engine_lib

    def run(clips):
        b = ctypes.c_void_p()
        _lib.check(L.bm3d_b200_batch_create(ctypes.byref(b), 0))
        try:
            outs = []
            for src, w, radius in clips:
                dst = torch.zeros_like(src)
                p = params(L, radius, 4, 6.0)
                _lib.check(L.bm3d_b200_batch_add(b, w, src.shape[1], src.shape[0],
                                                 ctypes.byref(p), src.data_ptr(), dst.data_ptr(),
                                                 None))
                outs.append(dst)
            _lib.check(L.bm3d_b200_batch_run(b, None))
            torch.cuda.synchronize()
            return outs
        finally:
            L.bm3d_b200_batch_destroy(b)

    def frames(n, h, w, seed):
        host = np.zeros((n, h, (w + 31) // 32 * 32), np.float32)
        host[:, :, :w] = S.texture_clip(n, h, w, seed=seed)[0]
        return torch.from_numpy(host).cuda()

    eight, other = frames(8, 8, 8, 1), frames(3, 45, 70, 2)
    want = run([(eight, 8, 0), (other, 70, 1)])
    many = eight.repeat(1 << 17, 1, 1)
    got = run([(many, 8, 0), (other, 70, 1)])
    assert torch.equal(got[0][..., :8].reshape(-1, 8, 8, 8),
                       want[0][..., :8].expand(1 << 17, 8, 8, 8))
    assert torch.equal(got[1][..., :70], want[1][..., :70])


@pytest.mark.parametrize("raw_stride,offset,dst_stride", [
    (16, 0, 16), (13, 0, 16), (15, 0, 16), (16, 1, 16), (16, 0, 17)])
@pytest.mark.parametrize("radius", [1, 3])
def test_vaggregate_layouts(cuda, engine_lib, radius, raw_stride, offset, dst_stride):
    """Single pixels (narrow rows), at every stride and offset."""
    import torch
    from bm3dcuda import _lib
    h, w, tw = 11, 13, 2 * radius + 1
    rng = np.random.default_rng(radius)
    raws = rng.uniform(0.5, 2.0, (tw, tw, 2, h, w)).astype(np.float32)
    keep, ptrs = [], (ctypes.c_void_p * tw)()
    for i in range(tw):
        host = np.full((tw, 2, h, raw_stride), np.nan, np.float32)
        host[..., :w] = raws[i]
        buf = torch.zeros(host.size + offset, device="cuda")
        buf[offset:] = torch.from_numpy(host.reshape(-1)).cuda()
        keep.append(buf)
        ptrs[i] = buf.data_ptr() + 4 * offset
    dst = torch.full((h, dst_stride), 5.0, device="cuda")
    n = radius  # no frame is clamped in a clip of 2r + 1
    _lib.check(engine_lib.bm3d_b200_vaggregate(dst.data_ptr(), dst_stride, ptrs, raw_stride, w, h,
                                               radius, n, tw, None))
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    sv, sw = np.zeros((h, w), np.float32), np.zeros((h, w), np.float32)
    for i in range(tw):
        sv += raws[i, tw - 1 - i, 0]
        sw += raws[i, tw - 1 - i, 1]
    np.testing.assert_array_equal(got[:, :w], sv / sw)
    assert (got[:, w:] == 5.0).all()


@pytest.mark.parametrize("w,stride,offset", [(128, 128, 0), (129, 132, 0), (131, 132, 0),
                                             (132, 132, 0), (515, 516, 0), (640, 640, 0),
                                             (640, 640, 1), (639, 639, 0)])
@pytest.mark.parametrize("radius", [0, 2, 3])
def test_vaggregate_widths(cuda, engine_lib, radius, w, stride, offset):
    """Rows of one block and more: quads from 129 columns on, with every remainder."""
    import torch
    from bm3dcuda import _lib
    h, tw = 5, 2 * radius + 1
    rng = np.random.default_rng(w)
    raws = rng.uniform(0.5, 2.0, (tw, tw, 2, h, stride)).astype(np.float32)
    keep, ptrs = [], (ctypes.c_void_p * tw)()
    for i in range(tw):
        buf = torch.zeros(raws[i].size + offset, device="cuda")
        buf[offset:] = torch.from_numpy(raws[i].reshape(-1)).cuda()
        keep.append(buf)
        ptrs[i] = buf.data_ptr() + 4 * offset
    dst = torch.full((h, stride), 5.0, device="cuda")
    _lib.check(engine_lib.bm3d_b200_vaggregate(dst.data_ptr(), stride, ptrs, stride, w, h, radius,
                                               radius, tw, None))
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    sv, sw = np.zeros((h, w), np.float32), np.zeros((h, w), np.float32)
    for i in range(tw):
        sv += raws[i, tw - 1 - i, 0, :, :w]
        sw += raws[i, tw - 1 - i, 1, :, :w]
    np.testing.assert_array_equal(got[:, :w], sv / sw)
    assert (got[:, w:] == 5.0).all()
