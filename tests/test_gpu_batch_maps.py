"""Batches prepared one after another in one process, whose tensor maps take each
other's places in device memory: every clip equals the clip run alone."""
import ctypes

import numpy as np
import pytest

from test_gpu_batch import clip_alone, params

pytestmark = pytest.mark.gpu

BATCHES = [  # width, height, frames, radius, block_step, sigma
    [(64, 48, 4, 0, 8, 6.0), (200, 120, 2, 1, 8, 9.0), (40, 40, 3, 1, 4, 5.0)],
    [(33, 57, 5, 1, 6, 6.0), (64, 48, 2, 0, 8, 6.0), (160, 8, 3, 2, 8, 4.0)],
    [(8, 8, 1, 0, 8, 7.0)],
    [(97, 31, 3, 2, 5, 6.0), (64, 200, 2, 0, 3, 9.0), (128, 128, 2, 1, 8, 3.0)],
]


class Batch:
    def __init__(self, L):
        from bm3dcuda import _lib
        self.L, self.check = L, _lib.check
        self.h = ctypes.c_void_p()
        self.clips = []
        self.check(L.bm3d_b200_batch_create(ctypes.byref(self.h), 0))

    def add(self, spec, seed, **search):
        import torch
        from bm3dcuda import synthetic as S
        w, h, n, r, bs, sigma = spec
        noisy, _ = S.texture_clip(n, h, w, seed=seed)
        host = np.zeros((n, h, (w + 31) // 32 * 32), np.float32)
        host[:, :, :w] = noisy
        src = torch.from_numpy(host).cuda()
        dst = torch.zeros_like(src)
        p = params(self.L, r, bs, sigma)
        for key, value in search.items():
            getattr(p, key)[0] = value
        idx = ctypes.c_int()
        self.check(self.L.bm3d_b200_batch_add(self.h, w, h, n, ctypes.byref(p), src.data_ptr(),
                                              dst.data_ptr(), ctypes.byref(idx)))
        self.clips.append((src, dst, w, clip_alone(self.L, torch, src, w, h, n, p)))

    def run(self):
        import torch
        for _, dst, _, _ in self.clips:
            dst.zero_()
        torch.cuda.synchronize()
        self.check(self.L.bm3d_b200_batch_run(self.h, None))
        torch.cuda.synchronize()
        for i, (_, dst, w, want) in enumerate(self.clips):
            np.testing.assert_array_equal(dst.cpu().numpy()[..., :w], want[..., :w], str(i))

    def close(self):
        self.L.bm3d_b200_batch_destroy(self.h)


def test_batches_in_turn(cuda, engine_lib):
    for rep in range(2):
        for k, specs in enumerate(BATCHES):
            b = Batch(engine_lib)
            try:
                for i, spec in enumerate(specs):
                    b.add(spec, seed=10 * k + i + rep)
                    b.run()  # prepared again with each clip
            finally:
                b.close()


def test_autotune_near_the_largest_tile(cuda, engine_lib):
    """One-warp CTAs with strips of 10 come within 100 bytes of the limit."""
    b = Batch(engine_lib)
    try:
        b.add((72, 56, 2, 0, 4, 6.0), seed=3, bm_range=100)
        b.check(engine_lib.bm3d_b200_batch_autotune(b.h, None))
        b.run()
    finally:
        b.close()
