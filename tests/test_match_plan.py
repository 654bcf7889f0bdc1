"""Every search that is accepted has a launch that fits on chip: the range check
keeps to one-warp CTAs of at most 220 KB, and the form picked for a launch stays
within a CTA's 227 KB. No device is needed."""
import ctypes

import pytest

OK, UNSUPPORTED = 0, 3


def range_bytes(block_step, bm_range, radius, ps_range, warps=1, strip=None):
    """Shared memory of the CTA (one warp for single launches) by which a range is
    accepted or refused."""
    ws, wt, reach = 2 * bm_range + 1, 2 * ps_range + 1, bm_range + radius * ps_range

    def over(w, k):
        return -(-w // k) * k - w

    def cost(k):
        total = 0.0
        for w, n in ((ws, ws * ws), (wt, 4.0 * radius * wt * wt)):
            total += n * (w + over(w, k)) / w * (143.0 + 8.0 * (k + 7) / k)
        return total

    k = strip or min(range(8, 13), key=cost)
    extra = max(over(ws, k), over(wt, k) if radius else 0)
    pitch = (4 * warps - 1) * block_step + 2 * reach + 16 + extra
    return 4 * pitch * (7 * block_step + 2 * reach + 8) + 1024 * warps


@pytest.mark.parametrize("block_step", range(1, 9))
def test_accepted_searches_fit(engine_lib, block_step):
    lanes, shared, limit = ctypes.c_int(), ctypes.c_longlong(), ctypes.c_longlong()
    forms, refused = set(), 0
    bm_ranges = [*range(1, 8), *range(8, 80, 6), *range(80, 116)]
    for radius, ps_num, ps_range in [(0, 2, 4), (1, 2, 1), (1, 2, 6), (1, 3, 6), (2, 1, 4),
                                     (2, 2, 6), (3, 8, 9), (7, 2, 3)]:
        for bm_range in bm_ranges:
            for w, h, windows in [(8, 8, 1), (300, 169, 1), (640, 360, 1), (960, 540, 2),
                                  (1920, 1080, 30)]:
                rc = engine_lib.bm3d_b200_selftest_match_plan(
                    w, h, block_step, bm_range, radius, ps_num, ps_range, windows,
                    ctypes.byref(lanes), ctypes.byref(shared), ctypes.byref(limit))
                case = (block_step, bm_range, radius, ps_num, ps_range, w, h, windows)
                if range_bytes(block_step, bm_range, radius, ps_range) > 220 * 1024:
                    assert rc == UNSUPPORTED, case
                    refused += 1
                    continue
                assert rc == OK, case
                assert limit.value == 227 * 1024
                assert shared.value <= limit.value, (case, lanes.value, shared.value)
                forms.add(lanes.value)
    assert {1, 8} <= forms and refused


@pytest.mark.parametrize("block_step", range(1, 9))
def test_accepted_batches_fit(engine_lib, block_step):
    shared, limit = ctypes.c_longlong(), ctypes.c_longlong()
    for radius, ps_num, ps_range in [(0, 2, 4), (1, 2, 1), (1, 2, 6), (1, 3, 6), (2, 2, 4),
                                     (2, 2, 6), (3, 8, 9)]:
        for bm_range in range(20, 116):
            for warps in (1, 2, 4):
                for strip in range(8, 13):
                    rc = engine_lib.bm3d_b200_selftest_batch_plan(
                        640, 360, block_step, bm_range, radius, ps_num, ps_range, warps, strip,
                        ctypes.byref(shared), ctypes.byref(limit))
                    case = (block_step, bm_range, radius, ps_num, ps_range, warps, strip)
                    need = range_bytes(block_step, bm_range, radius, ps_range, warps, strip)
                    assert rc == (UNSUPPORTED if need > 220 * 1024 else OK), case
                    if rc == OK:
                        assert shared.value <= limit.value == 227 * 1024, (case, shared.value)


def test_strips_suit_narrow_windows(engine_lib):
    """The run-time-compiled plugin's distances: no search computes its candidates
    2.25 times (strips of 8 over windows of 3 columns would compute 2.67 times)."""
    for bm_range in range(1, 41):
        for radius in range(4):
            for ps_num in range(1, 9):
                for ps_range in range(1, 11):
                    k = engine_lib.bm3d_b200_selftest_metric_strip(bm_range, radius, ps_num,
                                                                   ps_range)
                    windows = [(1, 2 * bm_range + 1), (2 * radius * ps_num, 2 * ps_range + 1)]
                    computed = sum(n * w * -(-w // k) * k for n, w in windows)
                    assert computed < 2.25 * sum(n * w * w for n, w in windows), (
                        bm_range, radius, ps_num, ps_range, k)


def test_small_windows_are_not_shared(engine_lib):
    """Several lanes per block scan a window of 25 candidates slower than one, once
    a launch has a few warps for every SM."""
    lanes, shared, limit = ctypes.c_int(), ctypes.c_longlong(), ctypes.c_longlong()
    for w, h, step, bm_range, want in [(640, 360, 8, 2, 8), (960, 540, 8, 2, 4),
                                       (1280, 720, 8, 2, 1), (1280, 720, 8, 1, 1),
                                       (700, 400, 4, 2, 1), (1280, 720, 8, 9, 4)]:
        assert engine_lib.bm3d_b200_selftest_match_plan(
            w, h, step, bm_range, 0, 2, 4, 1, ctypes.byref(lanes), ctypes.byref(shared),
            ctypes.byref(limit)) == OK
        assert lanes.value == want, (w, h, step, bm_range, lanes.value)
