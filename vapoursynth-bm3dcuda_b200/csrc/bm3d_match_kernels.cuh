// Block matching for BM3D / V-BM3D on sm_100a.
//
// Computes, for every reference block of every temporal window in a batch,
// the reference's 8-entry match list: exhaustive SSD search over the
// (2*bm_range+1)^2 window in the centre frame, then (radius > 0) the
// predictive search over ps_num windows of (2*ps_range+1)^2 per neighbour
// frame, then the centre-block insertion (source/kernel.cu:389-647,
// cpu_source/source.cpp:143-391, 787-844).
//
// Work layout
//   * one thread owns one reference block and scans all of its candidates in
//     the reference's scan order, so the strict-< list insertion gives
//     exactly the reference's list (ties keep the earlier candidate);
//   * a warp owns 4 x 8 reference blocks, a CTA WX such warps side by side.
//     A launch of few blocks leaves the chip idle that way (640x360: 120 warps
//     on 148 SMs), so there 4 or 8 lanes share a block, each scanning every
//     4th or 8th row, and merge their lists by (distance, scan order): the same
//     list (match_lanes has the rule and what it measured);
//   * the search runs as 1 + 2r stages (centre frame, then frames c-1 .. c-r,
//     then c+1 .. c+r). Each stage stages the CTA's pixel region of its frame
//     into shared memory, then every thread scans its windows of that stage
//     strip by strip (ssd_strip: one pixel load feeds up to 8 candidates);
//   * shared-memory rows are skewed by (row / 8) mod 8 words, which makes the
//     32 threads of a warp hit 32 distinct banks when block_step is 8; for
//     other steps the row pitch is picked for the fewest conflicts.
//
// Bound: the FP32 pipe and the issue slots (143 pipe slots per distance; 1.50 ms
// of distances for 12 windows of 1920x1080, radius 2), then the insertions and
// the registers: a strip's chains run side by side only as far as registers
// allow. 12 such windows take 2.41 ms (62% of the pipe), 2.85 before: two-entry
// temporal lists, strip widths of their own for the temporal windows (9 of 9
// columns used instead of 9 of 10) and the spatial list parked in shared memory.
// Measured and not kept: 4 CTAs per SM at 128 registers (1.10x the time), both
// halves of a block's columns as separate strips to skip the second (1.13x),
// two lanes per block with half its columns each and twice the warps (1.13x),
// the 19 columns of a window as one strip (0.98x at radius 0, 1.06x at 2).
#pragma once

#include <cuda_runtime.h>

#include "bm3d_device.cuh"
#include "bm3d_internal.h"

namespace bm3d {

namespace {

// CTA of the kernels whose lanes share blocks: kSplitWx x kSplitWy warps.
constexpr int kSplitWx = 2, kSplitWy = 2;

// Bits k of a strip starting at column cx0 whose column cx0 + k (k < 32) lies
// in [left, right].
__device__ __forceinline__ unsigned column_mask(int cx0, int left, int right) {
    const int lo = max(left - cx0, 0), hi = right - cx0;
    if (lo > 31 || hi < 0) return 0;
    return (0xffffffffu << lo) & (0xffffffffu >> (31 - min(hi, 31)));
}

// a[k] of a strip's distances by the bits of k (k < K <= 16).
template <int K>
__device__ __forceinline__ float pick_tree(const float (&a)[K], int k) {
    float v[(K + 1) / 2];
#pragma unroll
    for (int i = 0; i < (K + 1) / 2; ++i)
        v[i] = (k & 1) && 2 * i + 1 < K ? a[2 * i + 1 < K ? 2 * i + 1 : 0] : a[2 * i];
    constexpr int N1 = (K + 1) / 2, N2 = (N1 + 1) / 2, N3 = (N2 + 1) / 2;
#pragma unroll
    for (int i = 0; i < N2; ++i)
        v[i] = (k & 2) && 2 * i + 1 < N1 ? v[2 * i + 1 < N1 ? 2 * i + 1 : 0] : v[2 * i];
#pragma unroll
    for (int i = 0; i < N3; ++i)
        v[i] = (k & 4) && 2 * i + 1 < N2 ? v[2 * i + 1 < N2 ? 2 * i + 1 : 0] : v[2 * i];
    return N3 > 1 && (k & 8) ? v[N3 > 1 ? 1 : 0] : v[0];
}

// Scan the rows first, first + S, ... of one search window of a reference
// block in scan order (rows, then columns), feeding every in-range candidate
// to a list: all 8 entries of `cl` (SMALL, n == 8), else the n first entries of
// `list`, of which SMALL keeps two.
//   wx: unclamped window origin column (centre - range), image coordinates
//   [left, right] x [.., bottom]: the clamped candidate range
//   (tx0, ty0): image coordinates of the tile's (0, 0)
template <int K, int M, int S, bool SMALL>
__device__ __forceinline__ void scan_window(List8 &list, ColumnList &cl, int n,
                                            const f32x2 (&refp)[4][8], const RefStats &rs,
                                            const float *tile, int pitch, int tx0, int ty0, int wx,
                                            int left, int right, int first, int bottom, int nsub,
                                            int z) {
    for (int row = first; row <= bottom; row += S) {
        int roff[8];
        const int ty = row - ty0;
#pragma unroll
        for (int r = 0; r < 8; ++r) roff[r] = skewed(ty + r, wx - tx0, pitch);
        for (int s = 0; s < nsub; ++s) {
            float err[K];
            if (M == 0) {
                ssd_strip<K>(refp, tile, roff, err);
            } else {
                metric_strip<K, M>(refp, rs, tile, roff, err);
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) roff[r] += K;
            const int cx0 = wx + s * K;
            // cheap reject: once the list is full most strips improve nothing
            float best = err[0];
#pragma unroll
            for (int k = 1; k < K; ++k) best = fminf(best, err[k]);
            if (!(best < cl.thr)) continue;
            unsigned mask = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) mask |= (err[k] < cl.thr ? 1u : 0u) << k;
            mask &= column_mask(cx0, left, right);
            if (mask == 0) continue;
            // ascending k = the reference's scan order
            if (SMALL && n == 8) {
                List8 l;
                cl.load(l);
                while (mask) {
                    const int k = __ffs(mask) - 1;
                    mask &= mask - 1;
                    list_insert_n<8>(l, pick_tree(err, k), pack_pos(cx0 + k, row, z));
                }
                cl.store(l);
            } else {
                while (mask) {
                    const int k = __ffs(mask) - 1;
                    mask &= mask - 1;
                    list_insert_n<SMALL ? 2 : 8>(list, pick_tree(err, k), pack_pos(cx0 + k, row, z));
                }
                cl.thr = SMALL ? (n == 1 ? list.e[0] : list.e[1]) : pick(list.e, n - 1);
            }
        }
    }
}

// The same for a list of two entries: every candidate of a strip goes through
// the insertion, 8 operations each without a branch (one of them out of range
// enters as FLT_MAX, which is never kept).
template <int K, int S>
__device__ __forceinline__ void scan_window_pair(List8 &list, const f32x2 (&refp)[4][8],
                                                 const float *tile, int pitch, int tx0, int ty0,
                                                 int wx, int left, int right, int first,
                                                 int bottom, int nsub, int z) {
    for (int row = first; row <= bottom; row += S) {
        int roff[8];
        const int ty = row - ty0;
#pragma unroll
        for (int r = 0; r < 8; ++r) roff[r] = skewed(ty + r, wx - tx0, pitch);
        for (int s = 0; s < nsub; ++s) {
            float err[K];
            ssd_strip<K>(refp, tile, roff, err);
#pragma unroll
            for (int r = 0; r < 8; ++r) roff[r] += K;
            const int cx0 = wx + s * K;
            if (cx0 < left || cx0 + K - 1 > right) {
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (cx0 + k < left || cx0 + k > right) err[k] = FLT_MAX;
            }
            // pack_pos as a sum: cx0 may be negative, cx0 + k of a kept entry not
            const int pos = cx0 + (row << kCoordBits) + (z << (2 * kCoordBits));
#pragma unroll
            for (int k = 0; k < K; ++k) list_insert_n<2>(list, err[k], pos + k);
        }
    }
}

// The smaller of two list entries by (distance, scan order): positions packed
// with the window's index in place of the temporal slot compare, as unsigned
// numbers, in scan order (window, row, column).
__device__ __forceinline__ bool entry_before(float ea, int pa, float eb, int pb) {
    return ea < eb || (ea == eb && (unsigned)pa < (unsigned)pb);
}

// Merges the lists of the S lanes that share a reference block (each scanned
// every S-th row) into every one of them: the N smallest entries by (distance,
// scan order), which is the list that one lane scanning all rows would hold.
// Two sorted lists a, b: min(a[i], b[N-1-i]) are the N smallest of both, in
// bitonic order. Every lane of the warp calls it.
template <int N, int S>
__device__ __forceinline__ void merge_lanes(List8 &l) {
#pragma unroll
    for (int d = 1; d < S; d *= 2) {
        float oe[N];
        int op[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            oe[i] = __shfl_xor_sync(0xffffffffu, l.e[N - 1 - i], d);
            op[i] = __shfl_xor_sync(0xffffffffu, l.p[N - 1 - i], d);
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const bool take = entry_before(oe[i], op[i], l.e[i], l.p[i]);
            l.e[i] = take ? oe[i] : l.e[i];
            l.p[i] = take ? op[i] : l.p[i];
        }
#pragma unroll
        for (int h = N / 2; h > 0; h /= 2)
#pragma unroll
            for (int i = 0; i < N; ++i)
                if ((i & h) == 0) {
                    const bool swap = entry_before(l.e[i + h], l.p[i + h], l.e[i], l.p[i]);
                    const float e = l.e[i];
                    const int p = l.p[i];
                    l.e[i] = swap ? l.e[i + h] : e;
                    l.p[i] = swap ? l.p[i + h] : p;
                    l.e[i + h] = swap ? e : l.e[i + h];
                    l.p[i + h] = swap ? p : l.p[i + h];
                }
    }
}

// One CTA tile of reference blocks: tile (tile_x, tile_y) of window `win`.
// Every thread of the CTA must call it (it synchronises the CTA). S lanes
// share a reference block: a warp owns 4 x (8 / S) blocks. SMALL: the temporal
// stages keep at most two entries (ps_num <= 2, or no neighbour frames). K, KT:
// strip widths of the spatial and the temporal windows.
template <int K, int KT, int M, int S, bool SMALL>
__device__ __forceinline__ void match_tile(const MatchParams &p, int tile_x, int tile_y, int win,
                                           float *tile) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wcols = S == 1 ? (int)(blockDim.x >> 5) : kSplitWx;  // warps side by side
    const int nbx_cta = wcols * 4;
    const int nby_cta = S == 1 ? 8 : kSplitWy * (8 / S);
    const int wcol = S == 1 ? warp : warp % kSplitWx, wrow = S == 1 ? 0 : warp / kSplitWx;
    const int sub = lane % S, slot = lane / S;
    const int bx = tile_x * nbx_cta + wcol * 4 + (slot & 3);
    const int by = tile_y * nby_cta + wrow * (8 / S) + (slot >> 2);
    const bool active = bx < p.nbx && by < p.nby;

    const int x = min(bx * p.block_step, p.width - 8);
    const int y = min(by * p.block_step, p.height - 8);

    // CTA extent in reference-block origins
    const int bx_first = tile_x * nbx_cta;
    const int bx_last = min(bx_first + nbx_cta - 1, p.nbx - 1);
    const int by_first = tile_y * nby_cta;
    const int by_last = min(by_first + nby_cta - 1, p.nby - 1);
    const int xa = min(bx_first * p.block_step, p.width - 8);
    const int xb = min(bx_last * p.block_step, p.width - 8);
    const int ya = min(by_first * p.block_step, p.height - 8);
    const int yb = min(by_last * p.block_step, p.height - 8);

    const int r = p.radius;
    const int center = r;
    const float *const *frames = p.frames + (size_t)win * (2 * r + 1);

    f32x2 refp[4][8];
    RefStats rs{0.0f, 0.0f};
    // The block's list, in this thread's shared-memory column after the tile
    // (SMALL), else in `list` with the spatial positions, which seed the +1
    // direction, in the column.
    ColumnList cl{tile + (size_t)p.pitch * p.tile_rows + threadIdx.x, (int)blockDim.x, FLT_MAX};
    List8 list;
    constexpr int kLast = SMALL ? 2 : 8;
    int last[kLast], near[kLast];  // window centres; the spatial stage's, SMALL
    const int own = pack_pos(x, y, center);
    list_init(list, FLT_MAX, own);

    // stage 0: centre frame, exhaustive; stages 1..r: frames c-1..c-r;
    // stages r+1..2r: frames c+1..c+r (source/kernel.cu:503-613)
    for (int st = 0; st <= 2 * r; ++st) {
        const int t = st <= r ? st : st - r;
        const int z = st == 0 ? center : (st <= r ? center - t : center + t);
        const int m = p.bm_range + t * p.ps_range;  // reach of this stage's candidates
        const int tx0 = xa - m, ty0 = ya - m;
        const int twid = xb - xa + 2 * m + 8 + p.extra_cols;
        const int thei = yb - ya + 2 * m + 8;
        if (st > 0) __syncthreads();
        load_tile(tile, frames[z], p.width, p.height, p.stride, tx0, ty0, twid, thei, p.pitch);
        __syncthreads();
        if (st == 0) {
            // reference block as packed row pairs (rows 2q, 2q+1 of column c)
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    refp[q][c] = pack2(tile[skewed(y - ty0 + 2 * q, x - tx0 + c, p.pitch)],
                                       tile[skewed(y - ty0 + 2 * q + 1, x - tx0 + c, p.pitch)]);
            if (M != 0) rs = ref_stats<M>(refp);
        }
        if (S == 1 && !active) continue;
        if (st == r + 1) {
#pragma unroll
            for (int i = 0; i < kLast; ++i)
                last[i] = SMALL ? near[i] : __float_as_int(cl.col[i * cl.pitch]);
        }
        // A neighbour frame's list only ever gives its first ps_num entries
        // (the next frame's window centres, and the merge below), so only
        // those are kept: n entries instead of 8, fewer and cheaper insertions.
        const int n = st == 0 ? 8 : p.ps_num;
        // Lanes that share a block pack the window's index in place of the
        // temporal slot, so that positions compare in scan order (merge_lanes).
        List8 fl;
        list_init(fl, FLT_MAX, st == 0 ? (S == 1 ? own : pack_pos(x, y, 0))
                                       : (S == 1 ? pack_pos(0, 0, z) : 0));
        if (SMALL && st == 0) cl.store(fl);
        cl.thr = FLT_MAX;
        const int range = st == 0 ? p.bm_range : p.ps_range;
        const int nwin = st == 0 ? 1 : p.ps_num;
        const int nsub = st == 0 ? p.nsub_s : p.nsub_t;
        int rows = 0;  // rows of the windows before this one
        for (int i = 0; i < nwin; ++i) {
            int cx = x, cy = y;
            if (st > 0) {
                const int li = pick(last, i);
                // Window centres are earlier matches and lie within
                // bm_range + (t-1)*ps_range of the block; the clamp only bites
                // for lists polluted by non-finite distances.
                cx = min(max(pos_x(li), x - m + range), x + m - range);
                cy = min(max(pos_y(li), y - m + range), y + m - range);
            }
            const int left = max(cx - range, 0), right = min(cx + range, p.width - 8);
            const int top = max(cy - range, 0), bottom = min(cy + range, p.height - 8);
            // lane `sub` of the block takes every S-th row of the stage
            const int first = S == 1 ? top : top + (int)((unsigned)(sub - rows) % (unsigned)S);
            rows += bottom - top + 1;
            if (S > 1 && !active) continue;
            if (SMALL && M == 0 && n != 8)
                scan_window_pair<KT, S>(fl, refp, tile, p.pitch, tx0, ty0, cx - range, left,
                                        right, first, bottom, nsub, S == 1 ? z : i);
            else
                scan_window<K, M, S, SMALL>(fl, cl, n, refp, rs, tile, p.pitch, tx0, ty0,
                                            cx - range, left, right, first, bottom, nsub,
                                            S == 1 ? z : i);
        }
        if (st == 0) {
            if (SMALL) cl.load(fl);
            if (S > 1) {
                merge_lanes<8, S>(fl);
#pragma unroll
                for (int i = 0; i < 8; ++i) fl.p[i] = pack_pos(pos_x(fl.p[i]), pos_y(fl.p[i]), z);
                if (SMALL) cl.store(fl);
            }
            if (!SMALL) list = fl;
#pragma unroll
            for (int i = 0; i < kLast; ++i) last[i] = fl.p[i];
            if (SMALL) {
#pragma unroll
                for (int i = 0; i < kLast; ++i) near[i] = fl.p[i];
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) cl.col[i * cl.pitch] = __int_as_float(fl.p[i]);
            }
        } else {
            if (S > 1) {
                merge_lanes<kLast, S>(fl);
#pragma unroll
                for (int i = 0; i < kLast; ++i)
                    fl.p[i] = pack_pos(pos_x(fl.p[i]), pos_y(fl.p[i]), z);
            }
            // merge the frame's first ps_num entries (source/kernel.cu:589-608)
            if (SMALL) cl.load(list);
            for (int i = 0; i < p.ps_num; ++i) {
                const float e = SMALL ? (i == 0 ? fl.e[0] : fl.e[1]) : pick(fl.e, i);
                const int pos = SMALL ? (i == 0 ? fl.p[0] : fl.p[1]) : pick(fl.p, i);
                if (e < list.e[7]) list_insert_n<8>(list, e, pos);
            }
            if (SMALL) cl.store(list);
#pragma unroll
            for (int i = 0; i < kLast; ++i) last[i] = fl.p[i];
        }
    }

    if (!active || sub != 0) return;
    if (SMALL) cl.load(list);

    // ---- centre insertion (source/kernel.cu:616-647) ----------------------
    const int cpos = pack_pos(x, y, center);
    bool found = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) found |= list.p[i] == cpos;
    if (!found) {
#pragma unroll
        for (int i = 7; i > 0; --i) list.p[i] = list.p[i - 1];
        list.p[0] = cpos;
    }

    int4 *out = reinterpret_cast<int4 *>(p.matches + ((size_t)win * p.nbx * p.nby +
                                                      (size_t)by * p.nbx + bx) * 8);
    out[0] = make_int4(list.p[0], list.p[1], list.p[2], list.p[3]);
    out[1] = make_int4(list.p[4], list.p[5], list.p[6], list.p[7]);
}

// CTAS: resident CTAs per SM that the registers aim at. Two (up to 255 registers a
// thread) run a warp about 20% faster than three (168), which pays until a
// launch has CTAs enough to fill three places for several waves; match_ctas has
// the rule.
template <int K, int KT, int M, int S, bool SMALL, int CTAS>
__global__ void __launch_bounds__(128, CTAS) match_kernel(MatchParams p) {
    extern __shared__ float tile[];
    match_tile<K, KT, M, S, SMALL>(p, blockIdx.x, blockIdx.y, p.win0 + blockIdx.z, tile);
}

template <int K, int KT, int M, int S, bool SMALL, int CTAS = 2>
cudaError_t launch_match_t(const MatchParams &p, dim3 grid, dim3 block, size_t smem,
                           cudaStream_t stream) {
    auto fn = match_kernel<K, KT, M, S, SMALL, CTAS>;
    // The dynamic shared-memory opt-in is per device; raise it only when a
    // launch needs more than this device was configured for, so that launches
    // recorded into CUDA graphs do not repeat the attribute call.
    static int configured[64] = {0};
    cudaError_t e = raise_smem_limit(configured, (const void *)fn, smem);
    if (e != cudaSuccess) return e;
    fn<<<grid, block, smem, stream>>>(p);
    return cudaGetLastError();
}

template <int K, int KT, bool SMALL>
cudaError_t launch_match_lanes(const MatchParams &p, const MatchGeometry &g, int nwin, int lanes,
                               cudaStream_t stream) {
    if (lanes == 1) {
        if (g.smem > kMatchSmemMax) return cudaErrorInvalidValue;
        const dim3 grid((p.nbx + 4 * g.wx - 1) / (4 * g.wx), (p.nby + 7) / 8, nwin);
        if constexpr (SMALL)
            if (match_ctas(g, nwin) == 3)
                return launch_match_t<K, KT, 0, 1, true, 3>(p, grid, 32 * g.wx, g.smem, stream);
        return launch_match_t<K, KT, 0, 1, SMALL>(p, grid, 32 * g.wx, g.smem, stream);
    }
    const auto &sp = g.split[lanes == 4 ? 0 : 1];
    if (sp.smem > kMatchSmemMax) return cudaErrorInvalidValue;
    MatchParams q = p;
    q.pitch = sp.pitch;
    q.tile_rows = sp.tile_rows;
    const int rows = 8 / lanes * kSplitWy;  // block rows of a CTA
    const dim3 grid((p.nbx + 4 * kSplitWx - 1) / (4 * kSplitWx), (p.nby + rows - 1) / rows, nwin);
    const dim3 block(32 * kSplitWx * kSplitWy);
    return lanes == 4 ? launch_match_t<K, KT, 0, 4, SMALL>(q, grid, block, sp.smem, stream)
                      : launch_match_t<K, KT, 0, 8, SMALL>(q, grid, block, sp.smem, stream);
}

}  // namespace
}  // namespace bm3d
