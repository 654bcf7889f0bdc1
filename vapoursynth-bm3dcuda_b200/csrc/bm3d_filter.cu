// Collaborative filtering (3-D transform, shrinkage, inverse) and weighted
// scatter for BM3D / V-BM3D on sm_100a, plus the per-pixel aggregation
// kernels (spatial division and VAggregate).
//
// One group (8 matched 8x8 patches of one reference block) is handled by 8
// threads. The 3-D transform runs in the reference's pass order - rows, then
// columns, then across the group - with the reference's 1-D factorisation
// (source/kernel.cu:256-363, cpu_source/source.cpp:596-670):
//
//   thread = column c, holds (patch, row):  vertical pass in registers
//   exchange through shared memory -> thread = row r: horizontal pass
//   exchange back -> thread = column c: group pass, shrinkage
//   inverse: vertical pass, exchange, horizontal pass and group pass
//            (thread = row), exchange back -> thread = column: scatter
//
// The shrinkage runs with the coefficient layout the reference uses (lane =
// column frequency, in-register index = group frequency * 8 + row frequency),
// so the Wiener weight's sum of squares is accumulated in the same order.
//
// Scatter, in three forms (launch_filter_form chooses):
//   boxes with corner weights (clips and batches): each patch goes as one TMA
//     reduction of a 12 x 8 box, which takes the 64 additions per thread off the
//     load/store pipe; the weight of a patch is added once, at its top-left pixel,
//     and the aggregation kernel sums each pixel's 8x8 neighbourhood of corners,
//     which equals the per-pixel weight sum (exactly so with pre-rounding);
//   boxes with a weight for every pixel (single windows, raw stacks, streams): a
//     second box per patch;
//   the load/store pipe: the 8 threads of a group add 8 contiguous pixels of a
//     patch row per instruction. For layouts that boxes cannot address (scatter_map:
//     row strides that are no multiple of 4, bases off a 16-byte boundary, raw planes
//     that do not line up, 2^20 accumulators and more) and for the hard-threshold
//     windows where it is faster (crowded_windows, weight_boxes_cost_a_wave).
//
// Groups are scheduled block-row-major across windows: CTAs running together
// work on the same rows of every window, so the gathered patches and the
// accumulator rows they hit stay resident in L2.
//
// Bound: the load/store pipe and the issue slots, then the L2's additions. Of
// the 30-window 1920x1080 radius-2 launches (hard threshold / Wiener): gathers
// alone take 0.30 / 0.60 ms, the additions alone 0.57 (as reductions of the
// load/store pipe) or 0.70 (TMA, in parallel). The launches take 0.99 / 1.73 ms
// (1.25 / 2.41 with the load/store scatter, single-word exchanges and an unrolled
// prefetch, by which the Wiener kernel had 48 KB of code and its warps waited 1.4
// cycles an issue for instructions, 0.44 now).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "bm3d_device.cuh"
#include "bm3d_internal.h"

namespace bm3d {

namespace {

constexpr int kXchgGroup = 528;    // words per group in the exchange buffer (8*64 + 16)
constexpr int kXchgGroupTc = 584;  // the split-BF16 form's: rows of 9 words (8*72 + 8)
constexpr int kCoefGroup = 520;    // words per group of parked Wiener coefficients
constexpr int kGroupsPerCta = 16;
// Scatter boxes of the TMA form: a patch's 8 rows of 12 words (the 8 pixels and
// the words that complete their 16-byte quads), 128-byte aligned.
constexpr int kBoxWords = 96, kBoxGroup = 8 * kBoxWords;
// Scatter forms: reductions of the load/store pipe; TMA boxes with corner
// weights; TMA boxes with a weight for every pixel (raw stacks, single windows).
enum Scatter { kScatterLsu = 0, kScatterBoxes = 1, kScatterWeights = 2 };

// Layout exchanges between the 8 threads of a group (thread = column or row of
// the group's patches), through shared memory. Every access moves 128 bytes per
// wavefront without bank conflicts; what the two layouts choose is which values
// arrive in adjacent registers, since the pass that follows works on packed
// pairs and re-pairing 64 values costs moves:
//   pairs of patches (p, p + 1), before a pass within the patches
//     (col_to_row): the pair is one 8-byte unit; unit (row i, column c) of patch
//     pair q at word q*128 + i*16 + 2c with its 16-byte quads permuted by i / 2:
//     32 8-byte stores, 16 16-byte loads
//   pairs of rows (r, r + 1), before a pass across the group (row_to_col): unit
//     (r / 2, c) of patch p at word p*64 + (r / 2)*16 + 2 (c ^ f), f from r and the
//     group: 64 single stores, 32 8-byte loads
// against 64 and 64 single-word accesses each way.

// c ^ this is column c's unit in row pair r2 of group g (pairs-of-rows layout):
// with the groups 16 words apart, the 32 lanes of a store (8 rows x 4 groups)
// and the 16 of a load's half warp (8 columns x 2 groups) hit distinct banks.
__device__ __forceinline__ int row_pair_swizzle(int r2, int g) {
    return (r2 >> 1) | (g & 2) | ((r2 & 1) << 2);
}

// thread = column `me`, v[p][row] -> thread = row `me`, v[p][col]
__device__ __forceinline__ void col_to_row(float (&v)[8][8], float *S, int me) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float *unit = S + i * 16 + (((me >> 1) ^ (i >> 1)) << 2) + ((me & 1) << 1);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            *reinterpret_cast<float2 *>(unit + q * 128) = make_float2(v[2 * q][i], v[2 * q + 1][i]);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
        const float *quad = S + me * 16 + (((c >> 1) ^ (me >> 1)) << 2);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 t = *reinterpret_cast<const float4 *>(quad + q * 128);
            v[2 * q][c] = t.x;
            v[2 * q + 1][c] = t.y;
            v[2 * q][c + 1] = t.z;
            v[2 * q + 1][c + 1] = t.w;
        }
    }
    __syncwarp();
}

// thread = row `me`: v[p][col] into the pairs-of-rows layout of group g
__device__ __forceinline__ void put_row(float *S, const float (&v)[8][8], int me, int g) {
    const int f = row_pair_swizzle(me >> 1, g);
    float *row = S + (me >> 1) * 16 + (me & 1);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float *unit = row + ((c ^ f) << 1);
#pragma unroll
        for (int p = 0; p < 8; ++p) unit[p * 64] = v[p][c];
    }
}

// word of (row r, column c) of patch 0 in the pairs-of-rows layout of group g
__device__ __forceinline__ int row_pair_word(int r, int c, int g) {
    return (r >> 1) * 16 + ((c ^ row_pair_swizzle(r >> 1, g)) << 1) + (r & 1);
}

// thread = row `me`, v[p][col] -> thread = column `me`, v[p][row]
__device__ __forceinline__ void row_to_col(float (&v)[8][8], float *S, int me, int g) {
    put_row(S, v, me, g);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 8; r += 2) {
        const float *unit = S + row_pair_word(r, me, g);
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const float2 t = *reinterpret_cast<const float2 *>(unit + p * 64);
            v[p][r] = t.x;
            v[p][r + 1] = t.y;
        }
    }
    __syncwarp();
}

// The 8-point passes run two lines per packed FP32x2 instruction stream
// (lines of patches p and p + 1 within the patches; lines of elements i and
// i + 1 across the group); the results are those of the scalar codelets.
__device__ __forceinline__ void pass_in_patch(float (&v)[8][8], bool forward) {
#pragma unroll
    for (int p = 0; p < 8; p += 2) {
        f32x2 t[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = pack2(v[p][k], v[p + 1][k]);
        if (forward) dct8_fwd2(t); else dct8_inv2(t);
#pragma unroll
        for (int k = 0; k < 8; ++k) unpack2(t[k], v[p][k], v[p + 1][k]);
    }
}

__device__ __forceinline__ void pass_across_group(float (&v)[8][8], bool forward) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        f32x2 t[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) t[p] = pack2(v[p][i], v[p][i + 1]);
        if (forward) dct8_fwd2(t); else dct8_inv2(t);
#pragma unroll
        for (int p = 0; p < 8; ++p) unpack2(t[p], v[p][i], v[p][i + 1]);
    }
}

// The same passes with run-time transform kinds (the run-time-compiled
// plugin's transform_2d_s / transform_1d_s; kinds are uniform per launch).
__device__ __forceinline__ void pass_in_patch_var(float (&v)[8][8], bool forward, int kind) {
#pragma unroll
    for (int p = 0; p < 8; ++p) tx8(v[p], kind, forward);
}

__device__ __forceinline__ void pass_across_group_var(float (&v)[8][8], bool forward, int kind) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float t[8];
#pragma unroll
        for (int p = 0; p < 8; ++p) t[p] = v[p][i];
        tx8(t, kind, forward);
#pragma unroll
        for (int p = 0; p < 8; ++p) v[p][i] = t[p];
    }
}

__device__ __forceinline__ void forward3d_var(float (&v)[8][8], float *S, int me, int g, int t2d,
                                              int t1d) {
    pass_in_patch_var(v, true, t2d);
    col_to_row(v, S, me);
    pass_in_patch_var(v, true, t2d);
    row_to_col(v, S, me, g);
    pass_across_group_var(v, true, t1d);
}

// Forward 3-D transform: in thread = column layout, out thread = column layout.
__device__ __forceinline__ void forward3d(float (&v)[8][8], float *S, int me, int g) {
    pass_in_patch(v, true);   // rows (vertical)
    col_to_row(v, S, me);
    pass_in_patch(v, true);   // columns (horizontal)
    row_to_col(v, S, me, g);
    pass_across_group(v, true);
}

// ---------------------------------------------------------------------------
// Split-BF16 tensor-core transform (precision 1).
//
// The reference's 8-point factorisation is the linear map
//   C[k][n] = 2 c_k cos(pi (2n + 1) k / 16),  c_0 = 1/sqrt(2), c_k = 1,
// and its inverse is C^T (C^T C = 16 I, fwd(inv(x)) = 16 x). Each pass of the
// 3-D transform multiplies the 64 lines of a group along one axis by C (or
// C^T): a [64 x 8] x [8 x 8] contraction, four m16n8k8 BF16 tensor-core tiles.
// Operands are split into three BF16 parts (x = xh + xm + xl, each part the
// rounding of what the previous ones leave) and the six products of order up
// to 2^-16 relative are accumulated in FP32, smallest first:
//   xl Dh + xm Dm + xh Dl + xm Dh + xh Dm + xh Dh,
// which keeps the product accurate to about FP32 rounding (2^-24). The group
// sits in the warp's exchange buffer as G[p*72 + r*9 + c]; the four groups of
// a warp are transformed by the whole warp, one m16n8k8 tile at a time.
// ---------------------------------------------------------------------------
struct SplitB {
    uint32_t h, m, l;  // B fragments (k = 2t, 2t+1; n = lane / 4) of the three parts
};

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// 2 cos(pi m / 16), m = 0 .. 8
__constant__ double kTwoCos[9] = {
    2.0, 1.9615705608064609, 1.8477590650225735,
    1.6629392246050905, 1.4142135623730951, 1.1111404660392046,
    0.7653668647301797, 0.39018064403225666, 0.0};

// B fragments of the forward (C) or inverse (C^T) map for this lane: the mma
// computes out[line][n] = sum_k in[line][k] * B[k][n], B[k][n] = D[n][k]. (From a
// table: four double-precision cosines per thread cost a tenth of the kernel.)
__device__ __forceinline__ SplitB dct_fragment(bool forward, int lane) {
    const int n = lane >> 2, t = lane & 3;
    __nv_bfloat16 h[2], m[2], l[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int k = 2 * t + j;
        const int fr = forward ? n : k, ps = forward ? k : n;  // frequency, position
        // the angle pi a / 16, folded into [0, pi / 2]
        const int a = ((2 * ps + 1) * fr) & 31, b = a > 16 ? 32 - a : a;
        double d = b > 8 ? -kTwoCos[16 - b] : kTwoCos[b];
        if (fr == 0) d = 1.41421356237309504880;
        h[j] = __double2bfloat16(d);
        const double r1 = d - (double)__bfloat162float(h[j]);
        m[j] = __double2bfloat16(r1);
        l[j] = __double2bfloat16(r1 - (double)__bfloat162float(m[j]));
    }
    return SplitB{pack_bf16(h[0], h[1]), pack_bf16(m[0], m[1]), pack_bf16(l[0], l[1])};
}

// Two values into three pairs of BF16 parts (x0 in the low halves): each part is
// the rounding of what the previous ones leave. Conversions two at a time; a
// part's value is its half word as the top of a float.
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float bf16_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }

__device__ __forceinline__ void split3(float x0, float x1, uint32_t &h, uint32_t &m, uint32_t &l) {
    h = cvt_bf16x2(x0, x1);
    const float r0 = __fsub_rn(x0, bf16_lo(h)), r1 = __fsub_rn(x1, bf16_hi(h));
    m = cvt_bf16x2(r0, r1);
    l = cvt_bf16x2(__fsub_rn(r0, bf16_lo(m)), __fsub_rn(r1, bf16_hi(m)));
}

__device__ __forceinline__ void mma_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b));
}

// word offset of element k of line l of a pass along `axis`
// (0: along rows r, 1: along columns c, 2: across the group p)
__device__ __forceinline__ int tc_addr(int axis, int l, int k) {
    return axis == 0 ? (l >> 3) * 72 + k * 9 + (l & 7)
                     : axis == 1 ? (l >> 3) * 72 + (l & 7) * 9 + k
                                 : k * 72 + (l >> 3) * 9 + (l & 7);
}

// One pass along `axis` for the warp's four groups (buffers kXchgGroupTc apart).
__device__ __forceinline__ void tc_pass(float *W, int axis, const SplitB &B, int lane) {
    const int gq = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int gi = 0; gi < 4; ++gi) {
        float *G = W + gi * kXchgGroupTc;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const int l0 = mt * 16 + gq, l1 = l0 + 8;
            const int o00 = tc_addr(axis, l0, 2 * t), o01 = tc_addr(axis, l0, 2 * t + 1);
            const int o10 = tc_addr(axis, l1, 2 * t), o11 = tc_addr(axis, l1, 2 * t + 1);
            uint32_t ah0, am0, al0, ah1, am1, al1;
            split3(G[o00], G[o01], ah0, am0, al0);
            split3(G[o10], G[o11], ah1, am1, al1);
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_k8(acc, al0, al1, B.h);
            mma_k8(acc, am0, am1, B.m);
            mma_k8(acc, ah0, ah1, B.l);
            mma_k8(acc, am0, am1, B.h);
            mma_k8(acc, ah0, ah1, B.m);
            mma_k8(acc, ah0, ah1, B.h);
            G[o00] = acc[0];
            G[o01] = acc[1];
            G[o10] = acc[2];
            G[o11] = acc[3];
        }
    }
}

// 3-D transform of the warp's groups on the tensor cores: in with thread =
// column `me` of group S (v[p][row]); out the same way, or (READ_BACK false)
// left in S as S[p*72 + r*9 + c]. W = the warp's first buffer.
template <bool READ_BACK = true>
__device__ __forceinline__ void tc_transform3d(float (&v)[8][8], float *S, float *W, int me,
                                               int lane, const SplitB &B) {
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int r = 0; r < 8; ++r) S[p * 72 + r * 9 + me] = v[p][r];
    __syncwarp();
    tc_pass(W, 0, B, lane);
    __syncwarp();
    tc_pass(W, 1, B, lane);
    __syncwarp();
    tc_pass(W, 2, B, lane);
    __syncwarp();
    if constexpr (READ_BACK) {
#pragma unroll
        for (int p = 0; p < 8; ++p)
#pragma unroll
            for (int r = 0; r < 8; ++r) v[p][r] = S[p * 72 + r * 9 + me];
        __syncwarp();
    }
}

// The position of patch `me`.
__device__ __forceinline__ int pick_pos(const int (&pos)[8], int me) {
    int q = pos[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) q = me == k ? pos[k] : q;
    return q;
}

__device__ __forceinline__ void load_group(float (&v)[8][8], const float *const *planes,
                                           const int (&pos)[8], int stride, int c) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const float *b = planes[pos_z(pos[p])] + (size_t)pos_y(pos[p]) * stride + pos_x(pos[p]) + c;
#pragma unroll
        for (int r = 0; r < 8; ++r) v[p][r] = __ldg(b + (size_t)r * stride);
    }
}

// The same pixels as load_group, copied asynchronously into C[(p*8 + r)*8 + c]
// (the thread's own slots of the parked-coefficient buffer): they land while
// the thread works on something else, and only this thread reads them. A rolled
// loop (patch p's position comes from lane p): the Wiener kernel's code is at
// the size where warps wait for instructions.
__device__ __forceinline__ void prefetch_group(float *C, const float *const *planes, int pos_me,
                                               int stride, int c) {
    unsigned d = (unsigned)__cvta_generic_to_shared(C + c);
#pragma unroll 1
    for (int p = 0; p < 8; ++p, d += 256u) {
        const int pos = __shfl_sync(0xffffffffu, pos_me, p, 8);
        const float *b = planes[pos_z(pos)] + (size_t)pos_y(pos) * stride + pos_x(pos) + c;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 32u * r),
                         "l"(b + (size_t)r * stride)
                         : "memory");
    }
}

// Shared-memory words of a warp: its four groups' exchange buffers, then their
// parked Wiener coefficients; the scatter boxes of the TMA form take their place.
template <bool FINAL, bool TC, int SC>
__host__ __device__ constexpr int warp_words() {
    constexpr int work = 4 * ((TC ? kXchgGroupTc : kXchgGroup) + (FINAL ? kCoefGroup : 0));
    constexpr int boxes = 4 * (SC == kScatterLsu       ? 0
                               : SC == kScatterWeights ? kBoxGroup + 4 * kBoxWords
                                                       : kBoxGroup);
    return ((work > boxes ? work : boxes) + 31) / 32 * 32;
}

template <bool FINAL, bool TC, int SC>
constexpr size_t filter_smem() {
    return (size_t)(kGroupsPerCta / 4) * warp_words<FINAL, TC, SC>() * sizeof(float);
}

// Weighted scatter (source/kernel.cu:717-756) by reductions of the load/store
// pipe, from the exchange buffer.
template <bool TC>
__device__ __forceinline__ void scatter_lsu(const FilterParams &prm, const float *S, float weight,
                                            const int (&pos)[8], int win, bool active, int me,
                                            int g) {
    const int tw = 2 * prm.radius + 1;
    // Thread `me` owns column `me` of every patch and adds one patch per
    // iteration of a rolled loop (the patch position comes from lane `p` of the
    // group). Pre-rounding with 2^extractor_exp makes the sums independent of the
    // atomic order; a multiplicity of 1 multiplies exactly.
    // Lane `me` resolves patch `me`'s target (plane pointer, multiplicity)
    // once; the loop takes patch p's from lane p of the group.
    const int pos_me = pick_pos(pos, me);
    const int z_me = pos_z(pos_me);
    float *const plane_me = prm.acc[(size_t)win * tw + z_me];
    const float mul_me = prm.mult ? prm.mult[(size_t)win * tw + z_me] : 1.0f;
    const unsigned long long dst_me =
        plane_me ? reinterpret_cast<unsigned long long>(
                       plane_me + (size_t)pos_y(pos_me) * prm.acc_stride + pos_x(pos_me))
                 : 0ull;
    const float ext = prm.extractor;
    const float wq = __fsub_rn(__fadd_rn(weight, ext), ext);
#pragma unroll 1
    for (int p = 0; p < 8; ++p) {
        float *wd = reinterpret_cast<float *>(__shfl_sync(0xffffffffu, dst_me, p, 8));
        const float mul = __shfl_sync(0xffffffffu, mul_me, p, 8);
        if (!active || wd == nullptr) continue;
        const float wm = __fmul_rn(wq, mul);
        float *wt = wd + prm.weight_offset;
        const float *sp = S + p * (TC ? 72 : 64);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            float val = __fmul_rn(weight, TC ? sp[r * 9 + me] : sp[row_pair_word(r, me, g)]);
            val = __fsub_rn(__fadd_rn(val, ext), ext);
            atomicAdd(wd + (size_t)r * prm.acc_stride + me, __fmul_rn(val, mul));
            if (!prm.corner_weight) atomicAdd(wt + (size_t)r * prm.acc_stride + me, wm);
        }
        if (prm.corner_weight && me == 0) atomicAdd(wt, wm);
    }
}

// Row `me` of a patch's box: the 8 values at words o .. o + 7 of 12, zeros
// around them (adding zero leaves a neighbour's sum as it is).
__device__ __forceinline__ void store_box_row(float *row, const float (&v)[8], int o) {
    float t[9], u[12];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const float same = i < 8 ? v[i < 8 ? i : 0] : 0.0f, left = i > 0 ? v[i > 0 ? i - 1 : 0] : 0.0f;
        t[i] = o & 1 ? left : same;
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        const float same = i < 9 ? t[i < 9 ? i : 0] : 0.0f;
        const float left = i > 1 && i < 11 ? t[i > 1 && i < 11 ? i - 2 : 0] : 0.0f;
        u[i] = o & 2 ? left : same;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        *reinterpret_cast<float4 *>(row + 4 * i) =
            make_float4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]);
}

// Adds a 12 x 8 box of shared memory to the accumulators at (x, y) of the map.
__device__ __forceinline__ void reduce_box(const CUtensorMap *map, int x, int y, const float *box) {
    asm volatile(
        "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], "
        "[%3];" ::"l"(map),
        "r"(x), "r"(y), "r"((unsigned)__cvta_generic_to_shared(box))
        : "memory");
}

// Weighted scatter of a warp's four groups by TMA reductions (thread = row `me`
// of group g, v[p][column]): each patch goes as one 8 x 12 box added to the
// accumulators, from the 16-byte boundary at or below its first pixel, so
// that the additions leave the load/store pipe, which bounds the filter. Lane
// `me` issues patch `me`'s box. Same terms as scatter_lsu.
// WEIGHTS: the patch's weight goes to all its pixels, as a second box from the
// one of four (one per column offset) that the group fills with its weight;
// multiplicities are 1. Else once, at the patch's corner.
template <bool WEIGHTS>
__device__ __forceinline__ void scatter_tma(const FilterParams &prm, const CUtensorMap *map,
                                            float *box, const float (&v)[8][8], float weight,
                                            const int (&pos)[8], int win, bool active, int me) {
    const int tw = 2 * prm.radius + 1;
    const int pos_me = pick_pos(pos, me);
    const int z_me = pos_z(pos_me);
    float *const plane_me = prm.acc[(size_t)win * tw + z_me];
    const float mul_me = prm.mult ? prm.mult[(size_t)win * tw + z_me] : 1.0f;
    const float ext = prm.extractor;
    const float wq = __fsub_rn(__fadd_rn(weight, ext), ext);
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const float mul = __shfl_sync(0xffffffffu, mul_me, p, 8);
        float t[8];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            // + ext in scalar form: the assembler contracts a packed product
            // with a packed sum (seen as 3 of 9600 outputs off by a quantum)
            float a, b;
            unpack2(mul2(splat2(weight), pack2(v[p][j], v[p][j + 1])), a, b);
            const f32x2 sum = pack2(__fadd_rn(a, ext), __fadd_rn(b, ext));
            unpack2(mul2(sub2(sum, splat2(ext)), splat2(mul)), t[j], t[j + 1]);
        }
        store_box_row(box + p * kBoxWords + me * 12, t, pos[p] & 3);
    }
    if constexpr (WEIGHTS) {
        const float t[8] = {wq, wq, wq, wq, wq, wq, wq, wq};
#pragma unroll
        for (int o = 0; o < 4; ++o) store_box_row(box + kBoxGroup + o * kBoxWords + me * 12, t, o);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (active && plane_me != nullptr) {
        // the target's index among the accumulator pairs, exact below 2^20 pairs
        const int pair = __float2int_rn((float)(plane_me - prm.acc_base) * prm.acc_pair_inv);
        const int y = pair * prm.acc_pair_rows + pos_y(pos_me);
        const int x = pos_x(pos_me) & ~3;
        reduce_box(map, x, y, box + me * kBoxWords);
        if constexpr (WEIGHTS)
            reduce_box(map, x, y + (prm.acc_pair_rows >> 1),
                       box + kBoxGroup + (pos_x(pos_me) & 3) * kBoxWords);
        else
            atomicAdd(plane_me + prm.weight_offset + (size_t)pos_y(pos_me) * prm.acc_stride +
                          pos_x(pos_me),
                      __fmul_rn(wq, mul_me));
    }
    // the boxes stay until they have been read
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// The kGroupsPerCta groups of CTA index `cta` of one filter launch; TC runs
// the transforms on the tensor cores (split BF16), else in FP32 with the
// reference's factorisation; VAR takes the transform kinds from prm.t2d /
// prm.t1d (FP32).
template <bool FINAL, bool TC, bool VAR, int SC>
__device__ __forceinline__ void filter_cta(const FilterParams &prm, const CUtensorMap *map,
                                           long long cta, float *fsm) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int g = lane >> 3;
    const int me = lane & 7;
    const long long row_groups = (long long)prm.nwin * prm.nbx;  // one block row, all windows
    const long long ngroups = row_groups * (prm.nblk / prm.nbx);
    const long long gid = cta * kGroupsPerCta + warp * 4 + g;
    const bool active = gid < ngroups;
    const long long gidc = active ? gid : 0;
    const int brow = (int)(gidc / row_groups);
    const long long rem = gidc - (long long)brow * row_groups;
    const int wrel = (int)(rem / prm.nbx);
    const int blk = brow * prm.nbx + (int)(rem - (long long)wrel * prm.nbx);
    const int win = prm.win0 + wrel;
    const int tw = 2 * prm.radius + 1;
    constexpr int kXchg = TC ? kXchgGroupTc : kXchgGroup;
    float *W = fsm + warp * warp_words<FINAL, TC, SC>();
    float *S = W + g * kXchg;
    SplitB Bf{}, Bi{};
    if (TC) {
        Bf = dct_fragment(true, lane);
        Bi = dct_fragment(false, lane);
    }

    int pos[8];
    {
        const int4 *m = reinterpret_cast<const int4 *>(prm.matches +
                                                       ((size_t)win * prm.nblk + blk) * 8);
        const int4 a = __ldg(m), b = __ldg(m + 1);
        pos[0] = a.x; pos[1] = a.y; pos[2] = a.z; pos[3] = a.w;
        pos[4] = b.x; pos[5] = b.y; pos[6] = b.z; pos[7] = b.w;
    }

    const float inv4096 = 1.0f / 4096.0f;
    const float sigma = prm.sigma;
    float v[8][8];
    float weight;

    if (FINAL) {
        // empirical Wiener shrinkage against the basic estimate's spectrum
        // (source/kernel.cu:284-326, cpu_source/source.cpp:617-643). The
        // noisy patches are copied asynchronously into C while the basic
        // estimate's group is loaded and transformed; then each thread swaps
        // its own slots of C: the basic spectrum's Wiener coefficients in,
        // the noisy pixels out, and the noisy group is transformed and
        // scaled by 1/4096 and its coefficient (the reference's two roundings).
        float *C = W + 4 * kXchg + g * kCoefGroup;
        prefetch_group(C, prm.src + (size_t)win * tw, pick_pos(pos, me), prm.stride, me);
        load_group(v, prm.ref + (size_t)win * tw, pos, prm.stride, me);
        const float sqr_sigma = __fmul_rn(sigma, sigma);
        float norm = 0.0f;
        // both forward transforms run through one copy of the code (a rolled
        // loop keeps the kernel small enough for the instruction caches)
#pragma unroll 1
        for (int it = 0; it < 2; ++it) {
            if (TC) tc_transform3d(v, S, W, me, lane, Bf);
            else if (VAR) forward3d_var(v, S, me, g, prm.t2d, prm.t1d);
            else forward3d(v, S, me, g);
            if (it == 1) break;
            asm volatile("cp.async.wait_all;" ::: "memory");
            // Two coefficients (rows r, r + 1) per packed FP32x2 instruction
            // stream; every lane is the scalar IEEE operation, and the
            // weight's sum of squares still runs in the reference's order
            // (p, then r).
            const f32x2 sig2 = splat2(sqr_sigma), one2 = splat2(1.0f);
#pragma unroll
            for (int p = 0; p < 8; ++p) {
#pragma unroll
                for (int r = 0; r < 8; r += 2) {
                    const f32x2 x = pack2(v[p][r], v[p][r + 1]);
                    const f32x2 sq = mul2(x, x);
                    // sq + sigma^2 >= sigma^2 >= (FLT_EPSILON * 0.188)^2: a normal float
                    const f32x2 den = add2(sq, sig2), nden = mul2(den, splat2(-1.0f));
                    f32x2 y = pack2(rcp_approx(lo2(den)), rcp_approx(hi2(den)));
                    f32x2 e = fma2(nden, y, one2);  // reciprocal as rcp_rn_normal
                    y = fma2(e, y, y);
                    float c0, c1;
                    unpack2(mul2(sq, y), c0, c1);
                    if (p == 0 && r == 0 && me == 0) c0 = 1.0f;  // DC passes unchanged
                    norm = __fmaf_rn(c0, c0, norm);
                    norm = __fmaf_rn(c1, c1, norm);
                    float *slot = C + (p * 8 + r) * 8 + me;
                    v[p][r] = slot[0];
                    v[p][r + 1] = slot[8];
                    slot[0] = c0;
                    slot[8] = c1;
                }
            }
        }
#pragma unroll
        for (int p = 0; p < 8; ++p)
#pragma unroll
            for (int r = 0; r < 8; r += 2) {
                const float *slot = C + (p * 8 + r) * 8 + me;
                float x0, x1;
                unpack2(mul2(pack2(v[p][r], v[p][r + 1]), splat2(inv4096)), x0, x1);
                v[p][r] = __fmul_rn(x0, slot[0]);
                v[p][r + 1] = __fmul_rn(x1, slot[8]);
            }
        norm = __fadd_rn(norm, __shfl_xor_sync(0xffffffffu, norm, 1, 8));
        norm = __fadd_rn(norm, __shfl_xor_sync(0xffffffffu, norm, 2, 8));
        norm = __fadd_rn(norm, __shfl_xor_sync(0xffffffffu, norm, 4, 8));
        weight = __fdiv_rn(1.0f, norm);
    } else {
        // hard thresholding (source/kernel.cu:208-252, cpu_source/source.cpp:562-594)
        load_group(v, prm.src + (size_t)win * tw, pos, prm.stride, me);
        if (TC) tc_transform3d(v, S, W, me, lane, Bf);
        else if (VAR) forward3d_var(v, S, me, g, prm.t2d, prm.t1d);
        else forward3d(v, S, me, g);
        int nnz = 0;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float thr = (p == 0 && r == 0 && me == 0) ? 0.0f : sigma;  // DC kept
                const float x = v[p][r];
                const bool keep = fabsf(x) >= thr;
                nnz += keep ? 1 : 0;
                v[p][r] = keep ? x : 0.0f;
            }
        }
#pragma unroll
        for (int p = 0; p < 8; p += 2)
#pragma unroll
            for (int r = 0; r < 8; ++r)
                unpack2(mul2(pack2(v[p][r], v[p + 1][r]), splat2(inv4096)), v[p][r], v[p + 1][r]);
        nnz += __shfl_xor_sync(0xffffffffu, nnz, 1, 8);
        nnz += __shfl_xor_sync(0xffffffffu, nnz, 2, 8);
        nnz += __shfl_xor_sync(0xffffffffu, nnz, 4, 8);
        weight = __fdiv_rn(1.0f, (float)nnz);
    }

    // inverse: rows, columns, group
    if (TC) {
        tc_transform3d<false>(v, S, W, me, lane, Bi);
        if constexpr (SC != kScatterLsu) {
#pragma unroll
            for (int p = 0; p < 8; ++p)
#pragma unroll
                for (int j = 0; j < 8; ++j) v[p][j] = S[p * 72 + me * 9 + j];
            __syncwarp();
        }
    } else {
        if (VAR) {
            pass_in_patch_var(v, false, prm.t2d);
            col_to_row(v, S, me);
            pass_in_patch_var(v, false, prm.t2d);
            pass_across_group_var(v, false, prm.t1d);
        } else {
            pass_in_patch(v, false);
            col_to_row(v, S, me);
            pass_in_patch(v, false);
            pass_across_group(v, false);
        }
        if constexpr (SC == kScatterLsu) {
            put_row(S, v, me, g);
            __syncwarp();
        }
    }
    if constexpr (SC == kScatterWeights)
        scatter_tma<true>(prm, map, W + g * (kBoxGroup + 4 * kBoxWords), v, weight, pos, win,
                          active, me);
    else if constexpr (SC == kScatterBoxes)
        scatter_tma<false>(prm, map, W + g * kBoxGroup, v, weight, pos, win, active, me);
    else
        scatter_lsu<TC>(prm, S, weight, pos, win, active, me, g);
}

// Resident CTAs per SM the register allocation aims at: the load/store form of the
// hard-threshold FP32 kernel runs 5 at 96 registers, 12 bytes of them spilled (one
// 640x360 window, block_step 1: 638 us, 675 at 4 without spills); boxes leave room
// for 4, with weights 3; the Wiener kernel's shared memory allows 3.
template <bool FINAL, bool TC, bool VAR, int SC>
constexpr int filter_ctas_per_sm() {
    return FINAL || SC == kScatterWeights ? 3 : (TC || VAR || SC == kScatterBoxes ? 4 : 5);
}

template <bool FINAL, bool TC, bool VAR, int SC>
__global__ void __launch_bounds__(128, filter_ctas_per_sm<FINAL, TC, VAR, SC>())
    filter_kernel(FilterParams prm, const __grid_constant__ CUtensorMap map) {
    extern __shared__ __align__(128) float fsm[];
    filter_cta<FINAL, TC, VAR, SC>(prm, &map, blockIdx.x, fsm);
}

// Persistent form over a batch of clips: resident CTAs take CTA-sized group
// ranges from a shared counter, clip-major. TMA: every clip has a tensor map.
// The maps lie in global memory, where another batch's may have been before, so a
// CTA that moves to a clip first orders its copy with the reads of the TMA unit.
template <bool FINAL, bool TMA>
__global__ void __launch_bounds__(128, filter_ctas_per_sm<FINAL, false, false, kScatterBoxes>())
    filter_batch_kernel(FilterBatch b) {
    extern __shared__ __align__(128) float fsm[];
    __shared__ FilterParams ps;
    __shared__ long long item_s;
    const long long total = b.item_off[b.nclips];
    int clip = -1;
    for (;;) {
        if (threadIdx.x == 0) item_s = (long long)atomicAdd(b.counter, 1ULL);
        __syncthreads();
        const long long item = item_s;
        if (item >= total) break;
        int lo = 0, hi = b.nclips;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (b.item_off[mid] <= item) lo = mid; else hi = mid;
        }
        if (threadIdx.x == 0) ps = b.clips[lo];
        if (TMA && lo != clip) {
            asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(b.maps + lo)
                         : "memory");
            clip = lo;
        }
        __syncthreads();
        filter_cta<FINAL, false, false, TMA ? kScatterBoxes : kScatterLsu>(
            ps, TMA ? b.maps + lo : nullptr, item - b.item_off[lo], fsm);
        __syncthreads();
    }
}

// dst = wdst / weight; with corner weights the weight of a pixel is the sum of
// the corner plane over its 8x8 up-left neighbourhood; corner sums run
// vertically then horizontally in a fixed order.
// A CTA of 256 threads covers a 128 x 16 tile; each thread 8 consecutive
// pixels of one row, loaded and stored as float4 pairs when aligned.
constexpr int kAggTx = 128, kAggTy = 16, kAggThreads = 256;

__device__ __forceinline__ void load8(float (&v)[8], const float *src, int x, int width,
                                      bool vec) {
    if (vec && x + 8 <= width) {
        const float4 u = *reinterpret_cast<const float4 *>(src);
        const float4 w = *reinterpret_cast<const float4 *>(src + 4);
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
        v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = x + k < width ? src[k] : 1.0f;
    }
}

// corner tile: columns x0-8 .. x0+kAggTx-1 (float4 aligned when x0 is), rows
// y0-7 .. y0+kAggTy-1; the smem pitch keeps every row 16-byte aligned
constexpr int kAggCq = (kAggTx + 8) / 4;                      // float4 per corner row
constexpr int kAggCp = kAggTx + 12;                           // smem pitch (floats)
constexpr int kAggCItems = (kAggTy + 7) * kAggCq;             // float4 per tile
constexpr int kAggCIter = (kAggCItems + kAggThreads - 1) / kAggThreads;

__device__ __forceinline__ void aggregate_tile(const AggregateParams &p, int tile_x, int tile_y,
                                               int pl) {
    __shared__ __align__(16) float corner[kAggTy + 7][kAggCp];
    __shared__ float colsum[kAggTy][kAggTx + 8];
    const int x0 = tile_x * kAggTx, y0 = tile_y * kAggTy;
    const float *wd = p.wdst + pl * p.acc_plane_stride;
    const float *wt = wd + p.weight_offset;
    const int tid = threadIdx.x;
    const int ly = tid / (kAggTx / 8), lx = (tid % (kAggTx / 8)) * 8;
    const int y = y0 + ly, x = x0 + lx;
    const bool ok = y < p.height && x < p.width;
    float a[8], w[8];
    if (ok) load8(a, wd + (size_t)y * p.acc_stride + x, x, p.width, p.vec);
    if (p.corner_weight) {
        // the weight of a pixel is the sum of the corner plane over its 8x8
        // up-left neighbourhood: column sums, then row sums, in a fixed order.
        // All of a thread's corner loads are issued before the first store to
        // shared memory (one memory latency per tile, not one per element).
        float4 cv[kAggCIter];
#pragma unroll
        for (int j = 0; j < kAggCIter; ++j) {
            const int i = tid + j * kAggThreads;
            const int ty = i / kAggCq, q = i - ty * kAggCq;
            const int gy = y0 - 7 + ty, gx = x0 - 8 + 4 * q;
            float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (i < kAggCItems && gy >= 0 && gy < p.height) {
                const float *row = wt + (size_t)gy * p.acc_stride;
                if (p.vec && gx >= 0 && gx + 4 <= p.width) {
                    const float4 u = *reinterpret_cast<const float4 *>(row + gx);
                    t[0] = u.x; t[1] = u.y; t[2] = u.z; t[3] = u.w;
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (gx + k >= 0 && gx + k < p.width) t[k] = row[gx + k];
                }
            }
            cv[j] = make_float4(t[0], t[1], t[2], t[3]);
        }
#pragma unroll
        for (int j = 0; j < kAggCIter; ++j) {
            const int i = tid + j * kAggThreads;
            const int ty = i / kAggCq, q = i - ty * kAggCq;
            if (i < kAggCItems) *reinterpret_cast<float4 *>(&corner[ty][4 * q]) = cv[j];
        }
        __syncthreads();
        // colsum column tx covers corner column tx + 1 (pixel x0 - 7 + tx). A
        // task is one column of 8 output rows: its 15 corner values are read
        // once and summed 8 at a time in the fixed order.
        static_assert(kAggTy % 8 == 0, "column tasks of 8 rows");
        for (int i = tid; i < (kAggTy / 8) * (kAggTx + 7); i += kAggThreads) {
            const int ty0 = 8 * (i / (kAggTx + 7)), tx = i % (kAggTx + 7);
            float c[15];
#pragma unroll
            for (int j = 0; j < 15; ++j) c[j] = corner[ty0 + j][tx + 1];
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                float s = 0.0f;
#pragma unroll
                for (int d = 0; d < 8; ++d) s = __fadd_rn(s, c[t + d]);
                colsum[ty0 + t][tx] = s;
            }
        }
        __syncthreads();
        if (!ok) return;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float s = 0.0f;
#pragma unroll
            for (int d = 0; d < 8; ++d) s = __fadd_rn(s, colsum[ly][lx + k + d]);
            w[k] = s;
        }
    } else {
        if (!ok) return;
        load8(w, wt + (size_t)y * p.acc_stride + x, x, p.width, p.vec);
    }
    float o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = __fdiv_rn(a[k], w[k]);
    float *dst = p.dst + pl * p.dst_plane_stride + (size_t)y * p.dst_stride + x;
    if (p.vec && x + 8 <= p.width) {
        *reinterpret_cast<float4 *>(dst) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4 *>(dst + 4) = make_float4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (x + k < p.width) dst[k] = o[k];
    }
}

__global__ void __launch_bounds__(kAggThreads, 5) aggregate_kernel(AggregateParams p) {
    aggregate_tile(p, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Persistent aggregation over a batch of clips. When `remaining` is set, the
// CTA that finishes a clip's last tile stamps the clip's completion time.
__global__ void __launch_bounds__(kAggThreads) aggregate_batch_kernel(AggregateBatch b) {
    __shared__ AggregateParams ps;
    __shared__ long long item_s;
    const long long total = b.item_off[b.nclips];
    for (;;) {
        if (threadIdx.x == 0) item_s = (long long)atomicAdd(b.counter, 1ULL);
        __syncthreads();
        const long long item = item_s;
        if (item >= total) break;
        int lo = 0, hi = b.nclips;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (b.item_off[mid] <= item) lo = mid; else hi = mid;
        }
        if (threadIdx.x == 0) ps = b.clips[lo];
        __syncthreads();
        const long long j = item - b.item_off[lo];
        const int ntx = (ps.width + kAggTx - 1) / kAggTx, nty = (ps.height + kAggTy - 1) / kAggTy;
        aggregate_tile(ps, (int)(j % ntx), (int)((j / ntx) % nty), (int)(j / ((long long)ntx * nty)));
        __syncthreads();
        if (threadIdx.x == 0 && b.remaining) {
            __threadfence();
            if (atomicSub(b.remaining + lo, 1u) == 1u) b.end_ns[lo] = globaltimer_ns();
        }
    }
}

// The stack of slot i of output frame n at (x, y), with replication padding at the
// clip ends (source/source.cpp:832-836); its weight plane lies p.height rows below.
__device__ __forceinline__ const float *vaggregate_slot(const VAggregateParams &p, int n, int i,
                                                        int x, int y) {
    const int s = min(max(2 * p.radius - i, n - p.num_frames + 1 + p.radius), n + p.radius);
    const float *f = p.base ? p.base + (size_t)min(max(n - p.radius + i, 0), p.num_frames - 1) *
                                           p.raw_frame_floats
                            : p.vf[i];
    return f + ((size_t)s * 2 * p.height + y) * p.raw_stride + x;
}

__global__ void vaggregate_kernel(VAggregateParams p) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    const int k = blockIdx.z;
    if (x >= p.width) return;
    const int tw = 2 * p.radius + 1;
    float sw = 0.0f, sv = 0.0f;
    for (int i = 0; i < tw; ++i) {
        const float *a = vaggregate_slot(p, p.n0 + k, i, x, y);
        sv = __fadd_rn(sv, a[0]);
        sw = __fadd_rn(sw, a[(size_t)p.height * p.raw_stride]);
    }
    p.dst[k * p.dst_plane_stride + (size_t)y * p.dst_stride + x] = __fdiv_rn(sv, sw);
}

// Four pixels per thread; the stacks of up to 5 slots are loaded before the first
// sum needs them.
__global__ void __launch_bounds__(128) vaggregate_quad_kernel(VAggregateParams p) {
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const int y = blockIdx.y;
    const int k = blockIdx.z;
    if (x >= p.width) return;
    const int tw = 2 * p.radius + 1;
    const size_t slab = (size_t)p.height * p.raw_stride;
    float sv[4] = {}, sw[4] = {};
    for (int i0 = 0; i0 < tw; i0 += 5) {
        float4 a[5], w[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (i0 + j >= tw) break;
            const float *src = vaggregate_slot(p, p.n0 + k, i0 + j, x, y);
            a[j] = __ldg(reinterpret_cast<const float4 *>(src));
            w[j] = __ldg(reinterpret_cast<const float4 *>(src + slab));
        }
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            if (i0 + j >= tw) break;
            sv[0] = __fadd_rn(sv[0], a[j].x);
            sv[1] = __fadd_rn(sv[1], a[j].y);
            sv[2] = __fadd_rn(sv[2], a[j].z);
            sv[3] = __fadd_rn(sv[3], a[j].w);
            sw[0] = __fadd_rn(sw[0], w[j].x);
            sw[1] = __fadd_rn(sw[1], w[j].y);
            sw[2] = __fadd_rn(sw[2], w[j].z);
            sw[3] = __fadd_rn(sw[3], w[j].w);
        }
    }
    float *dst = p.dst + k * p.dst_plane_stride + (size_t)y * p.dst_stride + x;
    float q[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) q[c] = __fdiv_rn(sv[c], sw[c]);
    if (x + 4 <= p.width) {
        *reinterpret_cast<float4 *>(dst) = make_float4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (x + c < p.width) dst[c] = q[c];
    }
}

}  // namespace

namespace {

template <bool FINAL, bool TC, bool VAR, int SC>
cudaError_t launch_filter_t(const FilterParams &p, const CUtensorMap &map, dim3 grid,
                            cudaStream_t stream) {
    // opt in to more than 48 KB of dynamic shared memory once per device
    static int configured[64] = {};
    const auto fn = filter_kernel<FINAL, TC, VAR, SC>;
    constexpr size_t smem = filter_smem<FINAL, TC, SC>();
    cudaError_t e = raise_smem_limit(configured, (const void *)fn, smem);
    if (e != cudaSuccess) return e;
    fn<<<grid, 128, smem, stream>>>(p, map);
    return cudaGetLastError();
}

// Where the eight block rows that cover a pixel are in flight at once, all of one
// plane, the additions to the same words bound the kernel, and a weight box adds 96
// words for a patch's 64 weights. (At block_step 1 up to 888 blocks a row, with 3
// CTAs of 16 groups on each of 148 SMs. One window, hard threshold, us, as boxes / by
// the load/store pipe: 413x186 288 / 265, 640x360 737 / 698, 850x200 509 / 508, 1000x250
// 675 / 701. The Wiener kernel's own work hides the additions: 640x360 756 / 901.)
bool crowded_windows(const FilterParams &p, bool final_) {
    return !final_ && !p.corner_weight && p.radius == 0 && p.block_step == 1 &&
           (long long)p.nwin * p.nbx * 8 <= 148 * 3 * kGroupsPerCta;
}

// The weight boxes leave room for 3 CTAs on an SM. Hard thresholding with the other
// transforms runs 4 by the load/store pipe and is little slower by that: it takes that
// form in small launches where the fourth place saves a wave. (One window, Hadamard,
// radius 0, us, as boxes / by the load/store pipe: 357 CTAs 39.0 / 37.0, 510 51.6 / 41.3, 586
// 59.0 / 48.1, 770 61.7 / 69.6, 1094 81.0 / 76.2, 1598 103.6 / 101.3, 3600 195.8 / 197.2. The
// DCT's form of 5 gains less by its places: 586 44.6 / 41.6, 1094 59.9 / 65.8.)
template <bool VAR>
bool weight_boxes_cost_a_wave(const FilterParams &p, bool final_, long long ctas) {
    const int boxes = 148 * 3, lsu = 148 * 4;
    return VAR && !final_ && !p.corner_weight && ctas <= 2 * lsu &&
           (ctas + boxes - 1) / boxes > (ctas + lsu - 1) / lsu;
}

template <bool TC, bool VAR>
cudaError_t launch_filter_form(const FilterParams &p, bool final_, dim3 grid,
                               cudaStream_t stream) {
    CUtensorMap map{};
    if ((!TC && crowded_windows(p, final_)) ||
        weight_boxes_cost_a_wave<VAR>(p, final_, grid.x) || !scatter_map(p, &map))
        return final_ ? launch_filter_t<true, TC, VAR, kScatterLsu>(p, map, grid, stream)
                      : launch_filter_t<false, TC, VAR, kScatterLsu>(p, map, grid, stream);
    if (p.corner_weight)
        return final_ ? launch_filter_t<true, TC, VAR, kScatterBoxes>(p, map, grid, stream)
                      : launch_filter_t<false, TC, VAR, kScatterBoxes>(p, map, grid, stream);
    return final_ ? launch_filter_t<true, TC, VAR, kScatterWeights>(p, map, grid, stream)
                  : launch_filter_t<false, TC, VAR, kScatterWeights>(p, map, grid, stream);
}

}  // namespace

bool scatter_map(const FilterParams &p, CUtensorMap *map) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) !=
                cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    // the box starts on a 16-byte boundary of its row; pair indices are exact
    // below 2^20, and rows are 32-bit coordinates
    if (!encode || !p.acc_base || (!p.corner_weight && p.mult) || p.acc_stride % 4 != 0 ||
        reinterpret_cast<unsigned long long>(p.acc_base) % 16 != 0 || p.acc_pairs >= (1 << 20) ||
        (long long)p.acc_pairs * p.acc_pair_rows > 0x7fffffffLL)
        return false;
    const cuuint64_t dims[2] = {(cuuint64_t)p.acc_stride,
                                (cuuint64_t)p.acc_pairs * (cuuint64_t)p.acc_pair_rows};
    const cuuint64_t pitch[1] = {(cuuint64_t)p.acc_stride * sizeof(float)};
    const cuuint32_t box[2] = {12, 8}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.acc_base, dims, pitch, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_filter(const FilterParams &p, bool final_, cudaStream_t stream) {
    const long long ngroups = (long long)p.nwin * p.nblk;
    if (ngroups == 0) return cudaSuccess;
    if (p.nbx <= 0 || p.nblk % p.nbx != 0) return cudaErrorInvalidValue;
    const long long nblocks = (ngroups + kGroupsPerCta - 1) / kGroupsPerCta;
    if (nblocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)nblocks);
    if (p.t2d < 0 || p.t2d > 3 || p.t1d < 0 || p.t1d > 3) return cudaErrorInvalidValue;
    if (p.t2d != 0 || p.t1d != 0) {
        if (p.precision != 0) return cudaErrorInvalidValue;  // variants run in FP32
        return launch_filter_form<false, true>(p, final_, grid, stream);
    }
    if (p.precision == 2) return launch_filter_tc(p, final_, stream);
    return p.precision == 1 ? launch_filter_form<true, false>(p, final_, grid, stream)
                            : launch_filter_form<false, false>(p, final_, grid, stream);
}

namespace {

// Resident CTAs of a persistent launch: SMs x `per_sm_want` CTAs, at most
// the occupancy limit (per_sm_want <= 0: the limit).
int persistent_grid(const void *fn, int threads, size_t smem, int per_sm_want = 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    per_sm = std::max(1, per_sm);
    if (per_sm_want > 0) per_sm = std::min(per_sm, per_sm_want);
    return std::max(1, sms) * per_sm;
}

}  // namespace

namespace {

template <bool FINAL, bool TMA>
cudaError_t launch_filter_batch_t(const FilterBatch &b, cudaStream_t stream, int ctas_per_sm) {
    static int configured[64] = {};
    const auto fn = filter_batch_kernel<FINAL, TMA>;
    constexpr size_t smem = filter_smem<FINAL, false, TMA ? kScatterBoxes : kScatterLsu>();
    cudaError_t e = raise_smem_limit(configured, (const void *)fn, smem);
    if (e != cudaSuccess) return e;
    fn<<<persistent_grid((const void *)fn, 128, smem, ctas_per_sm), 128, smem, stream>>>(b);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_filter_batch(const FilterBatch &b, bool final_, cudaStream_t stream,
                                int ctas_per_sm) {
    if (b.maps)
        return final_ ? launch_filter_batch_t<true, true>(b, stream, ctas_per_sm)
                      : launch_filter_batch_t<false, true>(b, stream, ctas_per_sm);
    return final_ ? launch_filter_batch_t<true, false>(b, stream, ctas_per_sm)
                  : launch_filter_batch_t<false, false>(b, stream, ctas_per_sm);
}

long long filter_ctas(const FilterParams &p) {
    return ((long long)p.nwin * p.nblk + kGroupsPerCta - 1) / kGroupsPerCta;
}

long long aggregate_tiles(const AggregateParams &p) {
    return (long long)((p.width + kAggTx - 1) / kAggTx) * ((p.height + kAggTy - 1) / kAggTy) *
           p.nplanes;
}

bool aggregate_vec(const AggregateParams &p) {
    const unsigned long long align = reinterpret_cast<unsigned long long>(p.wdst) |
                                     reinterpret_cast<unsigned long long>(p.dst);
    return (align % 16 == 0) && p.acc_stride % 4 == 0 && p.dst_stride % 4 == 0 &&
           p.acc_plane_stride % 4 == 0 && p.dst_plane_stride % 4 == 0 && p.weight_offset % 4 == 0;
}

cudaError_t launch_aggregate_batch(const AggregateBatch &b, cudaStream_t stream,
                                   int ctas_per_sm) {
    const int grid = persistent_grid((const void *)aggregate_batch_kernel, kAggThreads, 0,
                                     ctas_per_sm);
    aggregate_batch_kernel<<<grid, kAggThreads, 0, stream>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_aggregate(const AggregateParams &p, cudaStream_t stream) {
    if (p.nplanes == 0) return cudaSuccess;
    AggregateParams q = p;
    // float4 access needs 16-byte aligned rows in every plane
    const unsigned long long align = reinterpret_cast<unsigned long long>(p.wdst) |
                                     reinterpret_cast<unsigned long long>(p.dst);
    q.vec = (align % 16 == 0) && p.acc_stride % 4 == 0 && p.dst_stride % 4 == 0 &&
            p.acc_plane_stride % 4 == 0 && p.dst_plane_stride % 4 == 0 &&
            p.weight_offset % 4 == 0;
    dim3 block(kAggThreads);
    dim3 grid((p.width + kAggTx - 1) / kAggTx, (p.height + kAggTy - 1) / kAggTy, p.nplanes);
    aggregate_kernel<<<grid, block, 0, stream>>>(q);
    return cudaGetLastError();
}

cudaError_t launch_vaggregate(const VAggregateParams &p, cudaStream_t stream) {
    if (p.nout == 0) return cudaSuccess;
    // Quads where every row of every stack starts on 16 bytes (rows then have room
    // for the last quad, the stride being a multiple of 4) and is wider than a block of
    // single pixels: below that both have as many blocks, and a quad's thread four times
    // the work. (One frame, single pixels / quads, us: 1920x1080, radius 2 18.6 / 10.4, 3 26.8
    // / 22.7; 160x2000, radius 3 7.4 / 6.3; 64x2000, radius 3 5.1 / 6.2.)
    unsigned long long align = reinterpret_cast<unsigned long long>(p.dst) |
                               reinterpret_cast<unsigned long long>(p.base);
    if (!p.base)
        for (int i = 0; i < 2 * p.radius + 1; ++i)
            align |= reinterpret_cast<unsigned long long>(p.vf[i]);
    const bool quads = p.width > 128 && align % 16 == 0 && p.raw_stride % 4 == 0 &&
                       p.dst_stride % 4 == 0 && p.raw_frame_floats % 4 == 0 &&
                       p.dst_plane_stride % 4 == 0;
    const int per_block = quads ? 512 : 128;
    const dim3 block(128), grid((p.width + per_block - 1) / per_block, p.height, p.nout);
    if (quads)
        vaggregate_quad_kernel<<<grid, block, 0, stream>>>(p);
    else
        vaggregate_kernel<<<grid, block, 0, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace bm3d
