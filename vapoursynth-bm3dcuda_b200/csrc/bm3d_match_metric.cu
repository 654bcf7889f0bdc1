// The general matching kernel with the run-time-compiled plugin's distances
// (bm3d_match_kernels.cuh).
#include "bm3d_match_kernels.cuh"

namespace bm3d {

namespace {

template <int K, int M, bool SMALL>
cudaError_t launch_metric(MatchParams q, const MatchGeometry &g, int nwin, int lanes,
                          cudaStream_t stream) {
    q.nsub_s = (2 * q.bm_range + K) / K;
    q.nsub_t = (2 * q.ps_range + K) / K;
    const int over_s = q.nsub_s * K - (2 * q.bm_range + 1);
    const int over_t = q.radius > 0 ? q.nsub_t * K - (2 * q.ps_range + 1) : 0;
    q.extra_cols = std::max(over_s, over_t);
    const int mmax = q.bm_range + q.radius * q.ps_range;
    const int wx = lanes == 1 ? g.wx : kSplitWx, wy = lanes == 1 ? 1 : kSplitWy;
    const int rows = 8 / lanes * wy;  // block rows of a CTA
    q.pitch = (4 * wx - 1) * q.block_step + 2 * mmax + 16 + q.extra_cols;
    q.tile_rows = (rows - 1) * q.block_step + 2 * mmax + 8;
    const size_t lists = (size_t)(SMALL ? 16 : 8) * 32 * wx * wy * sizeof(int);
    const auto bytes = [&] { return (size_t)q.pitch * q.tile_rows * sizeof(float) + lists; };
    // a range that only just fits: one candidate per strip needs no extra columns
    if (bytes() > kMatchSmemMax)
        return K == 1 ? cudaErrorInvalidValue
                      : launch_metric<1, M, false>(q, g, nwin, 1, stream);
    // Another pitch where the base one meets clearly more conflicts (it has 18 in 8
    // accesses at block_step 3 and 7, where 16 gain nothing: 158x501, ps_num 3: 529 us,
    // 557 at the other; 900x300 at block_step 1, bm_range 9, radius 1, ps_num 4,
    // 64 in 8: 9.26 ms in strips of 8, 4.49 with 15 in 8, 3.18 in strips of 10).
    q.pitch = match_pitch(q.pitch, q.block_step, lanes == 1 ? 0 : 2, q.tile_rows, lists,
                          12 / (wx * wy), kMatchSmemMax, 1.5);
    const size_t smem = bytes();
    const dim3 grid((q.nbx + 4 * wx - 1) / (4 * wx), (q.nby + rows - 1) / rows, nwin);
    const dim3 block(32 * wx * wy);
    if constexpr (SMALL) {
        if (lanes > 1) return launch_match_t<K, K, M, 4, true>(q, grid, block, smem, stream);
        // three CTAs per SM once there are several waves of them (1020 CTAs, 4 x
        // 1920x1080: SSD/NORM 648 us, 714 with two; 240 CTAs: 223, 213)
        if ((long long)grid.x * grid.y * grid.z > 600)
            return launch_match_t<K, K, M, 1, true, 3>(q, grid, block, smem, stream);
    }
    return launch_match_t<K, K, M, 1, SMALL>(q, grid, block, smem, stream);
}

template <int K, int M>
cudaError_t launch_metric_k(const MatchParams &p, const MatchGeometry &g, int nwin, int lanes,
                            cudaStream_t stream) {
    return p.radius > 0 && p.ps_num > 2 ? launch_metric<K, M, false>(p, g, nwin, 1, stream)
                                        : launch_metric<K, M, true>(p, g, nwin, lanes, stream);
}

template <int M>
cudaError_t launch_metric_m(const MatchParams &p, const MatchGeometry &g, int nwin, int K,
                            int lanes, cudaStream_t stream) {
    switch (K) {
        case 4: return launch_metric_k<4, M>(p, g, nwin, lanes, stream);
        case 10: return launch_metric_k<10, M>(p, g, nwin, lanes, stream);
        default: return launch_metric_k<8, M>(p, g, nwin, lanes, stream);
    }
}

}  // namespace

cudaError_t launch_match_metric(const MatchParams &p, const MatchGeometry &g, int nwin, int K,
                                int lanes, cudaStream_t stream) {
    switch (p.metric) {
        case 1: return launch_metric_m<1>(p, g, nwin, K, lanes, stream);
        case 2: return launch_metric_m<2>(p, g, nwin, K, lanes, stream);
        case 3: return launch_metric_m<3>(p, g, nwin, K, lanes, stream);
        case 4: return launch_metric_m<4>(p, g, nwin, K, lanes, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace bm3d
