// The two-entry matching kernels (ps_num <= 2 or no neighbour frames) for each
// pair of strip widths (bm3d_match_kernels.cuh).
#include "bm3d_match_kernels.cuh"

namespace bm3d {

namespace {

template <int K>
cudaError_t launch_match_small(const MatchParams &p, const MatchGeometry &g, int nwin, int lanes,
                               cudaStream_t stream) {
    switch (g.kt) {
        case 8: return launch_match_lanes<K, 8, true>(p, g, nwin, lanes, stream);
        case 11: return launch_match_lanes<K, 11, true>(p, g, nwin, lanes, stream);
        default: return launch_match_lanes<K, 9, true>(p, g, nwin, lanes, stream);
    }
}

}  // namespace

cudaError_t launch_match_pairs(const MatchParams &p, const MatchGeometry &g, int nwin, int lanes,
                               cudaStream_t stream) {
    switch (g.ks) {
        case 9: return launch_match_small<9>(p, g, nwin, lanes, stream);
        case 10: return launch_match_small<10>(p, g, nwin, lanes, stream);
        case 11: return launch_match_small<11>(p, g, nwin, lanes, stream);
        default: return launch_match_small<8>(p, g, nwin, lanes, stream);
    }
}

}  // namespace bm3d
