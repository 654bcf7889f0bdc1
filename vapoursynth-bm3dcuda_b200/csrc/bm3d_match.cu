// Block matching for BM3D / V-BM3D: geometry, dispatch, and the general kernels
// (bm3d_match_kernels.cuh).
#include "bm3d_match_kernels.cuh"

namespace bm3d {

namespace {

// Operations per candidate of windows of `w` columns in strips of K: the strip
// overrun, ~143 FP32 operations per distance and 8 (K + 7) / K shared-memory
// loads.
double strip_cost(int w, int K) {
    return (double)((w + K - 1) / K * K) / w * (143.0 + 8.0 * (K + 7) / K);
}

// Strip width K (candidates per strip) for a spatial window of ws columns and
// temporal windows of wt columns, both scanned with the same K: the K in
// [8, 12] with the fewest operations.
int choose_strip_width(int ws, int wt, int radius, int ps_num) {
    const double spatial = (double)ws * ws;
    const double temporal = radius > 0 ? 2.0 * radius * ps_num * wt * wt : 0.0;
    int best = 8;
    double best_cost = 1e300;
    for (int K = 8; K <= 12; ++K) {
        const double cost =
            spatial * strip_cost(ws, K) + (temporal > 0.0 ? temporal * strip_cost(wt, K) : 0.0);
        if (cost < best_cost) {
            best_cost = cost;
            best = K;
        }
    }
    return best;
}

// The same for windows of one width, among the widths compiled for them.
template <int N>
int choose_strip_width(int w, const int (&widths)[N]) {
    int best = widths[0];
    for (int K : widths)
        if (strip_cost(w, K) < strip_cost(w, best)) best = K;
    return best;
}

// Shared-memory row pitch of at least `base` words for a tile whose warps own
// 4 x rows reference blocks, 1 << log_lanes lanes each (lane `sub` of a block
// reads `sub` rows below): of the 16 next, the one with the fewest bank
// conflicts when all lanes read the same candidate offset, summed over the 8
// phases of the row skew. It runs with each call that plans its own search, so
// it counts bank masks instead of lanes (1.0 us for a pitch, 5.3 lane by
// lane). `gain`: a pitch has to save that factor of the base's conflicts.
int pick_pitch(int base, int block_step, int log_lanes, double gain) {
    const int rows = 8 >> log_lanes, lanes = 1 << log_lanes;
    // the banks of four neighbouring blocks, distinct for every block_step up to 8
    const unsigned quad = 1u | 1u << block_step | 1u << 2 * block_step | 1u << 3 * block_step;
    int best = base, best_cost = 1 << 30, base_cost = 0;
    for (int pitch = base; pitch < base + 16 && best_cost > 8; ++pitch) {
        int cost = 0;
        // a phase costs at least 1: stop where the pitch cannot win any more
        for (int phase = 0; phase < 8 && cost + 8 - phase <= best_cost; ++phase) {
            unsigned hit[8] = {};  // hit[k]: the banks with more than k accesses
            for (int r = 0; r < rows; ++r) {
                for (int sub = 0; sub < lanes; ++sub) {
                    const int ty = phase + r * block_step + sub;
                    const unsigned shift = (ty * pitch + ((ty >> 3) & 7)) & 31;
                    unsigned banks = quad << shift | quad >> ((32 - shift) & 31);
                    for (int k = 0; banks; ++k) {
                        const unsigned again = hit[k] & banks;
                        hit[k] |= banks;
                        banks = again;
                    }
                }
            }
            for (int k = 0; k < 8 && hit[k]; ++k) ++cost;
            if (phase < 7 && cost + 7 - phase >= best_cost) cost = best_cost;
        }
        if (pitch == base) base_cost = cost;
        if (cost < best_cost) {
            best_cost = cost;
            best = pitch;
        }
    }
    return best_cost * gain > base_cost ? base : best;
}

// A warp's match lists: 16 words per thread (SMALL), else 8.
constexpr size_t kSmallListBytes = 16 * 32 * sizeof(int), kListBytes = 8 * 32 * sizeof(int);
// Shared memory of an SM; the hardware reserves 1 KB of it per CTA.
constexpr size_t kSmemPerSm = 228 * 1024;

}  // namespace

int match_pitch(int base, int block_step, int log_lanes, int tile_rows, size_t list_bytes,
                int ctas, size_t limit, double gain) {
    const int pitch = pick_pitch(base, block_step, log_lanes, gain);
    const auto bytes = [&](int p) { return (size_t)p * tile_rows * sizeof(float) + list_bytes; };
    const auto resident = [&](int p) {
        return std::min<size_t>(ctas, kSmemPerSm / (bytes(p) + 1024));
    };
    return bytes(pitch) <= limit && resident(pitch) == resident(base) ? pitch : base;
}

// 8 or 10 as for the SSD; 4 where that spares a third of the candidates computed
// (the list costs more in narrow strips: windows of 11 columns run 4% faster in
// strips of 4 than of 8 in the spatial stage, up to 8% slower in the temporal ones).
// Whole-window time with strips of 4 / 8 / 10 against one candidate at a time, ZSSD,
// 1320x428 at block_step 2:
//   bm_range 1, radius 0                           0.87 0.91 0.93
//   bm_range 5, radius 1, ps_num 2, ps_range 1     0.72 0.83 0.92
//   bm_range 6, radius 0                           0.77 0.72 0.80
//   bm_range 9, radius 0                           0.52 0.53 0.47
//   bm_range 4, radius 1, ps_num 8, ps_range 1     0.86 1.08 1.12
//   bm_range 9, radius 1, ps_num 4, ps_range 4     0.82 0.83 0.58
int metric_strip_width(int bm_range, int radius, int ps_num, int ps_range) {
    const int ws = 2 * bm_range + 1, wt = 2 * ps_range + 1;
    const double spatial = (double)ws * ws, temporal = 2.0 * radius * ps_num * wt * wt;
    const auto cost = [&](int K) {
        return spatial * strip_cost(ws, K) + temporal * strip_cost(wt, K);
    };
    const auto computed = [&](int K) {
        return spatial * ((ws + K - 1) / K * K) / ws + temporal * ((wt + K - 1) / K * K) / wt;
    };
    const int K = cost(10) < cost(8) ? 10 : 8;
    return 1.5 * computed(4) <= computed(K) ? 4 : K;
}

int temporal_strip_width(int ps_range) {
    const int widths[] = {8, 9, 11};
    return choose_strip_width(2 * ps_range + 1, widths);
}

MatchGeometry match_geometry_with(int width, int height, int block_step, int bm_range, int radius,
                                  int ps_range, int wx, int ks, int kt, bool small) {
    MatchGeometry g{};
    g.nbx = (width - 8 + block_step - 1) / block_step + 1;
    g.nby = (height - 8 + block_step - 1) / block_step + 1;
    const int ws = 2 * bm_range + 1, wt = 2 * ps_range + 1;
    g.small = small;
    g.ks = ks;
    g.kt = kt;
    g.nsub_s = (ws + g.ks - 1) / g.ks;
    g.nsub_t = (wt + g.kt - 1) / g.kt;
    g.extra_cols = std::max(g.nsub_s * g.ks - ws, radius > 0 ? g.nsub_t * g.kt - wt : 0);
    const int mmax = bm_range + radius * ps_range;
    const size_t lists = small ? kSmallListBytes : kListBytes;
    g.wx = wx;
    g.pitch = (4 * wx - 1) * block_step + 2 * mmax + 8 + g.extra_cols + 8;
    g.tile_rows = 7 * block_step + 2 * mmax + 8;
    g.smem = (size_t)g.pitch * g.tile_rows * sizeof(float) + lists * wx;
    return g;
}

void choose_pitches(MatchGeometry &g, int block_step, int bm_range, int radius, int ps_range,
                    size_t limit) {
    const int mmax = bm_range + radius * ps_range;
    const size_t lists = g.small ? kSmallListBytes : kListBytes;
    // the conflict-free pitch where it costs no resident CTA (block steps 4 and
    // 2 meet 4-way bank conflicts at an arbitrary pitch)
    g.pitch = match_pitch(g.pitch, block_step, 0, g.tile_rows, lists * g.wx, 12 / g.wx, limit);
    g.smem = (size_t)g.pitch * g.tile_rows * sizeof(float) + lists * g.wx;
    for (int i = 0; i < 2; ++i) {
        const int lanes = 4 << i;
        auto &sp = g.split[i];
        const int tw = (4 * kSplitWx - 1) * block_step + 2 * mmax + 8 + g.extra_cols;
        sp.tile_rows = (kSplitWy * 8 / lanes - 1) * block_step + 2 * mmax + 8;
        sp.pitch = match_pitch(tw + 8, block_step, 2 + i, sp.tile_rows,
                               lists * kSplitWx * kSplitWy, 1, kMatchSmemMax);
        sp.smem = (size_t)sp.pitch * sp.tile_rows * sizeof(float) + lists * kSplitWx * kSplitWy;
    }
}

size_t match_range_bytes(int block_step, int bm_range, int radius, int ps_range, int wx, int K) {
    const int ws = 2 * bm_range + 1, wt = 2 * ps_range + 1, mmax = bm_range + radius * ps_range;
    const int over_s = (ws + K - 1) / K * K - ws;
    const int over_t = radius > 0 ? (wt + K - 1) / K * K - wt : 0;
    const size_t pitch = (4 * wx - 1) * block_step + 2 * mmax + 16 + std::max(over_s, over_t);
    return pitch * (7 * block_step + 2 * mmax + 8) * sizeof(float) + kListBytes * wx;
}

MatchGeometry match_geometry(int width, int height, int block_step, int bm_range, int radius,
                             int ps_num, int ps_range) {
    const int ws = 2 * bm_range + 1, wt = 2 * ps_range + 1;
    MatchGeometry g{};
    const bool small = radius == 0 || ps_num <= 2;
    // the CTA width with the most resident warps, the widest of equals (8 windows
    // of 1920x1080, radius 2, bm_range 16: two CTAs of 4 warps on an SM 2.88 ms,
    // three of 2 warps 3.7)
    auto widest = [&](int ks, int kt, bool two_entries) {
        MatchGeometry best{};
        int best_warps = 0;
        for (int wx = 4; wx >= 1; wx /= 2) {
            const MatchGeometry t = match_geometry_with(width, height, block_step, bm_range,
                                                        radius, ps_range, wx, ks, kt, two_entries);
            const int warps =
                std::min<int>(12, (int)(kSmemPerSm / (t.smem + 1024)) * wx);
            if (warps > best_warps || best.wx == 0) {
                best_warps = warps;
                best = t;
            }
        }
        return best;
    };
    if (small) {
        const int spatial[] = {8, 9, 10, 11};
        g = widest(choose_strip_width(ws, spatial), radius == 0 ? 9 : temporal_strip_width(ps_range),
                   true);
    }
    // a range that only just fits keeps to the strips that need the least room
    if (!small || g.smem > 200 * 1024) {
        const int K = choose_strip_width(ws, wt, radius, 2);
        g = widest(K, K, false);
    }
    choose_pitches(g, block_step, bm_range, radius, ps_range);
    return g;
}

bool match_too_large(int block_step, int bm_range, int radius, int ps_range) {
    const int K = choose_strip_width(2 * bm_range + 1, 2 * ps_range + 1, radius, 2);
    return match_range_bytes(block_step, bm_range, radius, ps_range, 1, K) > kMatchSmemLimit;
}

// Resident CTAs per SM for the small SSD search, one lane per block: times at
// 168 registers and three CTAs, and at about 200 and two, us:
//   240 CTAs (8 x 640x360, radius 0)              103    95
//   255 CTAs (1920x1080, radius 2)                276   251
//   460 CTAs (2560x1440, radius 0)                187   178
//   1020 CTAs (3840x2160, radius 0, bm_range 16)  801   791
//   1080 CTAs (3 x 853x479, step 3)              1609  1554
//   2040 CTAs (8 x 1920x1080, radius 0)           601   611
//   3060 CTAs (12 x 1920x1080, radius 2)         2405  2421
//   2040 CTAs whose tile leaves room for two:
//     8 x 1920x1080, radius 3                    2405  2135
int match_ctas(const MatchGeometry &g, int nwin) {
    return match_tiles(g, nwin) > 1100 && kSmemPerSm / (g.smem + 1024) >= 3 ? 3 : 2;
}

long long match_tiles(const MatchGeometry &g, int nwin) {
    return (long long)((g.nbx + 4 * g.wx - 1) / (4 * g.wx)) * ((g.nby + 7) / 8) * nwin;
}

// Lanes per reference block: one, unless the launch leaves most of the GPU's
// 148 x 12 resident warps idle, or the search range lets an SM hold only one
// CTA of four warps with one lane per block (the split tiles hold 32 blocks, not
// 128). More lanes shorten each thread's scan and cost insertions (every lane
// fills a list of its own) and a merge. Times with 1, 4 and 8 lanes, us:
//   120 warps (640x360, radius 0)      65   25   23
//   224 warps (640x360 step 6, r 2)   183   99  103
//   288 warps (960x540, r 1)          111   62   80
//   336 warps (2 x 333x211, r 1)      242  129  171
//   480 warps (1280x720, r 0)          64   60   69
//   480 warps (1280x720, r 3)         136  145  181
//   880 warps (1760x990, r 1)         173  175  230
//   960 warps (8 x 640x360, r 0)       95  107  123
//   one CTA per SM: 2 x 1920x1080, r 3, bm_range 16, ps_range 6   1839  1724
//                   2 x 1280x720, r 2, bm_range 20, ps_range 8    1046   923
// Windows of 5 x 5 and less are little work to share (bm_range 2, radius 0):
//   200 warps (800x450)              16.6 13.0 14.7
//   270 warps (960x540)              16.9 13.6 15.6
//   350 warps (1100x620)             17.0 18.5 18.8
//   480 warps (1280x720)             16.6 19.5 22.8
//   572 warps (700x400 step 4)       16.1 20.3 25.0
// Ranges near the limit fit the one-warp CTA of one lane per block but not the
// four-warp CTA of the split forms.
int match_lanes(const MatchGeometry &g, int bm_range, int radius, int nwin) {
    const long long warps =
        (long long)((g.nbx + 3) / 4) * ((g.nby + 7) / 8) * nwin;  // of 4 x 8 blocks
    const bool fits[2] = {g.split[0].smem <= kMatchSmemMax, g.split[1].smem <= kMatchSmemMax};
    if (warps <= 160 && fits[1]) return 8;
    const int few = radius == 0 ? (bm_range <= 2 ? 300 : 600) : 450;
    if (warps <= few && fits[0]) return 4;
    return kSmemPerSm / (g.smem + 1024) * g.wx <= 4 && g.split[0].smem < g.smem / 2 ? 4 : 1;
}

cudaError_t launch_match_split(const MatchParams &p, const MatchGeometry &g, int nwin, int lanes,
                               cudaStream_t stream) {
    if (g.small) return launch_match_pairs(p, g, nwin, lanes, stream);
    switch (g.ks) {
        case 9: return launch_match_lanes<9, 9, false>(p, g, nwin, lanes, stream);
        case 10: return launch_match_lanes<10, 10, false>(p, g, nwin, lanes, stream);
        case 11: return launch_match_lanes<11, 11, false>(p, g, nwin, lanes, stream);
        case 12: return launch_match_lanes<12, 12, false>(p, g, nwin, lanes, stream);
        default: return launch_match_lanes<8, 8, false>(p, g, nwin, lanes, stream);
    }
}

cudaError_t launch_match(const MatchParams &p, const MatchGeometry &g, int nwin,
                         cudaStream_t stream) {
    const int lanes = match_lanes(g, p.bm_range, p.radius, nwin);
    if (p.metric != 0) {
        const int K = metric_strip_width(p.bm_range, p.radius, p.ps_num, p.ps_range);
        return launch_match_metric(p, g, nwin, K, lanes == 1 ? 1 : 4, stream);
    }
    return launch_match_split(p, g, nwin, lanes, stream);
}

}  // namespace bm3d
