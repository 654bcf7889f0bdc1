// Block matching of a batch of clips: the persistent form of the matching
// kernels (bm3d_match_kernels.cuh).
#include "bm3d_match_kernels.cuh"

namespace bm3d {

namespace {

// Persistent form for a batch of clips with their own geometry and
// parameters: resident CTAs take CTA tiles from a shared counter, clip-major
// in the order the clips were added; per-clip parameters are staged in
// shared memory for the tile.
template <int K, int KT, bool SMALL, int CTAS>
__global__ void __launch_bounds__(128, CTAS) match_batch_kernel(MatchBatch b) {
    extern __shared__ float tile[];
    __shared__ MatchParams ps;
    __shared__ long long item_s;
    static_assert(sizeof(ps) + sizeof(item_s) <= kMatchBatchStatic, "room beside the tile");
    const long long total = b.item_off[b.nclips];
    const int nbx_cta = (blockDim.x >> 5) * 4;
    for (;;) {
        if (threadIdx.x == 0) {
            item_s = (long long)atomicAdd(b.counter, 1ULL);
            if (item_s == 0) *b.start_ns = globaltimer_ns();
        }
        __syncthreads();
        const long long item = item_s;
        if (item >= total) break;
        int lo = 0, hi = b.nclips;  // item_off[lo] <= item < item_off[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (b.item_off[mid] <= item) lo = mid; else hi = mid;
        }
        if (threadIdx.x == 0) ps = b.clips[lo];
        __syncthreads();
        const long long j = item - b.item_off[lo];
        const int ntx = (ps.nbx + nbx_cta - 1) / nbx_cta, nty = (ps.nby + 7) / 8;
        const int tx = (int)(j % ntx), ty = (int)((j / ntx) % nty), win = (int)(j / ((long long)ntx * nty));
        match_tile<K, KT, 0, 1, SMALL>(ps, tx, ty, win, tile);
        __syncthreads();
    }
}

template <int K, int KT, bool SMALL, int CTAS>
cudaError_t launch_match_batch_t(const MatchBatch &b, int wx, size_t smem, cudaStream_t stream) {
    auto fn = match_batch_kernel<K, KT, SMALL, CTAS>;
    static int configured[64] = {0};
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = raise_smem_limit(configured, (const void *)fn, smem)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * wx, smem)) !=
        cudaSuccess)
        return e;
    fn<<<sms * std::max(1, per_sm), 32 * wx, smem, stream>>>(b);
    return cudaGetLastError();
}

template <int K>
cudaError_t launch_match_batch_k(const MatchBatch &b, int kt, bool small, int wx, size_t smem,
                                 cudaStream_t stream) {
    if (!small) return launch_match_batch_t<K, K, false, 2>(b, wx, smem, stream);
    // the registers for three CTAs per SM where the largest tile leaves room
    // for them (match_ctas)
    if (3 * (smem + 1024) <= 228 * 1024)
        return kt == 11 ? launch_match_batch_t<K, 11, true, 3>(b, wx, smem, stream)
                        : launch_match_batch_t<K, 9, true, 3>(b, wx, smem, stream);
    return kt == 11 ? launch_match_batch_t<K, 11, true, 2>(b, wx, smem, stream)
                    : launch_match_batch_t<K, 9, true, 2>(b, wx, smem, stream);
}

}  // namespace

cudaError_t launch_match_batch(const MatchBatch &b, int K, int kt, bool small, int wx, size_t smem,
                               cudaStream_t stream) {
    if (smem > kMatchBatchSmemMax) return cudaErrorInvalidValue;
    switch (K) {
        case 9: return launch_match_batch_k<9>(b, kt, small, wx, smem, stream);
        case 10: return launch_match_batch_k<10>(b, kt, small, wx, smem, stream);
        case 11: return launch_match_batch_k<11>(b, kt, small, wx, smem, stream);
        case 12: return launch_match_batch_k<12>(b, kt, small, wx, smem, stream);
        default: return launch_match_batch_k<8>(b, kt, small, wx, smem, stream);
    }
}

}  // namespace bm3d
