// Instantiates the split-KV decode attention kernels for one head_dim (FTQ_D).
#include "ftq_attn_flow.cuh"
#include "ftq_launch.h"

#include <atomic>

#ifndef FTQ_D
#error "compile with -DFTQ_D=64, 128 or 256"
#endif
#define FTQ_CAT2(a, b) a##b
#define FTQ_CAT(a, b) FTQ_CAT2(a, b)

namespace ftq {

template <int BK, int BV, bool PAGED>
static cudaError_t run_split(const AttnParams& p, int n_lb, cudaStream_t stream) {
    constexpr int D = FTQ_D;
    constexpr int GH = AttnCfg<D>::GH;
    constexpr int page = kPageTokens * (packed_dim(D, BK) + packed_dim(D, BV) + 4);
    constexpr int merge = 4 * GH * (D + 2) * 4;
    constexpr int ring = ((kTileRing * kTilePages * page > merge ? kTileRing * kTilePages * page : merge) + 15) / 16 * 16;
    constexpr int tk = (1 << (2 * BK)) * 128, tv = (1 << (2 * BV)) * 128;
    constexpr int smem = ring + GH * D * 4 + tk;
    constexpr auto kern = attn_split_kernel<D, BK, BV, PAGED>;
    const cudaError_t e = allow_smem<kern>(smem + tv);
    if (e != cudaSuccess) return e;
    const dim3 grid(p.n_chunks, p.Hkv * p.n_hpass, n_lb);
    kern<<<grid, kAttnThreads, smem + (p.shared_table ? 0 : tv), stream>>>(p);
    return cudaGetLastError();
}

template <int BK, bool PAGED>
static cudaError_t by_bv(int bv, const AttnParams& p, int n_lb, cudaStream_t stream) {
    switch (bv) {
        case 2: return run_split<BK, 2, PAGED>(p, n_lb, stream);
        case 3: return run_split<BK, 3, PAGED>(p, n_lb, stream);
        case 4: return run_split<BK, 4, PAGED>(p, n_lb, stream);
    }
    return cudaErrorInvalidValue;
}

template <bool PAGED>
static cudaError_t by_bk(int bk, int bv, const AttnParams& p, int n_lb, cudaStream_t stream) {
    switch (bk) {
        case 2: return by_bv<2, PAGED>(bv, p, n_lb, stream);
        case 3: return by_bv<3, PAGED>(bv, p, n_lb, stream);
        case 4: return by_bv<4, PAGED>(bv, p, n_lb, stream);
    }
    return cudaErrorInvalidValue;
}

cudaError_t FTQ_CAT(launch_attn_split_d, FTQ_D)(int bits_k, int bits_v, bool paged,
                                                const AttnParams& p, int n_lb,
                                                cudaStream_t stream) {
    return paged ? by_bk<true>(bits_k, bits_v, p, n_lb, stream)
                 : by_bk<false>(bits_k, bits_v, p, n_lb, stream);
}

#if defined(FTQ_TEST_WAIT_EXPIRY)
extern "C" int ftq_test_withhold_epoch(int on) {   // (see ftq_attn_flow.cuh)
    return static_cast<int>(cudaMemcpyToSymbol(test_withhold_epoch, &on, sizeof(on)));
}
#endif

template <int BK, int BV, bool SHARED, int NH>
static cudaError_t run_flow(const AttnParams& p_in, cudaStream_t stream) {
    using C = FlowCfg<FTQ_D, BK, BV, NH>;
    static_assert(C::SMEM_BYTES <= C::LIMIT, "shared memory budget");
    constexpr auto kern = attn_flow_kernel<FTQ_D, BK, BV, SHARED, NH, false>;
    cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    AttnParams p = p_in;
    // a share is at least one stage per warp: less would only cut units into more rows to merge
    p.min_share = C::WARPS * C::NP;
    p.B_stride = p_in.B;
    for (p.b0 = 0; p.b0 < p_in.B; p.b0 += kFlowMaxSeqs) {
        p.B = p_in.B - p.b0 < kFlowMaxSeqs ? p_in.B - p.b0 : kFlowMaxSeqs;
        p.seq_lens = p_in.seq_lens + p.b0;
        p.block_table = p_in.block_table + static_cast<int64_t>(p.b0) * p.max_blocks;
        p.n_units = p.n_layers * p.B * p.Hkv;
        // (places, not pages: 164 sequences of 8 tokens, 4 heads of 64, K4V3, took 26 us on the 11 CTAs that their pages fill,
        // 10 on all)
        const int64_t places = (static_cast<int64_t>(p.max_seq) + kPageTokens - 1) / kPageTokens + C::PIECE;
        const int64_t want = (p.n_units * places + p.min_share * C::HALVES - 1) / (p.min_share * C::HALVES);
        const int64_t slots = sm_count();
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(want < 1 ? 1 : want < slots ? want : slots));
        cfg.blockDim = dim3(C::HALVES * C::THREADS);
        cfg.dynamicSmemBytes = C::SMEM_BYTES;
        cfg.stream = stream;
        // (programmatic stream serialisation: the tables are built while the kernel before drains)
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, kern, p);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Clusters of `size` CTAs of the kernel that the device holds at a time (asked once per device and size).
template <auto kern>
static int clusters_at_a_time(int size, int threads, int smem) {
    static std::atomic<int> known[64][3];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const int slot = size == 8 ? 0 : size == 4 ? 1 : 2;   // (a size of one is not asked for)
    if (dev < 64) {
        const int n = known[dev][slot].load(std::memory_order_relaxed);
        if (n) return n - 1;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(size) * 64);
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {static_cast<unsigned>(size), 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        n = 0;
    }
    if (dev < 64) known[dev][slot].store(n + 1, std::memory_order_relaxed);
    return n;
}

// Few units with short contexts (at most one per SM): a cluster of 8, 4, 2 CTAs or one CTA per unit, as many as the device
// holds at a time, whose parts are put together over distributed shared memory.  Rows in the workspace, a counter and
// the rows again are a chain of 5 us at the end of the equal-share kernel, and few long units have many rows; a
// cluster's merge takes 2 us, but leaves SMs idle where the units do not fill them and cannot even out a ragged batch.
// Steps (store included) by clusters : equal shares, parts of 40, 100 and 185 pages: 8 units of 128 coordinates, K4V4,
// in clusters of 8 16.3 : 22.3, 24.7 : 27.2, 37.0 : 30.9 us; 4 units, K3V3 17.4 : 25.6, 26.6 : 36.2, 39.2 : 35.1; 48
// units in clusters of 2 16.5 : 19.1, 24.9 : 24.1, 36.6 : 31.0; 104 units, one CTA each, 16.9 : 19.6, 25.3 : 24.5, 37.0 :
// 31.3, ragged 36.0 : 19.9.  So the lines, in pages of a half's part.  The host knows the longest context, not the others:
// ragged batches (one long sequence, half of them, log-uniform lengths) just below the lines and at 0.4 of them, 8 to 128
// units of four shapes, took 0.09 to 0.89 of the time of the kernel without clusters that was here before.
constexpr int kClusterPages8 = 112, kClusterPages = 72;
// Returns cudaErrorNotSupported where equal shares are the better ones.
template <int BK, int BV, bool SHARED, int NH>
static cudaError_t run_cluster(const AttnParams& p_in, cudaStream_t stream) {
    using C = FlowCfg<FTQ_D, BK, BV, NH, true>;
    static_assert(C::SMEM_BYTES <= C::LIMIT, "shared memory budget");
    constexpr auto kern = attn_flow_kernel<FTQ_D, BK, BV, SHARED, NH, true>;
    const int pages = (p_in.max_seq + kPageTokens - 1) / kPageTokens;
    if (p_in.n_units > sm_count() || pages > kClusterPages8 * 8 * C::HALVES) return cudaErrorNotSupported;
    cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    int size = 8;
    while (size > 1 && clusters_at_a_time<kern>(size, C::HALVES * C::THREADS, C::SMEM_BYTES) < p_in.n_units) size /= 2;
    if (pages > (size == 8 ? kClusterPages8 : kClusterPages) * size * C::HALVES) return cudaErrorNotSupported;
    AttnParams p = p_in;
    p.b0 = 0;
    p.B_stride = p_in.B;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(p.n_units * size));
    cfg.blockDim = dim3(C::HALVES * C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim = {static_cast<unsigned>(size), 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int BK, int BV, bool SHARED, int NH>
static cudaError_t run_mma_nh(const AttnParams& p, cudaStream_t stream) {
    const cudaError_t e = run_cluster<BK, BV, SHARED, NH>(p, stream);
    return e != cudaErrorNotSupported ? e : run_flow<BK, BV, SHARED, NH>(p, stream);
}

template <int BK, int BV, bool SHARED>
static cudaError_t run_mma(const AttnParams& p, cudaStream_t stream) {
    return p.Hq / p.Hkv <= 4 ? run_mma_nh<BK, BV, SHARED, 1>(p, stream)
                             : run_mma_nh<BK, BV, SHARED, 2>(p, stream);
}

// FTQ_ONLY_BITS=<b> (a development aid, never set by the build script) instantiates the
// tensor-core kernels for bits_k = bits_v = b only, which cuts the compile time of an experiment.
template <int BK>
static cudaError_t mma_by_bv(int bv, bool shared_lut, const AttnParams& p, cudaStream_t stream) {
#ifdef FTQ_ONLY_BITS
    if (BK != FTQ_ONLY_BITS || bv != FTQ_ONLY_BITS) return cudaErrorInvalidValue;
    if constexpr (BK == FTQ_ONLY_BITS) {
        return shared_lut ? run_mma<BK, BK, true>(p, stream)
                          : run_mma<BK, BK, false>(p, stream);
    }
#else
    if (shared_lut && bv == BK) return run_mma<BK, BK, true>(p, stream);
    switch (bv) {
        case 2: return run_mma<BK, 2, false>(p, stream);
        case 3: return run_mma<BK, 3, false>(p, stream);
        case 4: return run_mma<BK, 4, false>(p, stream);
    }
#endif
    return cudaErrorInvalidValue;
}

cudaError_t FTQ_CAT(launch_attn_mma_d, FTQ_D)(int bits_k, int bits_v, bool shared_lut,
                                              const AttnParams& p, cudaStream_t stream) {
    switch (bits_k) {
        case 2: return mma_by_bv<2>(bits_v, shared_lut, p, stream);
        case 3: return mma_by_bv<3>(bits_v, shared_lut, p, stream);
        case 4: return mma_by_bv<4>(bits_v, shared_lut, p, stream);
    }
    return cudaErrorInvalidValue;
}

template <typename OT>
static cudaError_t run_merge(const float* partials, void* out, const int32_t* seq_lens, int S, int B, int Hq,
                             int n_chunks, int chunk_tokens, int64_t n_vec, const SignBits& signs,
                             float rsqrt_d, const MergeStatus& status, cudaStream_t stream) {
    // a warp per vector where there are few of them (kWideMerge), an octet where they fill the chip as
    // it is: 128 vectors of 32 chunks 23 -> 4 us with four octets, 8192 vectors of 4 chunks 6 -> 10 us
    const int octets = n_vec <= kWideMerge * sm_count() ? 4 : 1;
    const unsigned grid = static_cast<unsigned>((n_vec * octets + 15) / 16);
    if (n_vec <= 0) return cudaSuccess;
    // (launched while the kernel before drains: it waits for that one's end itself)
    return launch_dependent(octets == 4 ? attn_merge_kernel<FTQ_D, OT, 4> : attn_merge_kernel<FTQ_D, OT, 1>, grid, 128, 0, stream,
                            partials, static_cast<OT*>(out), seq_lens, S, B, Hq, n_chunks, chunk_tokens, n_vec, signs, rsqrt_d, status);
}

cudaError_t FTQ_CAT(launch_attn_merge_d, FTQ_D)(int out_dtype, const float* partials, void* out,
                                                const int32_t* seq_lens, int S, int B, int Hq,
                                                int n_chunks, int chunk_tokens, int64_t n_vec,
                                                const SignBits& signs, float rsqrt_d, const MergeStatus& status,
                                                cudaStream_t stream) {
    switch (out_dtype) {
        case kF32:
            return run_merge<float>(partials, out, seq_lens, S, B, Hq, n_chunks, chunk_tokens, n_vec, signs,
                                    rsqrt_d, status, stream);
        case kF16:
            return run_merge<__half>(partials, out, seq_lens, S, B, Hq, n_chunks, chunk_tokens, n_vec, signs,
                                     rsqrt_d, status, stream);
        case kBF16:
            return run_merge<__nv_bfloat16>(partials, out, seq_lens, S, B, Hq, n_chunks, chunk_tokens, n_vec,
                                            signs, rsqrt_d, status, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ftq
