// Instantiates the split-KV decode attention kernels for one head_dim (FTQ_D).
#include "ftq_attn_flow.cuh"
#include "ftq_attn_stream.cuh"
#include "ftq_launch.h"

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
    constexpr int ring = ((2 * kTilePages * page > merge ? 2 * kTilePages * page : merge) + 15) / 16 * 16;
    constexpr int smem = ring + (GH * D + 2 * kMaxLevels) * 4;
    static_assert(smem <= 48 * 1024, "shared memory budget");
    const dim3 grid(p.n_chunks, p.Hkv * p.n_hpass, n_lb);
    attn_split_kernel<D, BK, BV, PAGED><<<grid, kAttnThreads, smem, stream>>>(p);
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

// The streaming kernel (no CTA-wide barriers, merge included) serves the configurations in
// which it was measured faster than the equal-share one: a 4-bit byte table (one CTA per SM) with
// a GQA group of at most 4 -- 16 warps at head_dim 64 / 128, 12 or 8 at head_dim 256 (16 rings and
// exchange slots do not fit beside the table there).  Measured on B200, streaming against equal
// shares, store included: 777 : 1137 us for the ragged head_dim-256 K4V2 batch, 21.5 : 25.1 us for
// one sequence of 900 tokens, 142 : 141 us for 64 x 8192 tokens of 8 K4V4 heads.
template <int BK, int BV, int NH>
constexpr bool use_stream_kernel() {
    using S = StreamCfg<FTQ_D, BK, BV, NH>;
#if defined(FTQ_NO_STREAM)
    return false;
#elif defined(FTQ_ALL_STREAM)
    return S::FITS;
#else
    return S::FITS && S::BYTE && NH == 1;
#endif
}

template <int BK, int BV, bool SHARED, int NH>
static cudaError_t run_flow(const AttnParams& p_in, cudaStream_t stream) {
    using C = MmaCfg<FTQ_D, BK, BV, NH>;
    static_assert(C::SMEM_BYTES <= C::LIMIT, "shared memory budget");
    constexpr auto kern = attn_flow_kernel<FTQ_D, BK, BV, SHARED, NH>;
    cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    AttnParams p = p_in;
    // a CTA's share is at least one stage per warp: less would only cut units into more rows to merge
    p.min_share = C::WARPS * C::NP;
    p.B_stride = p_in.B;
    for (p.b0 = 0; p.b0 < p_in.B; p.b0 += kFlowMaxSeqs) {
        p.B = p_in.B - p.b0 < kFlowMaxSeqs ? p_in.B - p.b0 : kFlowMaxSeqs;
        p.seq_lens = p_in.seq_lens + p.b0;
        p.block_table = p_in.block_table + static_cast<int64_t>(p.b0) * p.max_blocks;
        p.n_units = p.n_layers * p.B * p.Hkv;
        const int64_t most = static_cast<int64_t>(p.n_units) * ((static_cast<int64_t>(p.max_seq) + kPageTokens - 1) / kPageTokens);
        const int64_t want = (most + p.min_share - 1) / p.min_share;
        const int64_t slots = static_cast<int64_t>(sm_count()) * C::CTAS_PER_SM;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(want < 1 ? 1 : want < slots ? want : slots));
        cfg.blockDim = dim3(C::THREADS);
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

template <int BK, int BV, bool SHARED, int NH>
static cudaError_t run_mma_nh(const AttnParams& p, cudaStream_t stream) {
    constexpr int D = FTQ_D;
    if constexpr (use_stream_kernel<BK, BV, NH>()) {
        using S = StreamCfg<D, BK, BV, NH>;
        constexpr auto kern = attn_stream_kernel<D, BK, BV, SHARED, NH>;
        cudaError_t e = allow_smem<kern>(S::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        const int64_t items = p.split.total_items;
        const int64_t slots = static_cast<int64_t>(sm_count()) * S::CTAS_PER_SM;
        const unsigned grid = static_cast<unsigned>(items < slots ? items : slots);
        // One node per call: the kernel clears its own counters.  Programmatic stream
        // serialisation lets the set-up of this launch (tables in shared memory) run while the
        // kernel before it in the stream drains; the kernel waits for that kernel's completion
        // (griddepcontrol.wait) before it touches anything in global memory.
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(S::THREADS);
        cfg.dynamicSmemBytes = S::SMEM_BYTES;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kern, p, static_cast<int>(items));
    } else {
        return run_flow<BK, BV, SHARED, NH>(p, stream);
    }
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

// CTAs per SM of the streaming kernel where launch_attn_mma picks it for this configuration, 0
// where it picks the equal-share kernel (which needs no plan of the host)
template <int BK, int BV, int NH>
static constexpr int stream_ctas() {
    return use_stream_kernel<BK, BV, NH>() ? StreamCfg<FTQ_D, BK, BV, NH>::CTAS_PER_SM : 0;
}
template <int BK>
static int stream_ctas_by_bv(int bv, int nh) {
#ifdef FTQ_ONLY_BITS
    if (BK != FTQ_ONLY_BITS || bv != FTQ_ONLY_BITS) return 0;
    return nh == 1 ? stream_ctas<BK, BK, 1>() : stream_ctas<BK, BK, 2>();
#else
    switch (bv) {
        case 2: return nh == 1 ? stream_ctas<BK, 2, 1>() : stream_ctas<BK, 2, 2>();
        case 3: return nh == 1 ? stream_ctas<BK, 3, 1>() : stream_ctas<BK, 3, 2>();
        case 4: return nh == 1 ? stream_ctas<BK, 4, 1>() : stream_ctas<BK, 4, 2>();
    }
    return 0;
#endif
}
int FTQ_CAT(attn_mma_stream_ctas_d, FTQ_D)(int bits_k, int bits_v, int group) {
    const int nh = group <= 4 ? 1 : 2;
    switch (bits_k) {
        case 2: return stream_ctas_by_bv<2>(bits_v, nh);
        case 3: return stream_ctas_by_bv<3>(bits_v, nh);
        case 4: return stream_ctas_by_bv<4>(bits_v, nh);
    }
    return 0;
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
