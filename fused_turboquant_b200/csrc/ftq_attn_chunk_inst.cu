// Instantiates the chunk attention kernel for one head_dim (FTQ_D).
#include "ftq_attn_chunk.cuh"
#include "ftq_launch.h"

#ifndef FTQ_D
#error "compile with -DFTQ_D=64, 128 or 256"
#endif
#define FTQ_CAT2(a, b) a##b
#define FTQ_CAT(a, b) FTQ_CAT2(a, b)

namespace ftq {

template <int BK, int BV>
static cudaError_t run_chunk(const ChunkAttnParams& p, int B, cudaStream_t stream) {
    using C = ChunkCfg<FTQ_D, BK, BV>;
    constexpr auto kern = attn_chunk_kernel<FTQ_D, BK, BV>;
    const cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int rows = p.q_len * (p.Hq / p.Hkv), tiles = (rows + 128 * C::SLOTS - 1) / (128 * C::SLOTS);
    // (the tables are built while the kernel before drains)
    return launch_dependent(kern, dim3(p.splits, p.Hkv * tiles, B), C::THREADS, C::SMEM_BYTES, stream, p);
}

// FTQ_ONLY_BITS=<b>: bits_k = bits_v = b only (the wait-expiry test library)
template <int BK>
static cudaError_t chunk_by_bv(int bv, const ChunkAttnParams& p, int B, cudaStream_t stream) {
#ifdef FTQ_ONLY_BITS
    if constexpr (BK == FTQ_ONLY_BITS) {
        if (bv == BK) return run_chunk<BK, BK>(p, B, stream);
    }
#else
    switch (bv) {
        case 2: return run_chunk<BK, 2>(p, B, stream);
        case 3: return run_chunk<BK, 3>(p, B, stream);
        case 4: return run_chunk<BK, 4>(p, B, stream);
    }
#endif
    return cudaErrorInvalidValue;
}

cudaError_t FTQ_CAT(launch_attn_chunk_d, FTQ_D)(int bits_k, int bits_v, const ChunkAttnParams& p, int B,
                                                cudaStream_t stream) {
    switch (bits_k) {
        case 2: return chunk_by_bv<2>(bits_v, p, B, stream);
        case 3: return chunk_by_bv<3>(bits_v, p, B, stream);
        case 4: return chunk_by_bv<4>(bits_v, p, B, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ftq
