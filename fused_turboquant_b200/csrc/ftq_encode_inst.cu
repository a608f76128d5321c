// Instantiates the fused encode kernel for one head_dim (FTQ_D).
#include "ftq_launch.h"

#ifndef FTQ_D
#error "compile with -DFTQ_D=64, 128 or 256"
#endif
#define FTQ_CAT2(a, b) a##b
#define FTQ_CAT(a, b) FTQ_CAT2(a, b)

namespace ftq {

template <typename T>
static cudaError_t run(EncodeJobs jobs, int n_jobs, Encode kind, int n_layers, cudaStream_t stream) {
    const int64_t n = jobs.n_vec;
    if (kind == Encode::kTable) {
        // 16 warps per SM: two CTAs of 8 warps, or one of 16 where two transpose areas would not
        // fit next to two copies of the quantiser table (head_dim 256); a warp pass = 8 vectors.
        // Persistent: the jobs share one wave of CTAs, a job's layers share its part of them.
        constexpr int threads = encode2_threads(FTQ_D);
        constexpr int smem = encode2_smem_bytes(FTQ_D, threads / 32);
        constexpr auto one = encode2_kernel<FTQ_D, false, T>, many = encode2_kernel<FTQ_D, true, T>;
        const cudaError_t e = n_layers > 1 ? allow_smem<many>(smem) : allow_smem<one>(smem);
        if (e != cudaSuccess) return e;
        const int64_t want = ((n + 7) / 8 * n_layers + threads / 32 - 1) / (threads / 32);
        const int64_t cap = static_cast<int64_t>(sm_count()) * (512 / threads) / n_jobs;
        const dim3 grid(static_cast<unsigned>(want < cap ? want : cap), 1, n_jobs);
        jobs.n_layers = n_layers;
        return launch_dependent(n_layers > 1 ? many : one, grid, threads, smem, stream, jobs);
    }
    if (kind == Encode::kAnyCodebook) {
        constexpr int threads = 256;                   // 8 warps, four vectors each
        const int64_t want = (n + threads / 8 - 1) / (threads / 8);
        const int64_t cap = static_cast<int64_t>(sm_count()) * 8;
        const dim3 grid(static_cast<unsigned>(want < cap ? want : cap), n_layers, n_jobs);
        return launch_dependent(encode_octet_kernel<FTQ_D, T>, grid, threads, 0, stream, jobs);
    }
    constexpr int threads = 128;                       // 4 warps, a vector each
    const int64_t want = (n + threads / 32 - 1) / (threads / 32);
    const int64_t cap = static_cast<int64_t>(sm_count()) * 64;
    const dim3 grid(static_cast<unsigned>(want < cap ? want : cap), n_layers, n_jobs);
    // A paged store is launched while the attention of the step before drains.  Shared memory that the kernel does not use
    // keeps its CTAs from filling the first SMs that are free (many to an SM, they would wait there and then be all
    // of the work of a few SMs): as many fit an SM as there are for each.  Step of 16 x 4000 tokens ragged, 8 KV heads of 128,
    // groups of eight 79.8 -> 77.5 us, 64 x 4000 92.3 -> 90.5, of 256 166.1 -> 161.9.
    int smem = 0;
    const int64_t per_sm = (static_cast<int64_t>(grid.x) * n_layers * n_jobs + sm_count() - 1) / sm_count();
    if (n_jobs > 1 && per_sm <= 8) {
        constexpr auto kern = encode_kernel<FTQ_D, T>;
        constexpr int room = 220 * 1024;
        const cudaError_t e = allow_smem<kern>(room);
        if (e != cudaSuccess) return e;
        smem = room / static_cast<int>(per_sm) - 1024;
    }
    return launch_dependent(encode_kernel<FTQ_D, T>, grid, threads, smem, stream, jobs);
}

cudaError_t FTQ_CAT(launch_encode_d, FTQ_D)(int dtype, const EncodeJobs& jobs, int n_jobs, Encode kind,
                                            int n_layers, cudaStream_t stream) {
    switch (dtype) {
        case kF32: return run<float>(jobs, n_jobs, kind, n_layers, stream);
        case kF16: return run<__half>(jobs, n_jobs, kind, n_layers, stream);
        case kBF16: return run<__nv_bfloat16>(jobs, n_jobs, kind, n_layers, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace ftq
