// Host-side launchers, one translation unit per head_dim (compiled with
// -DFTQ_D=64|128|256) so the template instantiations build in parallel.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <utility>

#include "ftq_attn_chunk.cuh"
#include "ftq_encode2.cuh"

namespace ftq {

// which kernel encodes: a warp per vector; two vectors per octet and a quantiser table; an octet per vector
enum class Encode { kFew, kTable, kAnyCodebook };

#define FTQ_DECLARE_LAUNCHERS(DD)                                                              \
    cudaError_t launch_encode_d##DD(int dtype, const EncodeJobs& jobs, int n_jobs, Encode kind, \
                                    int n_layers, cudaStream_t stream);                         \
    cudaError_t launch_attn_split_d##DD(int bits_k, int bits_v, bool paged, const AttnParams& p, \
                                        int n_lb, cudaStream_t stream);                         \
    cudaError_t launch_attn_mma_d##DD(int bits_k, int bits_v, bool shared_lut, const AttnParams& p, \
                                      cudaStream_t stream);                                   \
    cudaError_t launch_attn_chunk_d##DD(int bits_k, int bits_v, const ChunkAttnParams& p, int B, \
                                        cudaStream_t stream);                                   \
    cudaError_t launch_attn_merge_d##DD(int out_dtype, const float* partials, void* out,        \
                                        const int32_t* seq_lens, int S, int B, int Hq,          \
                                        int n_chunks, int chunk_tokens, int64_t n_vec,          \
                                        const SignBits& signs, float rsqrt_d,               \
                                        const MergeStatus& status, cudaStream_t stream);

FTQ_DECLARE_LAUNCHERS(64)
FTQ_DECLARE_LAUNCHERS(128)
FTQ_DECLARE_LAUNCHERS(256)

// number of SMs of the current device (cached per device)
int sm_count();

namespace {   // (internal linkage: every library that holds these kernels keeps its own record)
// Allows `kern` more than 48 KB of dynamic shared memory, once per device (the attribute call costs
// the host about half a microsecond, which every launch used to pay).
template <auto kern>
inline cudaError_t allow_smem(int bytes) {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? 1ull << dev : 0;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    const cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (r == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return r;
}
// Launches a kernel that may start its set-up while the kernel before it drains (programmatic stream serialisation).
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, int threads, int smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}
}  // namespace

}  // namespace ftq
