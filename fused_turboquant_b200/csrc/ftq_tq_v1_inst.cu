// Instantiates the vLLM-v1 slot-format kernels for one head_dim (FTQ_D).  FTQ_TQ_PART selects
// what this object holds, so that the parts compile in parallel: 0 = the store kernels, 1 = the decode
// kernels (fp32 split, tensor-core split, merge), 2 = decode by shares of pages and its merge; undefined = all.
#include "ftq_launch.h"
#include "ftq_tq_v1.cuh"
#include "ftq_tq_v1_launch.h"
#if !defined(FTQ_TQ_PART) || FTQ_TQ_PART == 0
#define FTQ_TQ_STORE 1
#endif
#if !defined(FTQ_TQ_PART) || FTQ_TQ_PART == 1
#define FTQ_TQ_DECODE 1
#endif
#if !defined(FTQ_TQ_PART) || FTQ_TQ_PART == 2
#define FTQ_TQ_FLOW 1
#endif
#ifdef FTQ_TQ_STORE
#include "ftq_tq_v1_store2.cuh"
#endif
#if FTQ_D != 256 && defined(FTQ_TQ_FLOW)
#include "ftq_tq_v1_flow.cuh"
#include "ftq_tq_v1_fp8.cuh"
#endif
#if FTQ_D != 256 && defined(FTQ_TQ_DECODE)
#include "ftq_tq_v1_fp8.cuh"
#include "ftq_tq_v1_mma.cuh"
#endif

#ifndef FTQ_D
#error "compile with -DFTQ_D=64, 128 or 256"
#endif
#define FTQ_CAT2(a, b) a##b
#define FTQ_CAT(a, b) FTQ_CAT2(a, b)

namespace ftq {

#ifdef FTQ_TQ_STORE
template <int KB, int VB, typename T, bool K8M>
static cudaError_t store_run(const TqStoreParams& p, int value_mode, int64_t n_vec,
                             const TqTable<K8M>& t8, cudaStream_t stream) {
    const int64_t want = (n_vec + 31) / 32;  // 8 warps x 4 vectors per CTA pass
    const int layers = value_mode >> 8;      // (the launcher packs the layer count above the flags)
    const int64_t cap = (static_cast<int64_t>(sm_count()) * 8 + layers - 1) / layers;
    const dim3 gx(static_cast<unsigned>(want < 1 ? 1 : (want < cap ? want : cap)), layers);
    const bool rotate_v = (value_mode & kTqRotateValues) != 0;
    if constexpr (VB == 4 && KB != 8) {
        if (value_mode & kTqLloydMaxValues) {
            if (rotate_v) tq_store_kernel<FTQ_D, KB, VB, T, true, true><<<gx, 256, 0, stream>>>(p, n_vec, t8);
            else tq_store_kernel<FTQ_D, KB, VB, T, false, true><<<gx, 256, 0, stream>>>(p, n_vec, t8);
            return cudaGetLastError();
        }
    }
    if constexpr (VB != 8) {
        if (rotate_v) {
            tq_store_kernel<FTQ_D, KB, VB, T, true, false, K8M><<<gx, 256, 0, stream>>>(p, n_vec, t8);
            return cudaGetLastError();
        }
    } else if (rotate_v) {
        return cudaErrorInvalidValue;  // 8-bit values are rotated by the caller
    }
    tq_store_kernel<FTQ_D, KB, VB, T, false, false, K8M><<<gx, 256, 0, stream>>>(p, n_vec, t8);
    return cudaGetLastError();
}

template <int KB, int VB, bool K8M>
static cudaError_t store_by_dtype(int dtype, const TqStoreParams& p, int vmode, int64_t n_vec,
                                  const TqTable<K8M>& t8, cudaStream_t s) {
    switch (dtype) {
        case kF32: return store_run<KB, VB, float, K8M>(p, vmode, n_vec, t8, s);
        case kF16: return store_run<KB, VB, __half, K8M>(p, vmode, n_vec, t8, s);
        case kBF16: return store_run<KB, VB, __nv_bfloat16, K8M>(p, vmode, n_vec, t8, s);
    }
    return cudaErrorInvalidValue;
}

template <int KB, bool K8M = false>
static cudaError_t store_by_vb(int vb, int dtype, const TqStoreParams& p, int vmode, int64_t n_vec,
                               const TqTable<K8M>& t8, cudaStream_t s) {
    switch (vb) {
        case 1: return store_by_dtype<KB, 1, K8M>(dtype, p, vmode, n_vec, t8, s);
        case 2: return store_by_dtype<KB, 2, K8M>(dtype, p, vmode, n_vec, t8, s);
        case 3: return store_by_dtype<KB, 3, K8M>(dtype, p, vmode, n_vec, t8, s);
        case 4: return store_by_dtype<KB, 4, K8M>(dtype, p, vmode, n_vec, t8, s);
        case 8: return store_by_dtype<KB, 8, K8M>(dtype, p, vmode, n_vec, t8, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t FTQ_CAT(launch_tq_store_d, FTQ_D)(int kb, int vb, int dtype, const TqStoreParams& p,
                                             int value_mode, int64_t n_vec, const TqTable256* mid8,
                                             cudaStream_t stream) {
    const TqNoTable none{};
    switch (kb) {
        case 1: return store_by_vb<1>(vb, dtype, p, value_mode, n_vec, none, stream);
        case 2: return store_by_vb<2>(vb, dtype, p, value_mode, n_vec, none, stream);
        case 3: return store_by_vb<3>(vb, dtype, p, value_mode, n_vec, none, stream);
        case 4: return store_by_vb<4>(vb, dtype, p, value_mode, n_vec, none, stream);
        case 8:   // 8-bit Lloyd-Max codes with a table, FP8 keys without
            return mid8 ? store_by_vb<8, true>(vb, dtype, p, value_mode, n_vec, *mid8, stream)
                        : store_by_vb<8>(vb, dtype, p, value_mode, n_vec, none, stream);
    }
    return cudaErrorInvalidValue;
}

template <int KB, int VB, typename T, bool ROTV>
static cudaError_t store2_run(const TqStore2Params& p, int n_layers, cudaStream_t stream) {
    constexpr int threads = tq_store2_threads(FTQ_D), smem = encode2_smem_bytes(FTQ_D, threads / 32);
    constexpr auto kern = tq_store2_kernel<FTQ_D, KB, VB, T, ROTV>;
    const cudaError_t e = allow_smem<kern>(smem);
    if (e != cudaSuccess) return e;
    // one wave of CTAs, shared among the layers
    const int64_t want = (p.n_vec + threads / 4 - 1) / (threads / 4);
    const int64_t wave = static_cast<int64_t>(sm_count()) * (512 / threads);
    const int64_t cap = (wave + n_layers - 1) / n_layers;
    return launch_dependent(kern, dim3(static_cast<unsigned>(want < cap ? want : cap), n_layers), threads, smem, stream, p);
}
template <int KB, int VB>
static cudaError_t store2_by_type(int dtype, const TqStore2Params& p, bool rot, int n_layers, cudaStream_t s) {
    if (dtype == kBF16)
        return rot ? store2_run<KB, VB, __nv_bfloat16, true>(p, n_layers, s) : store2_run<KB, VB, __nv_bfloat16, false>(p, n_layers, s);
    if (dtype == kF16) return rot ? store2_run<KB, VB, __half, true>(p, n_layers, s) : store2_run<KB, VB, __half, false>(p, n_layers, s);
    return cudaErrorInvalidValue;
}
template <int KB>
static cudaError_t store2_by_vb(int vb, int dtype, const TqStore2Params& p, bool rot, int n_layers, cudaStream_t s) {
    return vb == 3 ? store2_by_type<KB, 3>(dtype, p, rot, n_layers, s)
           : vb == 4 ? store2_by_type<KB, 4>(dtype, p, rot, n_layers, s) : cudaErrorInvalidValue;
}
cudaError_t FTQ_CAT(launch_tq_store2_d, FTQ_D)(int kb, int vb, int dtype, const TqStoreParams& sp, bool rotate_v,
                                              int64_t n_vec, int n_layers, cudaStream_t stream) {
    TqStore2Params p{};
    p.s = sp;
    p.n_vec = static_cast<uint32_t>(n_vec);
    switch (kb) {
        case 3: return store2_by_vb<3>(vb, dtype, p, rotate_v, n_layers, stream);
        case 4: return store2_by_vb<4>(vb, dtype, p, rotate_v, n_layers, stream);
        case 8: return store2_by_vb<8>(vb, dtype, p, rotate_v, n_layers, stream);
    }
    return cudaErrorInvalidValue;
}

#endif  // FTQ_TQ_STORE

#ifdef FTQ_TQ_DECODE
template <int KB, int VB, bool K8M>
static cudaError_t split_run(const TqDecodeParams& p, const TqTable<K8M>& t8, cudaStream_t stream) {
    constexpr int smem = tq_split_smem_bytes<FTQ_D>(KB, VB, K8M);
    static_assert(smem <= 48 * 1024, "tile does not fit the default shared-memory carve-out");
    const dim3 grid(p.splits, p.Hkv * p.n_hpass, p.B);
    tq_split_kernel<FTQ_D, KB, VB, K8M><<<grid, kAttnThreads, smem, stream>>>(p, t8);
    return cudaGetLastError();
}

template <int KB, bool K8M = false>
static cudaError_t split_by_vb(int vb, const TqDecodeParams& p, const TqTable<K8M>& t8,
                               cudaStream_t s) {
    switch (vb) {
        case 1: return split_run<KB, 1, K8M>(p, t8, s);
        case 2: return split_run<KB, 2, K8M>(p, t8, s);
        case 3: return split_run<KB, 3, K8M>(p, t8, s);
        case 4: return split_run<KB, 4, K8M>(p, t8, s);
        case 8: return split_run<KB, 8, K8M>(p, t8, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t FTQ_CAT(launch_tq_split_d, FTQ_D)(int kb, int vb, const TqDecodeParams& p,
                                             const TqTable256* cent8, cudaStream_t stream) {
    const TqNoTable none{};
    switch (kb) {
        case 1: return split_by_vb<1>(vb, p, none, stream);
        case 2: return split_by_vb<2>(vb, p, none, stream);
        case 3: return split_by_vb<3>(vb, p, none, stream);
        case 4: return split_by_vb<4>(vb, p, none, stream);
        case 8:   // 8-bit Lloyd-Max codes with a table, FP8 keys without
            return cent8 ? split_by_vb<8, true>(vb, p, *cent8, stream)
                         : split_by_vb<8>(vb, p, none, stream);
    }
    return cudaErrorInvalidValue;
}

#if FTQ_D != 256
template <int KB, int VB, int NH>
static cudaError_t mma_run(const TqDecodeParams& p, int n_items, cudaStream_t stream) {
    using C = TqMmaCfg<FTQ_D, KB, VB, NH>;
    static_assert(C::SMEM_BYTES <= 227 * 1024, "shared memory budget");
    constexpr auto kern = tq_mma_kernel<FTQ_D, KB, VB, NH>;
    cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t slots = static_cast<int64_t>(sm_count()) * C::CTAS_PER_SM;
    const unsigned gx = static_cast<unsigned>(n_items < slots ? n_items : slots);
    kern<<<gx, C::THREADS, C::SMEM_BYTES, stream>>>(p, n_items);
    return cudaGetLastError();
}

template <int KB, int VB>
static cudaError_t mma_by_nh(int nh, const TqDecodeParams& p, int n_items, cudaStream_t s) {
    return nh == 1 ? mma_run<KB, VB, 1>(p, n_items, s) : mma_run<KB, VB, 2>(p, n_items, s);
}

template <int KB>
static cudaError_t mma_by_vb(int vb, int nh, const TqDecodeParams& p, int n_items, cudaStream_t s) {
    switch (vb) {
        case 2: return mma_by_nh<KB, 2>(nh, p, n_items, s);
        case 3: return mma_by_nh<KB, 3>(nh, p, n_items, s);
        case 4: return mma_by_nh<KB, 4>(nh, p, n_items, s);
    }
    return cudaErrorInvalidValue;
}
#endif

template <int VB, int NH>
static cudaError_t fp8_run(const TqDecodeParams& p, int n_items, cudaStream_t stream) {
#if FTQ_D != 256
    using C = TqFp8Cfg<FTQ_D, VB, NH>;
    constexpr auto kern = tq_fp8_kernel<FTQ_D, VB, NH>;
    const cudaError_t e = allow_smem<kern>(C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t slots = static_cast<int64_t>(sm_count()) * 2;
    const unsigned gx = static_cast<unsigned>(n_items < slots ? n_items : slots);
    kern<<<gx, C::THREADS, C::SMEM_BYTES, stream>>>(p, n_items);
    return cudaGetLastError();
#else
    return cudaErrorInvalidValue;
#endif
}
// Tensor-core stage 1 for FP8 keys (16-bit queries, GQA group <= 8, 2- to 4-bit values, head_dim 64 /
// 128, 4-byte aligned slots).
cudaError_t FTQ_CAT(launch_tq_fp8_d, FTQ_D)(int vb, int nh, const TqDecodeParams& p, int n_items,
                                           cudaStream_t stream) {
    switch (vb) {
        case 2: return nh == 1 ? fp8_run<2, 1>(p, n_items, stream) : fp8_run<2, 2>(p, n_items, stream);
        case 3: return nh == 1 ? fp8_run<3, 1>(p, n_items, stream) : fp8_run<3, 2>(p, n_items, stream);
        case 4: return nh == 1 ? fp8_run<4, 1>(p, n_items, stream) : fp8_run<4, 2>(p, n_items, stream);
    }
    return cudaErrorInvalidValue;
}

// Tensor-core stage 1 (16-bit queries, GQA group <= 8, value_bits != 8, head_dim 64 / 128).
cudaError_t FTQ_CAT(launch_tq_mma_d, FTQ_D)(int kb, int vb, int nh, const TqDecodeParams& p,
                                           int n_items, cudaStream_t stream) {
#if FTQ_D != 256
    switch (kb) {
        case 2: return mma_by_vb<2>(vb, nh, p, n_items, stream);
        case 3: return mma_by_vb<3>(vb, nh, p, n_items, stream);
        case 4: return mma_by_vb<4>(vb, nh, p, n_items, stream);
    }
#endif
    return cudaErrorInvalidValue;
}

template <typename OT>
static cudaError_t run_tq_merge(const TqMergeParams& p, cudaStream_t stream) {
    // (as in the page-layout merge: a warp per row where there are few of them)
    if (p.n_rows <= 0) return cudaSuccess;
    const int octets = p.n_rows <= kWideMerge * sm_count() ? 4 : 1;
    const unsigned grid = static_cast<unsigned>((p.n_rows * octets + 15) / 16);
    if (octets == 4) tq_merge_kernel<FTQ_D, OT, 4><<<grid, 128, 0, stream>>>(p);
    else tq_merge_kernel<FTQ_D, OT, 1><<<grid, 128, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t FTQ_CAT(launch_tq_merge_d, FTQ_D)(int out_dtype, const TqMergeParams& p,
                                             cudaStream_t stream) {
    switch (out_dtype) {
        case kF32: return run_tq_merge<float>(p, stream);
        case kF16: return run_tq_merge<__half>(p, stream);
        case kBF16: return run_tq_merge<__nv_bfloat16>(p, stream);
    }
    return cudaErrorInvalidValue;
}

#endif  // FTQ_TQ_DECODE

#ifdef FTQ_TQ_FLOW
#if FTQ_D != 256
template <class Engine>
static cudaError_t flow_run(const TqFlowParams& p, cudaStream_t stream) {
    constexpr auto kern = tq_flow_kernel<Engine>;
    const cudaError_t e = allow_smem<kern>(kTqFlowSmem);
    if (e != cudaSuccess) return e;
    // (its set-up, 64 KB of tables, overlaps the tail of the kernel before it)
    return launch_dependent(kern, static_cast<unsigned>(sm_count()), kTqFlowThreads, kTqFlowSmem, stream, p);
}
template <int KB, int VB, int NH>
static cudaError_t flow_engine(const TqFlowParams& p, cudaStream_t s) {
    if constexpr (KB != 8) return flow_run<TqCodes<FTQ_D, KB, VB, NH>>(p, s);
    else if constexpr (kTqFlowFp8<FTQ_D, NH>) return flow_run<TqFp8<FTQ_D, VB, NH, false>>(p, s);
    else return cudaErrorInvalidValue;
}
template <int KB, int VB>
static cudaError_t flow_by_nh(int nh, const TqFlowParams& p, cudaStream_t s) {
    return nh == 1 ? flow_engine<KB, VB, 1>(p, s) : flow_engine<KB, VB, 2>(p, s);
}
template <int KB>
static cudaError_t flow_by_vb(int vb, int nh, const TqFlowParams& p, cudaStream_t s) {
    switch (vb) {
        case 2: return flow_by_nh<KB, 2>(nh, p, s);
        case 3: return flow_by_nh<KB, 3>(nh, p, s);
        case 4: return flow_by_nh<KB, 4>(nh, p, s);
    }
    return cudaErrorInvalidValue;
}
// (launched while stage 1 drains: it waits for stage 1's end itself)
template <typename OT>
static cudaError_t join_run(const TqJoinParams& p, cudaStream_t stream) {
    return launch_dependent(tq_join_kernel<FTQ_D, OT>, static_cast<unsigned>((p.m.n_rows + 1) / 2), 128, 0, stream, p);
}
#endif
// FTQ_ONLY_BITS=<b>: key and value codes of b bits only (the wait-expiry test library)
cudaError_t FTQ_CAT(launch_tq_flow_d, FTQ_D)(int kb, int vb, int nh, const TqFlowParams& p, cudaStream_t stream) {
#if defined(FTQ_ONLY_BITS)
    if (kb == FTQ_ONLY_BITS && vb == FTQ_ONLY_BITS) return flow_by_nh<FTQ_ONLY_BITS, FTQ_ONLY_BITS>(nh, p, stream);
#elif FTQ_D != 256
    switch (kb) {
        case 2: return flow_by_vb<2>(vb, nh, p, stream);
        case 3: return flow_by_vb<3>(vb, nh, p, stream);
        case 4: return flow_by_vb<4>(vb, nh, p, stream);
        case 8: return flow_by_vb<8>(vb, nh, p, stream);   // FP8 keys
    }
#endif
    return cudaErrorInvalidValue;
}
cudaError_t FTQ_CAT(launch_tq_join_d, FTQ_D)(int out_dtype, const TqJoinParams& p, cudaStream_t stream) {
#if FTQ_D != 256
    switch (out_dtype) {
        case kF32: return join_run<float>(p, stream);
        case kF16: return join_run<__half>(p, stream);
        case kBF16: return join_run<__nv_bfloat16>(p, stream);
    }
#endif
    return cudaErrorInvalidValue;
}
#endif  // FTQ_TQ_FLOW

}  // namespace ftq
