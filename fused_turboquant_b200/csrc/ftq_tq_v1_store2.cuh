// vLLM-v1 slot format, store of many vectors: the bytes of tq_store_kernel (ftq_tq_v1.cuh; the reference's
// vllm_plugin/triton_inkernel_store.py:365-440 and 39-330) with the instruction count of the page-layout
// encoder (ftq_encode2.cuh).
//
// tq_store_kernel issues some 59 instructions per coordinate (15-way midpoint search by selects, scalar
// butterflies with a shuffle per lane bit, two IEEE divisions), which bounds it: 16384 tokens of 8 heads of 128,
// 4-bit keys and rotated 4-bit values in bf16, took 70 us.  This one issues 23 and takes 38.  Here a lane carries TWO
// vectors in packed fp32 pairs (each half an ordinary IEEE operation, in the same order), the transposition goes through shared memory,
// and
//  * x / den is q = x r (r the correctly rounded reciprocal) corrected twice with exact FMA residuals, which is
//    the correctly rounded quotient as long as nothing underflows on the way;
//  * code = #{midpoints <= y} comes out of one table look-up: a cell of [-1, 1] holds at most one midpoint m, and
//    [m > y] is a saturating FMA;
//  * value codes are floor(q + 0.5) by one addition of 2^23 rounded down, shifted into place by an integer
//    multiply-add.
// What that arithmetic does not cover -- a norm or value scale that is not finite or above 2^20 / 2^100, non-zero
// key elements below 2^-40 (residuals and differences could underflow), with FP8 keys elements equal to -0 (the
// corrected quotient is +0) -- sends the warp's eight vectors through tq_store_octets, the other kernel's code.
// Squares of 16-bit inputs are exact in fp32, so that summing them by FMAs rounds like adding them.
#pragma once

#include "ftq_tq_v1.cuh"

namespace ftq {

struct TqStore2Params {
    TqStoreParams s;
    uint32_t n_vec;       // vectors of K (and of V) per layer, below 2^31
};

__host__ __device__ constexpr int tq_store2_threads(int D) { return D >= 256 ? 512 : 256; }

__device__ __forceinline__ u64 add2_down(u64 a, u64 b) {   // rounded towards minus infinity
    u64 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Which words hold a non-zero element of magnitude below `limit` (or, with NEG0, -0): running minimum over the
// 16-bit halves, to be compared with limit - 1.
template <bool NEG0>
__device__ __forceinline__ uint32_t small_min(uint32_t w, uint32_t m) {
    if constexpr (NEG0) {   // negative numbers from -0 on are 0, 1, ...; positive ones from the smallest on too
        m = __viaddmin_u16x2(w, 0x80008000u, m);
        return __viaddmin_u16x2(w, 0xffffffffu, m);
    } else {
        return __viaddmin_u16x2(w & 0x7fff7fffu, 0xffffffffu, m);
    }
}

template <typename T> struct Pair16;   // two 16-bit values of T
template <> struct Pair16<__half> {
    using type = __half2;
    static __device__ __forceinline__ type round(float a, float b) { return __floats2half2_rn(a, b); }
    static constexpr uint32_t kTiny = 0u;          // no non-zero fp16 is below 2^-40
};
template <> struct Pair16<__nv_bfloat16> {
    using type = __nv_bfloat162;
    static __device__ __forceinline__ type round(float a, float b) { return __floats2bfloat162_rn(a, b); }
    static constexpr uint32_t kTiny = (127 - 40) << 7;   // 2^-40
};
template <typename T>
__device__ __forceinline__ float2 widen_pair(uint32_t w) {
    if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&w));
    else return make_float2(bf16_lo(w), bf16_hi(w));
}

// Words of a row of BITS-bit codes at `dst` (nullptr: nowhere): 4-bit codes one word per lane, 3-bit ones 24-bit groups
// regrouped into six words.
template <int BITS, int NCH>
__device__ __forceinline__ void tq_emit_runs(const uint32_t (&w)[NCH], uint8_t* dst, int t) {
#pragma unroll
    for (int i = 0; i < NCH; i++) {
        if constexpr (BITS == 3) {
            const int g0 = (4 * t) / 3;
            const uint32_t lo = __shfl_sync(0xffffffffu, w[i], g0, 8);
            const uint32_t hi = __shfl_sync(0xffffffffu, w[i], g0 + 1, 8);
            const uint64_t cat = (static_cast<uint64_t>(hi) << 24) | lo;
            if (dst && t < 6) store_u32_as_halves(dst + 4 * (6 * i + t), static_cast<uint32_t>(cat >> (8 * ((4 * t) % 3))));
        } else {
            if (dst) store_u32_as_halves(dst + 4 * (t + 8 * i), w[i]);
        }
    }
}
// The same for codes of the coordinates l + 8 k, packed eight to a word.
template <int BITS, int NCH>
__device__ __forceinline__ void tq_emit_columns(uint32_t (&w)[NCH], uint8_t* dst, int t, const TransposeConsts<BITS>& tc) {
#pragma unroll
    for (int i = 0; i < NCH; i++) w[i] = octet_transpose_items<BITS>(w[i], tc);
    tq_emit_runs<BITS, NCH>(w, dst, t);
}

// (not inlined: hardly ever taken)
template <int D, int KB, int VB, typename T, bool ROTV>
__device__ __noinline__ void tq_store2_plain(const TqStoreParams& p, int64_t n_vec, int64_t base, int lane) {
    tq_store_octets<D, KB, VB, T, ROTV, false, false>(p, n_vec, base, 4, base + 8, lane, nullptr);
}

template <int D, int KB, int VB, typename T, bool ROTV>
__global__ void __launch_bounds__(tq_store2_threads(D), 512 / tq_store2_threads(D))
tq_store2_kernel(const __grid_constant__ TqStore2Params pp) {
    static_assert(sizeof(T) == 2 && (KB == 8 || KB == 3 || KB == 4) && (VB == 3 || VB == 4), "");
    const TqStoreParams& p = pp.s;
    constexpr int E = D / kOctet, NCH = E / 8;
    constexpr bool KFP8 = KB == 8;
    constexpr int MSE = D * KB / 8, KPS = MSE + (KFP8 ? 0 : 2), VDB = tq_value_bytes(D, VB);
    constexpr int KT = KFP8 ? 4 : KB;
    constexpr int SLOT = encode2_slot_floats(D);
    constexpr int CPF = 24 / KT, FPW = (8 + CPF - 1) / CPF;   // codes per fp32 accumulator, accumulators per word
    constexpr float kVMax = static_cast<float>((1 << VB) - 1);
    using P = Pair16<T>;
    using P2 = typename P::type;

    __shared__ __align__(128) QuantTable lut;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, wip = tid >> 5, t = lane & 7, sub = lane >> 3;
    float* slot_buf = reinterpret_cast<float*>(smem_raw) + (wip * 4 + sub) * SLOT;
    const TransposeConsts<KT> tc = transpose_consts<KT>(lane);
    const TransposeConsts<VB> tcv = transpose_consts<VB>(lane);
    (void)tc;
    (void)tcv;
    if constexpr (!KFP8) {
        // per cell: (midpoint inside it * 2^100, midpoints up to and including the cell): code = second -
        // sat(2^100 (m - y)); without a midpoint the first is -FLT_MAX and the saturated term 0
        for (int c = tid; c < kQuantCells; c += blockDim.x) {
            float thr = -FLT_MAX, upto = 0.f;
#pragma unroll
            for (int j = 0; j < (1 << KB) - 1; j++) {
                const float m = p.midpoints[j];
                const int cm = static_cast<int>(quant_cell(m));
                if (cm == c) thr = m * kStepScale;
                if (cm <= c) upto += 1.f;
            }
#pragma unroll
            for (int i = 0; i < 16; i++) lut[c][(i + c) & 15] = make_float2(thr, upto);
        }
        __syncthreads();
    }
    let_next_kernel_start();
    after_previous_kernel();
    const uint32_t lut_col = (lane & 15) * 8;
    const u64 scale2 = pk2(p.rsqrt_d, p.rsqrt_d), cs2 = pk2(kCellScale, kCellScale), cm2 = pk2(kCellMagic, kCellMagic);

    // butterfly of the pair, load layout -> coordinates l + 8 k
    auto fwht2 = [&](u64 (&x)[E]) {
        stage2<E, 0>(x);
        stage2<E, 1>(x);
        stage2<E, 2>(x);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NCH; i++) {
            float* run = slot_buf + (t + 8 * i) * kRunStride;
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
                ulonglong2 v2;
                v2.x = x[8 * i + c];
                v2.y = x[8 * i + c + 1];
                *reinterpret_cast<ulonglong2*>(run + 2 * c) = v2;
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < E; k++) x[k] = *reinterpret_cast<const u64*>(slot_buf + k * kRunStride + 2 * t);
        stage2<E, 0>(x);
        stage2<E, 1>(x);
        stage2<E, 2>(x);
        if constexpr (E >= 16) stage2<E, 3>(x);
        if constexpr (E >= 32) stage2<E, 4>(x);
    };
    // correctly rounded x / d: r2 = reciprocals, nd2 = -d
    auto quotient = [](u64 x, u64 r2, u64 nd2) {
        u64 q = mul2(x, r2);
        q = fma2(fma2(nd2, q, x), r2, q);
        return fma2(fma2(nd2, q, x), r2, q);
    };
    const uint32_t n_vec = pp.n_vec;
    const uint32_t step = 8 * ((gridDim.x * blockDim.x) >> 5);
    const T* const kbase = static_cast<const T*>(p.key) + blockIdx.y * p.kv_layer_stride;
    const T* const vbase = static_cast<const T*>(p.value) + blockIdx.y * p.kv_layer_stride;
    uint32_t base = 8 * ((blockIdx.x * blockDim.x + tid) >> 5);

    Raw8<T> raw[2][NCH];          // the pair's K, then its V
    int64_t row[2], slot[2];      // row offsets and slots of the group whose K is in `raw`
    uint32_t head[2];
    auto load_rows = [&](const T* tensor, uint32_t at) {
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const bool ok = at + 4 * x + sub < n_vec;
#pragma unroll
            for (int i = 0; i < NCH; i++) {
                if (ok) load_raw8<T>(tensor + row[x] + 8 * (t + 8 * i), raw[x][i]);
                else zero_raw8<T>(raw[x][i]);
            }
        }
    };
    auto start_group = [&]() {
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const uint32_t v = base + 4 * x + sub;
            const bool ok = v < n_vec;
            const uint32_t token = ok ? fast_div(v, p.div_hkv) : 0u;
            head[x] = ok ? v - token * p.Hkv : 0u;
            row[x] = static_cast<int64_t>(token) * p.token_stride + static_cast<int64_t>(head[x]) * p.head_stride;
            slot[x] = ok ? p.slot_mapping[token] : -1;   // (looked at after the key's arithmetic)
        }
        load_rows(kbase, base);
    };
    if (base < n_vec) start_group();

    while (base < n_vec) {
        // ---- key: norm of the raw vector, normalise, butterfly, code
        u64 x[E];
        uint32_t smallest = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < NCH; i++) {
            const uint32_t wa[4] = {raw[0][i].v.x, raw[0][i].v.y, raw[0][i].v.z, raw[0][i].v.w};
            const uint32_t wb[4] = {raw[1][i].v.x, raw[1][i].v.y, raw[1][i].v.z, raw[1][i].v.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if constexpr (KFP8 || P::kTiny > 0u) {
                    smallest = small_min<KFP8>(wa[j], smallest);
                    smallest = small_min<KFP8>(wb[j], smallest);
                }
                const float2 a = widen_pair<T>(wa[j]), b = widen_pair<T>(wb[j]);
                x[8 * i + 2 * j] = pk2(a.x, b.x);
                x[8 * i + 2 * j + 1] = pk2(a.y, b.y);
            }
        }
        load_rows(vbase, base);
        u64 s2 = pk2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < E; r++) s2 = fma2(x[r], x[r], s2);
#pragma unroll
        for (int m = 1; m < 8; m <<= 1) s2 = add2(s2, __shfl_xor_sync(0xffffffffu, s2, m));
        float sA, sB;
        upk2(s2, sA, sB);
        const float normA = __fsqrt_rn(__fadd_rn(sA, 1e-16f)), normB = __fsqrt_rn(__fadd_rn(sB, 1e-16f));
        const float dA = __fadd_rn(normA, 1e-8f), dB = __fadd_rn(normB, 1e-8f);
        // (for bf16 the limit is the pattern of 2^-40; with FP8 keys a half of `smallest` below it is -0 or tiny)
        constexpr uint32_t kLimit = P::kTiny > 0u ? P::kTiny - 1u : 1u;
        bool odd_case = !(normA < 1048576.f) || !(normB < 1048576.f);
        if constexpr (KFP8 || P::kTiny > 0u) odd_case |= (smallest & 0xffffu) < kLimit || (smallest >> 16) < kLimit;
        {
            const u64 r2 = pk2(__frcp_rn(dA), __frcp_rn(dB)), nd2 = pk2(-dA, -dB);
#pragma unroll
            for (int r = 0; r < E; r++) x[r] = quotient(x[r], r2, nd2);
        }
        fwht2(x);

        // ---- where the pair's slots are: negative = padding (triton_inkernel_store.py:398-399), beyond the
        // cache's end is dropped the same way
        uint8_t* dst[2];
#pragma unroll
        for (int y = 0; y < 2; y++) {
            dst[y] = nullptr;
            if (static_cast<uint64_t>(slot[y]) < static_cast<uint64_t>(p.slot_limit)) {
                int64_t blk, off;
                if (slot[y] < (1ll << 31)) {
                    const uint32_t b32 = fast_div(static_cast<uint32_t>(slot[y]), p.div_block);
                    blk = b32;
                    off = static_cast<uint32_t>(slot[y]) - b32 * p.block_size;
                } else {
                    blk = slot[y] / p.block_size;
                    off = slot[y] - blk * p.block_size;
                }
                dst[y] = p.kv_cache + blockIdx.y * p.cache_layer_stride + blk * p.stride_block + off * p.stride_pos +
                         head[y] * p.stride_head;
            }
        }
        if (__any_sync(0xffffffffu, odd_case)) {
            tq_store2_plain<D, KB, VB, T, ROTV>(p, n_vec, base, lane);
            base += step;
            if (base < n_vec) start_group();
            continue;
        }
        if constexpr (KFP8) {
            const u64 n2 = pk2(normA, normB);
#pragma unroll
            for (int k = 0; k < E; k += 2) {
                float a0, b0, a1, b1;
                upk2(mul2(mul2(x[k], scale2), n2), a0, b0);
                upk2(mul2(mul2(x[k + 1], scale2), n2), a1, b1);
                // neighbouring lanes trade bytes: the even lane stores the pair of coordinate row k, the odd one
                // that of row k + 1
                const uint32_t own = __nv_cvt_float2_to_fp8x2(make_float2(a0, a1), __NV_SATFINITE, __NV_E4M3) |
                                     (static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(b0, b1), __NV_SATFINITE, __NV_E4M3)) << 16);
                const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
                const uint32_t two = __byte_perm(own, other, (lane & 1) ? 0x3715u : 0x6240u);   // A's pair, B's pair
                const int coord = (lane & 1) ? t - 1 + 8 * (k + 1) : t + 8 * k;
                if (dst[0]) *reinterpret_cast<uint16_t*>(dst[0] + coord) = static_cast<uint16_t>(two);
                if (dst[1]) *reinterpret_cast<uint16_t*>(dst[1] + coord) = static_cast<uint16_t>(two >> 16);
            }
        } else {
            u64 wf[NCH * FPW];
#pragma unroll
            for (int i = 0; i < NCH * FPW; i++) wf[i] = pk2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < E; k++) {
                const u64 y = mul2(x[k], scale2);
                float cA, cB, yA, yB;
                upk2(fma2(y, cs2, cm2), cA, cB);
                upk2(y, yA, yB);
                const float2 eA = *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(&lut) +
                                                                   ((__float_as_uint(cA) & 0xFF80u) | lut_col));
                const float2 eB = *reinterpret_cast<const float2*>(reinterpret_cast<const uint8_t*>(&lut) +
                                                                   ((__float_as_uint(cB) & 0xFF80u) | lut_col));
                const u64 code = sub2(pk2(eA.y, eB.y), pk2(fma_sat(yA, -kStepScale, eA.x), fma_sat(yB, -kStepScale, eB.x)));
                const int pos = k & 7, fi = (k >> 3) * FPW + pos / CPF;
                const float sc = static_cast<float>(1u << (KT * (pos % CPF)));
                wf[fi] = fma2(code, pk2(sc, sc), wf[fi]);
            }
            uint32_t wA[NCH], wB[NCH];
#pragma unroll
            for (int i = 0; i < NCH; i++) {
                float a0, b0;
                upk2(wf[i * FPW], a0, b0);
                wA[i] = __float2uint_rn(a0);
                wB[i] = __float2uint_rn(b0);
                if constexpr (FPW == 2) {
                    float a1, b1;
                    upk2(wf[i * FPW + 1], a1, b1);
                    wA[i] |= __float2uint_rn(a1) << (KT * CPF);
                    wB[i] |= __float2uint_rn(b1) << (KT * CPF);
                }
            }
            tq_emit_columns<KT, NCH>(wA, dst[0], t, tc);
            tq_emit_columns<KT, NCH>(wB, dst[1], t, tc);
            if (t == 0) {
                if (dst[0]) *reinterpret_cast<__half*>(dst[0] + MSE) = __float2half_rn(normA);
                if (dst[1]) *reinterpret_cast<__half*>(dst[1] + MSE) = __float2half_rn(normB);
            }
        }

        // ---- value: (rotate and round to T,) range of the vector, uniform codes
        uint32_t w16[2][E / 2];   // [vector] the values as pairs of T
        if constexpr (ROTV) {
#pragma unroll
            for (int i = 0; i < NCH; i++) {
                const uint32_t wa[4] = {raw[0][i].v.x, raw[0][i].v.y, raw[0][i].v.z, raw[0][i].v.w};
                const uint32_t wb[4] = {raw[1][i].v.x, raw[1][i].v.y, raw[1][i].v.z, raw[1][i].v.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float2 a = widen_pair<T>(wa[j]), b = widen_pair<T>(wb[j]);
                    x[8 * i + 2 * j] = pk2(a.x, b.x);
                    x[8 * i + 2 * j + 1] = pk2(a.y, b.y);
                }
            }
            fwht2(x);
#pragma unroll
            for (int k = 0; k < E; k += 2) {
                float a0, b0, a1, b1;
                upk2(mul2(x[k], scale2), a0, b0);
                upk2(mul2(x[k + 1], scale2), a1, b1);
                const P2 a = P::round(a0, a1), b = P::round(b0, b1);
                w16[0][k / 2] = *reinterpret_cast<const uint32_t*>(&a);
                w16[1][k / 2] = *reinterpret_cast<const uint32_t*>(&b);
            }
        } else {
#pragma unroll
            for (int y = 0; y < 2; y++)
#pragma unroll
                for (int i = 0; i < NCH; i++) {
                    w16[y][4 * i] = raw[y][i].v.x;
                    w16[y][4 * i + 1] = raw[y][i].v.y;
                    w16[y][4 * i + 2] = raw[y][i].v.z;
                    w16[y][4 * i + 3] = raw[y][i].v.w;
                }
        }
        float mn[2], sc[2];
        bool wild = false;
#pragma unroll
        for (int y = 0; y < 2; y++) {
            auto as2 = [](uint32_t w) { return *reinterpret_cast<const P2*>(&w); };
            P2 lo = as2(w16[y][0]), hi = lo;
#pragma unroll
            for (int k = 1; k < E / 2; k++) {   // (a NaN stays: the vector is not for this kernel then)
                lo = __hmin2_nan(lo, as2(w16[y][k]));
                hi = __hmax2_nan(hi, as2(w16[y][k]));
            }
            // (minimum, minus the maximum) as one pair
            P2 both;
            both.x = __hmin_nan(lo.x, lo.y);
            both.y = __hneg(__hmax_nan(hi.x, hi.y));
#pragma unroll
            for (int m = 1; m < 8; m <<= 1) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t*>(&both), m);
                both = __hmin2_nan(both, as2(o));
            }
            const float2 f = widen_pair<T>(*reinterpret_cast<const uint32_t*>(&both));
            mn[y] = f.x;
            sc[y] = __fdiv_rn(__fsub_rn(-f.y, f.x), kVMax);
            wild |= !(sc[y] < 1.2676506e30f);
            sc[y] = sc[y] > 1e-8f ? sc[y] : 1e-8f;
        }
        if (__any_sync(0xffffffffu, wild)) {
            tq_store2_plain<D, KB, VB, T, ROTV>(p, n_vec, base, lane);
            base += step;
            if (base < n_vec) start_group();
            continue;
        }
        const u64 r2 = pk2(__frcp_rn(sc[0]), __frcp_rn(sc[1])), ns2 = pk2(-sc[0], -sc[1]), nm2 = pk2(-mn[0], -mn[1]);
        const u64 half2 = pk2(0.5f, 0.5f), magic2 = pk2(8388608.f, 8388608.f);
        // (the sum of the words' 2^23 patterns, taken off at the end)
        uint32_t vw[2][NCH];
#pragma unroll
        for (int i = 0; i < NCH; i++) {
            uint32_t off = 0;
#pragma unroll
            for (int c = 0; c < 8; c++) off += 0x4B000000u << (VB * c);
            vw[0][i] = vw[1][i] = 0u - off;
        }
#pragma unroll
        for (int k = 0; k < E / 2; k++) {
            const float2 a = widen_pair<T>(w16[0][k]), b = widen_pair<T>(w16[1][k]);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const u64 v2 = add2(j ? pk2(a.y, b.y) : pk2(a.x, b.x), nm2);
                const u64 c2 = add2_down(add2(quotient(v2, r2, ns2), half2), magic2);
                float cA, cB;
                upk2(c2, cA, cB);
                const int pos = (2 * k + j) & 7, i = (2 * k + j) >> 3;
                vw[0][i] += __float_as_uint(cA) << (VB * pos);
                vw[1][i] += __float_as_uint(cB) << (VB * pos);
            }
        }
        uint8_t* const va = dst[0] ? dst[0] + KPS : nullptr;
        uint8_t* const vb = dst[1] ? dst[1] + KPS : nullptr;
        // next group's keys fly while this one's value codes are stored
        base += step;
        if (base < n_vec) start_group();
        if constexpr (ROTV) {
            tq_emit_columns<VB, NCH>(vw[0], va, t, tcv);
            tq_emit_columns<VB, NCH>(vw[1], vb, t, tcv);
        } else {
            tq_emit_runs<VB, NCH>(vw[0], va, t);
            tq_emit_runs<VB, NCH>(vw[1], vb, t);
        }
        if (t == 0) {
            if (va) {
                *reinterpret_cast<__half*>(va + VDB) = __float2half_rn(sc[0]);
                *reinterpret_cast<__half*>(va + VDB + 2) = __float2half_rn(mn[0]);
            }
            if (vb) {
                *reinterpret_cast<__half*>(vb + VDB) = __float2half_rn(sc[1]);
                *reinterpret_cast<__half*>(vb + VDB + 2) = __float2half_rn(mn[1]);
            }
        }
    }
}

}  // namespace ftq
