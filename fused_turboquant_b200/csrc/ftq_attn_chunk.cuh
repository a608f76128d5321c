// Causal attention of a chunk of new tokens per sequence over the paged cache (chunked prefill,
// speculative verification) on the fifth-generation tensor cores.
//
// The reference runs the decode kernel on one synthetic sequence per query
// (src/fused_turboquant/vllm_plugin/v1_backend.py:1359-1384): every query walks the whole cache again,
// and 64 queries dequantise every page 64 times (252 us for 4 x 64 queries over 4096 tokens, 32 / 8
// heads of 128, K4V4).  Here the queries of a GQA group are the M dimension of a matrix product: row
// r of a unit (sequence, KV head) is query r / group, head r % group, a row tile has 128 rows, and a
// page is dequantised once per CTA for SLOTS row tiles.
//
//   S = Q.K^T   tcgen05.mma, M = 128 rows, N = KT tokens, K = D; Q and K in shared memory (K-major,
//               128-byte swizzle), S in TMEM
//   softmax     one thread per row: TMEM -> registers, key norms, causal limit, online maximum
//   O += P.V    tcgen05.mma, M = 128, N = D, K = KT; the weights p * vnorm (fp16, as in the decode
//               kernels) go back to TMEM as the A operand, V is read MN-major from the same layout
//               that K has; O stays in TMEM
//
// Rounding is that of the decode kernels: fp16 centroids (scaled by the host for the smallest error),
// fp16 rotated queries, fp16 weights, fp32 accumulation, fp32 softmax.
//
// Warps: SLOTS x 4 softmax warps, KT * D / 1024 dequantising warps (codes of a tile are loaded into
// registers one tile ahead, looked up in the lane-replicated tables, written as fp16 tiles, three
// stages), one warp that issues the MMAs: scores of tile i are issued before P.V of tile i - 1, so that
// softmax, dequantisation and the tensor core overlap.  What bounds it is that last warp's line of work: by the clock
// of a CTA (4 x 64 queries over 4096 tokens, 32 / 8 heads of 128, K4V4) a tile of 64 tokens and 256 rows took 4200 cycles,
// 1000 of them waiting for the tile, 1780 for the scores' sixteen MMAs, 1250 for P.V's eight; now 3060, with a third
// stage and operands in uniform registers.  61.5 -> 53.4 us with its merge, 50.9 with the queries' loads side by side and the
// tables built while the kernel before drains; 2 x 512 queries 172 -> 130.
//
// The tiles of a row tile's causal range are cut into up to `splits` parts (grid.x); every CTA leaves its rows
// (O, m, l) in the workspace and attn_merge_kernel finishes.
//
// Every wait is bounded; one that runs out makes the CTA's rows NaN and sets a bit of the status word.
// Block ids outside [0, num_blocks) are never dereferenced and have the same effect on the rows that attend
// a token of such a page.
#pragma once

#include <cfloat>
#include <climits>

#include "ftq_attn_mma.cuh"

namespace ftq {

struct ChunkAttnParams {
    const void* q;              // [B, q_len, Hq, D]
    const uint8_t* pool;        // one layer: [num_blocks, Hkv, page_bytes]
    const int32_t* block_table; // [B, max_blocks]
    const int32_t* seq_lens;    // [B], the new tokens included
    int64_t num_blocks;
    int max_blocks, max_seq, q_len, Hq, Hkv, q_dtype;
    int splits, splits_even;    // parts of a context: rows per query vector and grid.x; used for even lengths
    float q_scale;              // softmax scale / (key table's scale) * log2(e) / sqrt(D)
    float inv_v_scale;
    float* partials;            // [B * q_len * Hq][splits][D + 4]
    // what went wrong (expired waits, bad block ids): a word holds `epoch` if it did; the merge kernel turns them into the
    // call's status word
    unsigned long long* errors;
    unsigned long long epoch;
    Codebook lk, lv;            // scaled for their fp16 rounding
    SignBits signs;
};

template <int D, int BK, int BV>
struct ChunkCfg {
    // head_dim 256: the accumulator of one row tile takes half of TMEM and its queries 64 KB
    static constexpr int SLOTS = D == 256 ? 1 : 2;
    static constexpr int KT = D == 256 ? 32 : 64;          // tokens per tile
    static constexpr int SM_WARPS = 4 * SLOTS;
    static constexpr int NG = D / 32;                      // 32-coordinate groups of a row
    static constexpr int DQ_THREADS = KT * NG, DQ_WARPS = DQ_THREADS / 32;
    static constexpr int THREADS = 32 * (SM_WARPS + DQ_WARPS + 1);
    static constexpr int PDK = packed_dim(D, BK), PDV = packed_dim(D, BV);
    static constexpr int OFF_KN = kPageTokens * PDK;
    static constexpr int OFF_VC = OFF_KN + 2 * kPageTokens;
    static constexpr int OFF_VN = OFF_VC + kPageTokens * PDV;
    static constexpr int PAGE_BYTES = OFF_VN + 2 * kPageTokens;
    static constexpr int TK_BYTES = (1 << (2 * BK)) * 128, TV_BYTES = (1 << (2 * BV)) * 128;
    // K and V tiles: with two, a tile was dequantised (1000 cycles) after P.V of the tile before the last and before its own
    // scores, i.e. in series with the tensor core
    static constexpr int STAGES = 3;
    // shared memory, 1024-byte aligned parts: Q tiles, K and V tiles, tables, norms, barriers
    static constexpr int Q_TILE = 128 * D * 2, KV_TILE = KT * D * 2;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_K = OFF_Q + SLOTS * Q_TILE;
    static constexpr int OFF_V = OFF_K + STAGES * KV_TILE;
    static constexpr int OFF_TK = OFF_V + STAGES * KV_TILE;
    static constexpr int OFF_TV = OFF_TK + TK_BYTES;
    static constexpr int OFF_NORM = OFF_TV + TV_BYTES;     // [STAGES][2][KT] floats
    static constexpr int OFF_BAR = OFF_NORM + STAGES * 2 * KT * 4;
    static constexpr int USED = OFF_BAR + 160 + 1024;      // (1024: alignment of the base)
    // one CTA per SM: a second one would only wait for TMEM
    static constexpr int SMEM_BYTES = USED > 120 * 1024 ? USED : 120 * 1024;
    // TMEM columns of a slot: O (fp32), S (fp32), P (fp16 pairs)
    static constexpr int COL_S = D, COL_P = D + KT, COLS = D + KT + KT / 2;
    static_assert(SLOTS * COLS <= 512 && SMEM_BYTES <= 227 * 1024 && THREADS <= 1024, "");
};

// Polls of a wait of the chunk kernel.  FTQ_TEST_WAIT_EXPIRY (only the test library of build.py defines it):
// the first dequantising warp of CTA (0, 0, 0) does not report its second tile, so that the waits for the
// tile run out and the give-up path executes; the limit is then small.
#ifdef FTQ_TEST_WAIT_EXPIRY
constexpr int kChunkSpinLimit = 1 << 12;
#else
constexpr int kChunkSpinLimit = kMbarSpinLimit;
#endif
constexpr int kDrainSpinLimit = 1 << 20;   // for the CTA's own MMAs in flight

// ---- tcgen05 (cta_group::1): addresses of TMEM are lane << 16 | column
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// (Run by a whole warp, whose lane `one` issues: the operands are uniform registers, and code that only one lane
// runs has to move each of them there.  Shared-memory descriptors as lower and upper halves; the upper one is
// common to both operands.)
__device__ __forceinline__ void tc_mma_ss(bool one, uint32_t d, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n.reg .pred p, q;\n.reg .b64 da, db;\nmov.b64 da, {%1, %3};\nmov.b64 db, {%2, %3};\nsetp.ne.b32 p, %5, 0;\n"
        "setp.ne.b32 q, %6, 0;\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n}\n" ::"r"(d), "r"(a), "r"(b),
        "r"(hi), "r"(idesc), "r"(static_cast<uint32_t>(acc)), "r"(static_cast<uint32_t>(one)) : "memory");
}
__device__ __forceinline__ void tc_mma_ts(bool one, uint32_t d, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n.reg .pred p, q;\n.reg .b64 db;\nmov.b64 db, {%2, %3};\nsetp.ne.b32 p, %5, 0;\n"
        "setp.ne.b32 q, %6, 0;\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}\n" ::"r"(d), "r"(a), "r"(b),
        "r"(hi), "r"(idesc), "r"(static_cast<uint32_t>(acc)), "r"(static_cast<uint32_t>(one)) : "memory");
}
// 32 lanes x 16 columns of 32 bits, one row per lane
__device__ __forceinline__ void tc_ld16(uint32_t addr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ void tc_st16(uint32_t addr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::
            "r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
            "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// (the registers of earlier tc_ld16 calls pass through, so that nothing uses them before the wait)
__device__ __forceinline__ void tc_wait_ld(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle: bits 0-13 address / 16, 16-29 the distance of 64-element chunks / 16
// (MN-major; K-major: unused), 32-45 of 8-row (K-major) or 8-k (MN-major) groups / 16, 46 set, 61-63 = 2.  Addresses are
// below 256 KB.
template <int D, int BK, int BV>
__global__ void __launch_bounds__(ChunkCfg<D, BK, BV>::THREADS, 1)
attn_chunk_kernel(const __grid_constant__ ChunkAttnParams p) {
    using C = ChunkCfg<D, BK, BV>;
    constexpr int KT = C::KT, SLOTS = C::SLOTS, E = D / kOctet, ROW = D + 4;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t raw = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    const uint32_t sbase = (raw + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (sbase - raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

    // ---- tables: an entry (the fp16 centroids of two adjacent codes) 32 times, bank = lane
    {
        auto build = [&](int off, int bits, const Codebook& cb) {
            uint32_t* t = reinterpret_cast<uint32_t*>(smem + off);
            const float lev = cb.v[lane & 15];
            for (int e = warp; e < (1 << (2 * bits)); e += C::THREADS / 32) {
                const __half2 h = __floats2half2_rn(__shfl_sync(0xffffffffu, lev, e & ((1 << bits) - 1)),
                                                    __shfl_sync(0xffffffffu, lev, e >> bits));
                t[e * 32 + lane] = *reinterpret_cast<const uint32_t*>(&h);
            }
        };
        build(C::OFF_TK, BK, p.lk);
        build(C::OFF_TV, BV, p.lv);
    }
    after_previous_kernel();    // (nothing in global memory was touched so far)

    // ---- what this CTA works on
    const int group = p.Hq / p.Hkv, rows = p.q_len * group;
    const int split = blockIdx.x, b = blockIdx.z;
    const int hkv = blockIdx.y % p.Hkv, row0 = (blockIdx.y / p.Hkv) * (128 * SLOTS);
    const int n_slots = min(SLOTS, (rows - row0 + 127) / 128);
    const int row_end = min(rows, row0 + 128 * SLOTS);
    const int seq = min(p.seq_lens[b], p.max_seq);
    // query i attends positions below limit0 + i (and max_seq); no row of this CTA attends one at or
    // behind the limit of its last row
    const int limit0 = p.seq_lens[b] - p.q_len + 1;
    const int reach = max(0, min(p.max_seq, limit0 + (row_end - 1) / group));
    const int all_tiles = (reach + KT - 1) / KT;
    // parts: p.splits_even when the contexts are of about one length, else p.splits, of eight tiles or more
    // (more than half of the longest on average is "about"; the host makes both the same number where it
    // does not matter)
    int parts = p.splits_even, per = 0;
    if (p.splits != p.splits_even) {   // (grid-uniform; every warp looks for itself)
        uint32_t longest = 0, sum = 0;   // in pages
        for (int i = lane; i < static_cast<int>(gridDim.z); i += 32) {
            const uint32_t n = (max(0, min(p.seq_lens[i], p.max_seq)) + kPageTokens - 1) / kPageTokens;
            longest = max(longest, n);
            sum += n;
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (2ull * sum < static_cast<unsigned long long>(longest) * gridDim.z) {
            parts = p.splits;
            per = 8;
        }
    }
    per = max(per, (all_tiles + parts - 1) / parts);
    const int tile0 = min(split * per, all_tiles), n_tiles = min(per, all_tiles - tile0);
    auto partial_row = [&](int r) {   // r: row of the unit
        const int i = r / group;
        return p.partials + (((static_cast<int64_t>(b) * p.q_len + i) * p.Hq + hkv * group + (r - i * group)) *
                                 p.splits + split) * ROW;
    };
    if (n_tiles <= 0) {   // (CTA-uniform)
        for (int r = row0 + tid; r < row_end; r += C::THREADS) {
            float* dst = partial_row(r);
            dst[D] = -INFINITY;
            dst[D + 1] = 0.f;
        }
        return;
    }

    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;     // a wait ran out
    __shared__ int s_bad_pos;   // first token on a page whose block id is out of range
    __shared__ int s_nan_pos;   // first token whose value norm is NaN
    const volatile int* const abort_now = &s_abort;
    const uint32_t bars = sbase + C::OFF_BAR;
    constexpr int NST = C::STAGES;
    const uint32_t kv_full = bars, kv_empty = bars + 32,                    // NST of each
                   s_full = bars + 64, s_free = bars + 80, p_full = bars + 96, o_done = bars + 112,   // two of each
                   drained = bars + 128;
    if (warp == C::SM_WARPS + C::DQ_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&s_tmem))) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
        if (lane == 0) {
            for (int i = 0; i < NST; i++) {
                mbar_init(kv_full + 8 * i, C::DQ_WARPS);
                mbar_init(kv_empty + 8 * i, 1);
            }
            for (int i = 0; i < 2; i++) {
                mbar_init(s_full + 8 * i, 1);
                mbar_init(s_free + 8 * i, 4);
                mbar_init(p_full + 8 * i, 4);
                mbar_init(o_done + 8 * i, 1);
            }
            mbar_init(drained, 1);
            mbar_fence_init();
        }
        tc_fence_before();
    }
    if (tid == 0) {
        s_abort = 0;
        s_bad_pos = s_nan_pos = INT_MAX;
    }
    // ---- queries: rotated, scaled, fp16, K-major with 128-byte swizzle; an octet per row, all rows' loads first
    constexpr int PER = C::THREADS / 8, ROUNDS = (SLOTS * 128 + PER - 1) / PER;
    uint4 raw_q[ROUNDS][E / 8];
#pragma unroll
    for (int j = 0; j < ROUNDS; j++) {
        const int gr = row0 + j * PER + (tid >> 3);
        const int i = gr < row_end ? gr / group : 0, h = gr < row_end ? gr - i * group : 0;
        const int64_t qoff = ((static_cast<int64_t>(b) * p.q_len + i) * p.Hq + hkv * group + h) * D;
#pragma unroll
        for (int k = 0; k < E / 8; k++)
            raw_q[j][k] = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.q) + qoff + 8 * ((lane & 7) + 8 * k));
    }
#pragma unroll
    for (int j = 0; j < ROUNDS; j++) {
        const int r = j * PER + (tid >> 3), t8 = lane & 7;
        if (j * PER + 4 * warp >= n_slots * 128) continue;   // (warp-uniform)
        const bool valid = row0 + r < rows;
        float a[E];
#pragma unroll
        for (int k = 0; k < E / 8; k++) {
            float tmp[8];
            if (p.q_dtype == kBF16) load8<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(&raw_q[j][k]), tmp);
            else load8<__half>(reinterpret_cast<const __half*>(&raw_q[j][k]), tmp);
#pragma unroll
            for (int c = 0; c < 8; c++)
                a[8 * k + c] = __uint_as_float(
                    __float_as_uint(tmp[c]) ^ sign_mask(p.signs, load_coord(t8, 8 * k + c)));
        }
        octet_fwht<E>(a, lane);
        const int slot = r >> 7, rr = r & 127;
        uint8_t* dst = smem + C::OFF_Q + slot * C::Q_TILE + rr * 128 + 2 * t8;
        if (r < n_slots * 128) {
#pragma unroll
            for (int k = 0; k < E; k++) {   // coordinate t8 + 8 k: 16-byte chunk k & 7 of 64-coordinate chunk k / 8
                const __half v = __float2half_rn(valid ? a[k] * p.q_scale : 0.f);
                *reinterpret_cast<__half*>(dst + (k >> 3) * (128 * 128) + (((k & 7) ^ (rr & 7)) << 4)) = v;
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

    // bounded wait; false: give up (somebody's wait ran out)
    auto wait = [&](uint32_t bar, uint32_t parity) {
        for (int i = 0; i < kChunkSpinLimit; i++) {
            if (mbar_try_wait(bar, parity & 1u)) return true;
            if ((i & 63) == 63 && *abort_now) return false;
        }
        s_abort = 1;
        return false;
    };

    if (warp < C::SM_WARPS) {
        // ================= softmax: one thread per row
        const int slot = warp >> 2, quarter = warp & 3;
        const int r = row0 + slot * 128 + quarter * 32 + lane;
        if (slot < n_slots) {
            const uint32_t tm = tmem + slot * C::COLS + (static_cast<uint32_t>(quarter * 32) << 16);
            const int limit = r < rows ? min(p.max_seq, limit0 + r / group) : 0;
            const float* norms = reinterpret_cast<const float*>(smem + C::OFF_NORM);
            float m_run = -INFINITY, l_run = 0.f;
            bool alive = true;
            for (int it = 0; it < n_tiles; it++) {
                const int st = it % NST;
                alive = wait(kv_full + 8 * st, it / NST) && wait(s_full + 8 * slot, it);
                if (!__all_sync(0xffffffffu, alive)) break;
                tc_fence_after();
                uint32_t sr[KT];
#pragma unroll
                for (int c = 0; c < KT; c += 16) tc_ld16(tm + C::COL_S + c, sr + c);
#pragma unroll
                for (int c = 0; c < KT; c += 16) tc_wait_ld(sr + c);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free + 8 * slot);
                const float4* kn = reinterpret_cast<const float4*>(norms + st * 2 * KT);
                const float4* vn = kn + KT / 4;
                float mx = -INFINITY;
                const int left = limit - (tile0 + it) * KT;   // tokens of this tile the row attends
                if (__all_sync(0xffffffffu, left >= KT)) {
#pragma unroll
                    for (int c = 0; c < KT; c += 4) {
                        const float4 n = kn[c / 4];
                        const float x0 = __uint_as_float(sr[c]) * n.x, x1 = __uint_as_float(sr[c + 1]) * n.y;
                        const float x2 = __uint_as_float(sr[c + 2]) * n.z, x3 = __uint_as_float(sr[c + 3]) * n.w;
                        mx = fmaxf(fmaxf(mx, fmaxf(x0, x1)), fmaxf(x2, x3));
                        sr[c] = __float_as_uint(x0);
                        sr[c + 1] = __float_as_uint(x1);
                        sr[c + 2] = __float_as_uint(x2);
                        sr[c + 3] = __float_as_uint(x3);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < KT; c += 4) {
                        const float4 n = kn[c / 4];
                        const float x0 = c < left ? __uint_as_float(sr[c]) * n.x : -INFINITY;
                        const float x1 = c + 1 < left ? __uint_as_float(sr[c + 1]) * n.y : -INFINITY;
                        const float x2 = c + 2 < left ? __uint_as_float(sr[c + 2]) * n.z : -INFINITY;
                        const float x3 = c + 3 < left ? __uint_as_float(sr[c + 3]) * n.w : -INFINITY;
                        mx = fmaxf(fmaxf(mx, fmaxf(x0, x1)), fmaxf(x2, x3));
                        sr[c] = __float_as_uint(x0);
                        sr[c + 1] = __float_as_uint(x1);
                        sr[c + 2] = __float_as_uint(x2);
                        sr[c + 3] = __float_as_uint(x3);
                    }
                }
                // P.V of the tile before has read P and written O
                if (it > 0) {
                    alive = wait(o_done + 8 * slot, it - 1);
                    if (!__all_sync(0xffffffffu, alive)) break;
                    tc_fence_after();
                }
                // lazy reference maximum, as in the decode kernels (weights stay below 2^kLazyMaxSlack)
                const bool above = mx > m_run + kLazyMaxSlack;
                if (__any_sync(0xffffffffu, above)) {
                    const float m_new = fmaxf(m_run, mx);
                    const float corr = m_run == -INFINITY ? 0.f : fast_exp2(m_run - m_new);
                    l_run *= corr;
                    m_run = m_new;
                    if (it > 0) {
#pragma unroll 1
                        for (int c = 0; c < D; c += 16) {
                            uint32_t o[16];
                            tc_ld16(tm + c, o);
                            tc_wait_ld(o);
#pragma unroll
                            for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
                            tc_st16(tm + c, o);
                        }
                    }
                }
                const float m_use = m_run == -INFINITY ? 0.f : m_run;   // (nothing attended so far)
                float l0 = 0.f, l1 = 0.f;
#pragma unroll
                for (int c = 0; c < KT; c += 4) {
                    const float4 n = vn[c / 4];   // (finite; tokens that the row does not attend have p = 0)
                    const float p0 = fast_exp2(__uint_as_float(sr[c]) - m_use), p1 = fast_exp2(__uint_as_float(sr[c + 1]) - m_use);
                    const float p2 = fast_exp2(__uint_as_float(sr[c + 2]) - m_use), p3 = fast_exp2(__uint_as_float(sr[c + 3]) - m_use);
                    l0 += p0 + p1;
                    l1 += p2 + p3;
                    sr[c / 2] = f2h2_sat(p0 * n.x, p1 * n.y);
                    sr[c / 2 + 1] = f2h2_sat(p2 * n.z, p3 * n.w);
                }
                l_run += l0 + l1;
#pragma unroll
                for (int c = 0; c < KT / 2; c += 16) tc_st16(tm + C::COL_P + c, sr + c);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + 8 * slot);
            }
            alive = __all_sync(0xffffffffu, alive) && __all_sync(0xffffffffu, wait(o_done + 8 * slot, n_tiles - 1));
            tc_fence_after();
            float* dst = r < rows ? partial_row(r) : nullptr;
#pragma unroll 1
            for (int c = 0; c < D; c += 16) {
                uint32_t o[16];
                tc_ld16(tm + c, o);
                tc_wait_ld(o);
                if (dst) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(dst + c + j) =
                            make_float4(__uint_as_float(o[j]) * p.inv_v_scale, __uint_as_float(o[j + 1]) * p.inv_v_scale,
                                        __uint_as_float(o[j + 2]) * p.inv_v_scale, __uint_as_float(o[j + 3]) * p.inv_v_scale);
                }
            }
            if (dst) {
                dst[D] = m_run == -INFINITY ? -INFINITY : m_run * kLn2;
                dst[D + 1] = l_run;
            }
            tc_fence_before();
        }
    } else if (warp < C::SM_WARPS + C::DQ_WARPS) {
        // ================= dequantisation: a thread turns 32 codes of a K row and of a V row into fp16
        const int idx = tid - 32 * C::SM_WARPS;
        const int gq = (idx >> 3) % C::NG, t = (idx & 7) + 8 * ((idx >> 3) / C::NG);   // group, token of the tile
        const int tok = t & (kPageTokens - 1);
        const int32_t* btab = p.block_table + static_cast<int64_t>(b) * p.max_blocks;
        const int n_pages = (seq + kPageTokens - 1) / kPageTokens;
        const uint8_t* head = p.pool + static_cast<int64_t>(hkv) * C::PAGE_BYTES;
        const int64_t blk_stride = static_cast<int64_t>(p.Hkv) * C::PAGE_BYTES;
        // the pool stores a V row with its halves exchanged for tokens with bit 1 set
        const int k_off = tok * C::PDK + gq * 4 * BK;
        const int v_off = C::OFF_VC + tok * C::PDV + (gq ^ ((tok & 2) ? C::NG / 2 : 0)) * 4 * BV;
        // (ordinary loads: the kernel before this one may have written what they read, see load8)
        auto page_id = [&](int it) {
            const int pg = ((tile0 + it) * KT + t) / kPageTokens;
            return it < n_tiles && pg < n_pages ? btab[pg] : -1;
        };
        auto words = [&](const uint8_t* src, auto bits, uint32_t* w) {
            constexpr int NB = decltype(bits)::value;
            if constexpr (NB == 4) {
                const uint4 x = *reinterpret_cast<const uint4*>(src);
                w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
            } else if constexpr (NB == 2) {
                const uint2 x = *reinterpret_cast<const uint2*>(src);
                w[0] = x.x; w[1] = x.y;
            } else {
#pragma unroll
                for (int i = 0; i < NB; i++) w[i] = reinterpret_cast<const uint32_t*>(src)[i];
            }
        };
        uint32_t kw[BK], vw[BV];
        float kn = 0.f, vn = 0.f;
        auto load = [&](int it, int id) {
#pragma unroll
            for (int i = 0; i < BK; i++) kw[i] = 0u;
#pragma unroll
            for (int i = 0; i < BV; i++) vw[i] = 0u;
            kn = vn = 0.f;
            const int pos = (tile0 + it) * KT + t;
            if (it >= n_tiles || pos >= seq) return;
            if (static_cast<uint64_t>(static_cast<int64_t>(id)) >= static_cast<uint64_t>(p.num_blocks)) {
                atomicMin(&s_bad_pos, pos);
                return;
            }
            const uint8_t* page = head + id * blk_stride;
            words(page + k_off, std::integral_constant<int, BK>{}, kw);
            words(page + v_off, std::integral_constant<int, BV>{}, vw);
            if (gq == 0) {
                kn = __half2float(reinterpret_cast<const __half*>(page + C::OFF_KN)[tok]);
                vn = __half2float(reinterpret_cast<const __half*>(page + C::OFF_VN)[tok]);
            }
        };
        const uint32_t tk = sbase + C::OFF_TK + lane * 4, tv = sbase + C::OFF_TV + lane * 4;
        float* norms = reinterpret_cast<float*>(smem + C::OFF_NORM);
        // row t of the tile: 64-coordinate chunk gq / 2, 16-byte chunks 4 * (gq & 1) ..
        const uint32_t row = (gq >> 1) * (KT * 128) + t * 128;
        auto put = [&](uint32_t tile, auto bits, const uint32_t* w, uint32_t table) {
            constexpr int NB = decltype(bits)::value;
            uint32_t ww[NB];
#pragma unroll
            for (int i = 0; i < NB; i++) ww[i] = w[i];
            uint32_t x[16];
#pragma unroll
            for (int e = 0; e < 16; e++) x[e] = lds32(table + pair_index<2 * NB>(ww, e));
#pragma unroll
            for (int j = 0; j < 4; j++)
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(
                                 tile + row + (((4 * (gq & 1) + j) ^ (t & 7)) << 4)),
                             "r"(x[4 * j]), "r"(x[4 * j + 1]), "r"(x[4 * j + 2]), "r"(x[4 * j + 3]) : "memory");
        };
        int id = page_id(0), id_next = page_id(1);
        load(0, id);
        for (int it = 0; it < n_tiles; it++) {
            const int st = it % NST;
            uint32_t k0[BK], v0[BV];
#pragma unroll
            for (int i = 0; i < BK; i++) k0[i] = kw[i];
#pragma unroll
            for (int i = 0; i < BV; i++) v0[i] = vw[i];
            const float kn0 = kn, vn0 = vn;
            load(it + 1, id_next);
            id_next = page_id(it + 2);
            bool alive = it < NST || wait(kv_empty + 8 * st, it / NST - 1);
            if (!__all_sync(0xffffffffu, alive)) break;
            put(sbase + C::OFF_K + st * C::KV_TILE, std::integral_constant<int, BK>{}, k0, tk);
            put(sbase + C::OFF_V + st * C::KV_TILE, std::integral_constant<int, BV>{}, v0, tv);
            if (gq == 0) {
                // The weights of a tile are multiplied by its norms whether a row attends the token or not,
                // so what 0 * norm must not turn into NaN is kept out of them: an infinite norm becomes the
                // largest number, whose weights saturate like its own; a NaN makes the rows that attend it
                // NaN at the end.  (Selecting by row in the softmax warps: 221 us instead of 205 for 8 queries
                // over 131072 tokens, 32 / 8 heads of 128.)
                float v = vn0;
                if (!(fabsf(v) <= 65504.f)) {
                    if (v != v) atomicMin(&s_nan_pos, (tile0 + it) * KT + t);
                    v = v != v ? 0.f : copysignf(FLT_MAX, v);
                }
                norms[st * 2 * KT + t] = kn0;
                norms[st * 2 * KT + KT + t] = v;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
#ifdef FTQ_TEST_WAIT_EXPIRY
            if (it == 1 && idx < 32 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) continue;
#endif
            if (lane == 0) mbar_arrive(kv_full + 8 * st);
        }
    } else {
        // ================= the MMAs
        const bool one = lane == 0;
        constexpr uint32_t kIdescS = (1u << 4) | (static_cast<uint32_t>(KT / 8) << 17) | (8u << 24);
        constexpr uint32_t kIdescO = (1u << 4) | (1u << 16) | (static_cast<uint32_t>(D / 8) << 17) | (8u << 24);
        // descriptors: the upper halves are constants, the lower ones a base and a constant
        constexpr uint32_t kHi = (1024u >> 4) | (1u << 14) | (2u << 29);
        constexpr uint32_t kLeadK = (16u >> 4) << 16, kLeadV = (static_cast<uint32_t>(KT * 128) >> 4) << 16;
        const uint32_t q_lo = ((sbase + C::OFF_Q) >> 4) | kLeadK, k_lo = ((sbase + C::OFF_K) >> 4) | kLeadK,
                       v_lo = ((sbase + C::OFF_V) >> 4) | kLeadV;
        auto pv = [&](int it) {
            const int st = it % NST;
            const uint32_t v = v_lo + st * (C::KV_TILE >> 4);
            for (int s = 0; s < n_slots; s++) {
                if (!__all_sync(0xffffffffu, wait(p_full + 8 * s, it))) return false;
                tc_fence_after();
                const uint32_t tm = tmem + s * C::COLS;
#pragma unroll
                for (int ks = 0; ks < KT / 16; ks++)
                    tc_mma_ts(one, tm, tm + C::COL_P + 8 * ks, v + ks * (2048 >> 4), kHi, kIdescO, it > 0 || ks > 0);
                if (one) tc_commit(o_done + 8 * s);
                __syncwarp();
            }
            if (one) tc_commit(kv_empty + 8 * st);
            __syncwarp();
            return true;
        };
        bool ok = true;
        for (int it = 0; it < n_tiles && ok; it++) {
            const int st = it % NST;
            const uint32_t k = k_lo + st * (C::KV_TILE >> 4);
            ok = __all_sync(0xffffffffu, wait(kv_full + 8 * st, it / NST));
            for (int s = 0; s < n_slots && ok; s++) {
                if (it > 0) ok = __all_sync(0xffffffffu, wait(s_free + 8 * s, it - 1));
                if (!ok) break;
                tc_fence_after();
                const uint32_t q = q_lo + s * (C::Q_TILE >> 4);
#pragma unroll
                for (int kb = 0; kb < D / 16; kb++)
                    tc_mma_ss(one, tmem + s * C::COLS + C::COL_S, q + ((kb >> 2) * (128 * 128) + (kb & 3) * 32) / 16,
                              k + ((kb >> 2) * (KT * 128) + (kb & 3) * 32) / 16, kHi, kIdescS, kb > 0);
                if (one) tc_commit(s_full + 8 * s);
                __syncwarp();
            }
            if (ok && it > 0) ok = pv(it - 1);
        }
        if (ok) ok = pv(n_tiles - 1);
        if (!ok) {   // nothing may be in flight when TMEM is given back
            if (one) tc_commit(drained);
            __syncwarp();
            for (int i = 0; i < kDrainSpinLimit && !mbar_try_wait(drained, 0); i++) {}
        }
    }
    __syncwarp();
    __syncthreads();
    const bool expired = s_abort != 0;
    const int bad_pos = s_bad_pos, poison = min(bad_pos, s_nan_pos);
    if (expired || poison != INT_MAX) {
        for (int r = row0 + tid; r < row_end; r += C::THREADS)
            if (expired || poison < min(p.max_seq, limit0 + r / group)) partial_row(r)[D] = __int_as_float(0x7fc00000);
        if (tid == 0 && expired) __stcg(p.errors, p.epoch);
        if (tid == 0 && bad_pos != INT_MAX) __stcg(p.errors + 1, p.epoch);
    }
    if (warp == C::SM_WARPS + C::DQ_WARPS) {
        tc_fence_after();
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
    }
}

}  // namespace ftq
