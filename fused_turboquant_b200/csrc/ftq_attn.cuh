// Split-KV decode attention over compressed K/V (fp32 arithmetic) + merge.
//
// One query token per sequence.  A CTA owns (sequence, KV head, KV chunk): it
// stages the chunk's pages into shared memory with cp.async (page ids come
// from the block table, or the pages are cut from contiguous tensors), scores
// every key in the ROTATED space against all query heads of the GQA group, so
// each packed byte is fetched once per KV head, runs an online softmax, and
// accumulates V in the rotated space.  The chunk's (max, sum, accumulator) go
// to a caller-provided workspace; the merge kernel combines the chunks and
// applies the inverse rotation once per (sequence, query head).
//
// Arithmetic follows the reference's fused formulation
// (src/fused_turboquant/kernels/triton_flash_decode.py:33-324):
//   score = knorm * scale * sum_d q_rot[d] * C_k[code_k[d]]
//   acc  += exp(score - m) * vnorm * C_v[code_v[:]]      (with the m rescale)
//   out   = inverse_rht(acc / l)
// and additionally fuses the query rotation (hf/fused_cache.py:579-581) and the
// page-table walk (vllm_plugin/cache_ops.py:151-205).
#pragma once

#include <math.h>

#include "ftq_common.cuh"

namespace ftq {

constexpr int kFlowMaxSeqs = 1024;       // sequences per launch (their prefix sums lie in shared memory)

struct AttnParams {
    const void* q;              // [L*B, Hq, D]
    // paged source
    const uint8_t* pool;        // [L][num_blocks, Hkv, page_bytes]
    int64_t pool_layer_stride;  // bytes
    const int32_t* block_table; // [B, max_blocks]
    int max_blocks;
    // contiguous source
    const uint8_t* k_codes;     // [B, Hkv, S, pdk]
    const uint16_t* k_norms;    // [B, Hkv, S]
    const uint8_t* v_codes;
    const uint16_t* v_norms;
    int S;
    const int32_t* seq_lens;    // [B] or nullptr
    int B, Hq, Hkv;
    float scale;
    int q_is_rotated;
    int q_dtype;                // kF32 / kF16 / kBF16
    int cp16;                   // contiguous source: every span 16-byte aligned
    int chunk_tokens, n_chunks, n_hpass;
    // rows (O, m, l): attn_split_kernel [L*B*Hq][n_chunks][D + 4]; attn_flow_kernel [halves of the grid][2][group][D + 4],
    // the pieces of cut units at the start and the end of each half's share
    float* partials;
    // Counters of the tensor-core kernel, which clears them itself: CTA 0 zeroes work_counter[1]
    // (CTAs that have left) and the unit counters, then stores `epoch` (unique per call, never 0) into
    // the 64-bit word at work_counter + 2; everybody checks for it before the first atomic on a
    // counter, and the last CTA to leave stores 0 there, so that a replay of the same launch, or the
    // call's next launch, does not find its own epoch.
    // work_counter[4] is the call's status word (kStatus* bits, cleared with the counters): what
    // the kernels of this call met; the host reads it on request (ftq_paged_decode_status).
    // nullptr for the contiguous entry points.
    int* work_counter;
    // the tensor-core kernel finishes the split-KV merge itself
    int* unit_counter;          // [n_units = L*B*Hkv] pieces delivered per unit
    int n_units;
    unsigned long long epoch;
    // tensor-core kernel: sequences b0 .. b0 + B - 1 of the batch's B_stride, n_layers layers; context
    // lengths are cut to max_seq; places per share at least min_share
    int n_layers, b0, B_stride, max_seq, min_share;
    void* out;                  // [L*B, Hq, D]
    int out_dtype;
    int64_t num_blocks;         // block ids are checked against it
    Codebook lk, lv;
    int shared_table;           // fp32 kernel: keys and values have the same codebook
    SignBits signs;
    float rsqrt_d;
    // tensor-core path: V centroids pre-multiplied by v_scale before the fp16 rounding
    // (lv_scaled), undone through the weights (inv_v_scale)
    Codebook lv_scaled;
    float inv_v_scale;
};

constexpr int kStatusWord = 4;         // index into AttnParams::work_counter
constexpr int kStatusBadBlock = 1;     // a block id outside [0, num_blocks) was met (its rows are NaN)
constexpr int kStatusWaitExpired = 2;  // a bounded wait of a kernel ran out (its rows are NaN)

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, int src_bytes) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_4(void* smem, const void* gmem, int src_bytes) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Copy `valid` of `total` bytes (both multiples of CP) into shared memory, zero-filling the rest.
template <int CP>
__device__ __forceinline__ void stage_span(uint8_t* dst, const uint8_t* src, int total, int valid,
                                           int tid, int nthreads) {
    for (int off = tid * CP; off < total; off += nthreads * CP) {
        int nb = valid - off;
        nb = nb < 0 ? 0 : (nb > CP ? CP : nb);
        // a zero-byte copy still needs a valid, aligned source address
        const uint8_t* s = nb > 0 ? src + off : src;
        if constexpr (CP == 16) cp_async_16(dst + off, s, nb);
        else cp_async_4(dst + off, s, nb);
    }
}

// A lane's slice of one packed vector: NB bytes starting at p (shared memory).
template <int NB>
__device__ __forceinline__ void load_code_bytes(const uint8_t* p, uint32_t (&w)[(NB + 3) / 4]) {
    if constexpr (NB == 16) {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (NB == 8) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        w[0] = v.x; w[1] = v.y;
    } else if constexpr (NB % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NB / 4; i++) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
    } else if constexpr (NB == 6) {
        const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
        w[0] = static_cast<uint32_t>(h[0]) | (static_cast<uint32_t>(h[1]) << 16);
        w[1] = h[2];
    } else if constexpr (NB == 3) {
        w[0] = static_cast<uint32_t>(p[0]) | (static_cast<uint32_t>(p[1]) << 8) |
               (static_cast<uint32_t>(p[2]) << 16);
    } else if constexpr (NB == 2) {
        w[0] = *reinterpret_cast<const uint16_t*>(p);
    } else {
        static_assert(NB == 1, "unsupported slice size");
        w[0] = p[0];
    }
}

// Code j of a little-endian stream of BITS-wide codes held in w[].
template <int BITS, int NWORDS>
__device__ __forceinline__ uint32_t extract_code(const uint32_t (&w)[NWORDS], int j) {
    const int off = j * BITS;
    const int lo = off >> 5, sh = off & 31;
    constexpr uint32_t mask = (1u << BITS) - 1u;
    if (sh + BITS <= 32) return (w[lo] >> sh) & mask;
    return __funnelshift_r(w[lo], w[lo + 1 < NWORDS ? lo + 1 : lo], sh) & mask;
}

// Shared-memory byte offset (entry * 128) of the table entry for code pair `pair`
// of a slice: bits [pair*IW, pair*IW + IW) of the little-endian stream in w[].
template <int IW, int NW>
__device__ __forceinline__ uint32_t pair_index(const uint32_t (&w)[NW], int pair) {
    constexpr uint32_t mask = ((1u << IW) - 1u) << 7;
    const int bo = pair * IW;
    const int j = bo >> 5, sh = bo & 31;
    uint32_t x;
    if (sh + IW <= 32) x = sh >= 7 ? (w[j] >> (sh - 7)) : (w[j] << (7 - sh));
    else x = __funnelshift_r(w[j], w[j + 1 < NW ? j + 1 : j], sh - 7);
    return x & mask;
}

constexpr int kTilePages = 4;
constexpr int kTileRing = 2;       // buffers of a page of a warp (three measure alike)
constexpr int kAttnThreads = 128;

template <int D>
struct AttnCfg {
    static constexpr int E = D / kOctet;
    static constexpr int GH = 64 / E;  // query heads per pass: 8 / 4 / 2 for D = 64 / 128 / 256
};

// Bound by instruction issue and its latencies at two CTAs of four warps per SM (some 230 registers a thread hold the
// queries and the accumulators; three CTAs of 168 spill: 32.7 us in place of 24.6 below).  So: a pair of codes is one
// look-up of an 8-byte entry (extracting and looking up each code took four instructions), the octet's dot products
// are added up in a tree that leaves every lane one head (a third of the shuffles, a quarter of the exponentials), and
// every warp fetches its own pages without a barrier of the CTA in the loop.  4 x 4001 tokens, 32 / 8 heads of 128,
// K4V4, contiguous: 32.8 -> 28.6 -> 24.6 us with its merge; 16 x 3000, 8 / 8 heads 108 -> 52; paged, 16 x 2000, 32 / 8
// heads, with the store 66 -> 56.  Each sum is made in the order it had.
// PAGED: pages come from the pool through the block table; otherwise they are
// cut from contiguous [B,Hkv,S,*] tensors (cp.async granule 16 bytes when every
// span is 16-byte aligned, p.cp16, else 4).
template <int D, int BK, int BV, bool PAGED>
__global__ void __launch_bounds__(kAttnThreads)
attn_split_kernel(const AttnParams p) {
    constexpr int E = AttnCfg<D>::E;
    constexpr int GH = AttnCfg<D>::GH;
    constexpr int PDK = packed_dim(D, BK), PDV = packed_dim(D, BV);
    constexpr int NBK = PDK / kOctet, NBV = PDV / kOctet;  // bytes per lane per vector
    constexpr int OFF_KN = kPageTokens * PDK;
    constexpr int OFF_VC = OFF_KN + 2 * kPageTokens;
    constexpr int OFF_VN = OFF_VC + kPageTokens * PDV;
    constexpr int PAGE_BYTES = OFF_VN + 2 * kPageTokens;
    constexpr int TILE_BYTES = kTilePages * PAGE_BYTES;
    constexpr int ROW = D + 4;  // floats per partial row: acc[D], m, l, pad, pad

    // the tile ring doubles as the cross-warp merge area once the loop is over
    constexpr int MERGE_BYTES = 4 * GH * (D + 2) * 4;
    constexpr int RING_BYTES =
        ((kTileRing * TILE_BYTES > MERGE_BYTES ? kTileRing * TILE_BYTES : MERGE_BYTES) + 15) / 16 * 16;

    extern __shared__ __align__(16) uint8_t smem_raw[];
    uint8_t* tiles = smem_raw;                                   // RING_BYTES
    float* qs = reinterpret_cast<float*>(smem_raw + RING_BYTES);      // [GH][D]
    // dequantisation tables: an entry is the two centroids of a pair of codes, sixteen copies of it a row, so that a half
    // warp's 8-byte look-ups never meet in a bank
    constexpr int TAB_K = RING_BYTES + GH * D * 4, TK_BYTES = (1 << (2 * BK)) * 128;
    const int tab_v = TAB_K + (p.shared_table ? 0 : TK_BYTES);

    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int t = lane & 7, o = lane >> 3;

    const int chunk = blockIdx.x;
    const int hkv = blockIdx.y / p.n_hpass;
    const int hp = blockIdx.y - hkv * p.n_hpass;
    const int lb = blockIdx.z;
    const int layer = lb / p.B;
    const int b = lb - layer * p.B;
    const int group = p.Hq / p.Hkv;
    const int h0 = hp * GH;
    const int nh = min(GH, group - h0);

    int seq_len = p.seq_lens ? p.seq_lens[b] : p.S;
    if (!PAGED) seq_len = min(seq_len, p.S);
    const int t0 = chunk * p.chunk_tokens;
    const int t1 = min(seq_len, t0 + p.chunk_tokens);
    float* prow = p.partials +
                  ((static_cast<int64_t>(lb) * p.Hq + hkv * group + h0) * p.n_chunks + chunk) * ROW;
    const int64_t prow_head_stride = static_cast<int64_t>(p.n_chunks) * ROW;
    if (t0 >= t1) {
        if (tid < nh) {
            prow[tid * prow_head_stride + D] = -INFINITY;
            prow[tid * prow_head_stride + D + 1] = 0.f;
        }
        return;
    }

    const uint8_t* pool = PAGED ? p.pool + layer * p.pool_layer_stride : nullptr;
    const int32_t* btab = PAGED ? p.block_table + static_cast<int64_t>(b) * p.max_blocks : nullptr;
    const int64_t cbase = (static_cast<int64_t>(b) * p.Hkv + hkv) * p.S;

    // A warp's page of tile ti (tokens t0 + 64 ti + 16 warp ..) on its way to the warp's buffer: nobody else reads it, so
    // the loop has no barrier of the whole CTA.  The norms of a contiguous source lie on 2-byte boundaries: a lane keeps
    // the one it loads until the page is waited for.
    bool bad_block = false;
    uint16_t norm[kTileRing] = {};
    auto issue_page = [&](int ti, int buf) {
        const int ts = t0 + ti * (kTilePages * kPageTokens) + warp * kPageTokens;
        if (ts < t1) {
            uint8_t* pd = tiles + buf * TILE_BYTES + warp * PAGE_BYTES;
            if constexpr (PAGED) {
                // a block id outside the pool is never dereferenced: block 0 stands in and the
                // chunk's result is replaced by NaN below
                int64_t blk = btab[ts / kPageTokens];
                if (static_cast<uint64_t>(blk) >= static_cast<uint64_t>(p.num_blocks)) {
                    blk = 0;
                    bad_block = true;
                }
                const uint8_t* src = pool + (blk * p.Hkv + hkv) * PAGE_BYTES;
                stage_span<16>(pd, src, PAGE_BYTES, PAGE_BYTES, lane, 32);
            } else {
                const int ntok = min(kPageTokens, t1 - ts);
                if (p.cp16) {
                    stage_span<16>(pd, p.k_codes + (cbase + ts) * PDK, kPageTokens * PDK,
                                   ntok * PDK, lane, 32);
                    stage_span<16>(pd + OFF_VC, p.v_codes + (cbase + ts) * PDV, kPageTokens * PDV,
                                   ntok * PDV, lane, 32);
                } else {
                    stage_span<4>(pd, p.k_codes + (cbase + ts) * PDK, kPageTokens * PDK,
                                  ntok * PDK, lane, 32);
                    stage_span<4>(pd + OFF_VC, p.v_codes + (cbase + ts) * PDV, kPageTokens * PDV,
                                  ntok * PDV, lane, 32);
                }
                const int tk = lane & (kPageTokens - 1);
                norm[buf] = tk < ntok ? (lane >= kPageTokens ? p.v_norms : p.k_norms)[cbase + ts + tk] : uint16_t(0);
            }
        }
        cp_async_commit();
    };

    const int n_tiles = (t1 - t0 + kTilePages * kPageTokens - 1) / (kTilePages * kPageTokens);
#pragma unroll
    for (int i = 0; i < kTileRing - 1; i++) issue_page(i, i);

    // ---- prologue: tables and the rotated, pre-scaled queries of this pass
    auto build = [&](int at, const Codebook& levels, int bits) {
        // (a thread's two copies of an entry: one 16-byte store)
        for (int i = tid; i < 8 << (2 * bits); i += kAttnThreads) {
            const int e = i >> 3;
            const float lo = levels.v[e & ((1 << bits) - 1)], hi = levels.v[e >> bits];
            *reinterpret_cast<float4*>(smem_raw + at + i * 16) = make_float4(lo, hi, lo, hi);
        }
    };
    build(TAB_K, p.lk, BK);
    if (!p.shared_table) build(tab_v, p.lv, BV);
    {
        const int hh = warp * 4 + o;  // one octet rotates one query head (GH <= 8 < 16 octets)
        const bool hv = hh < nh;
        const int64_t qoff =
            (static_cast<int64_t>(lb) * p.Hq + hkv * group + h0 + (hv ? hh : 0)) * D;
        float a[E];
#pragma unroll
        for (int i = 0; i < E / 8; i++) {
            float tmp[8];
            const int64_t eo = qoff + 8 * (t + 8 * i);
            if (p.q_dtype == kF32) load8<float>(static_cast<const float*>(p.q) + eo, tmp);
            else if (p.q_dtype == kBF16)
                load8<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(p.q) + eo, tmp);
            else load8<__half>(static_cast<const __half*>(p.q) + eo, tmp);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const uint32_t m = p.q_is_rotated ? 0u : sign_mask(p.signs, load_coord(t, 8 * i + c));
                a[8 * i + c] = __uint_as_float(__float_as_uint(tmp[c]) ^ m);
            }
        }
        if (p.q_is_rotated) {
            if (hh < GH) {
#pragma unroll
                for (int r = 0; r < E; r++)
                    qs[hh * D + load_coord(t, r)] = hv ? a[r] * p.scale : 0.f;
            }
        } else {
            octet_fwht<E>(a, lane);
            if (hh < GH) {
#pragma unroll
                for (int k = 0; k < E; k++)
                    qs[hh * D + t + 8 * k] = hv ? a[k] * p.rsqrt_d * p.scale : 0.f;
            }
        }
    }
    __syncthreads();

    // queries and accumulators as pairs of adjacent coordinates: packed fp32 FMAs (two independent IEEE
    // FMAs per instruction)
    constexpr int EP = E / 2;
    u64 qr[GH][EP], acc[GH][EP];
#pragma unroll
    for (int h = 0; h < GH; h++)
#pragma unroll
        for (int i = 0; i < EP; i++)
            qr[h][i] = pk2(qs[h * D + t * E + 2 * i], qs[h * D + t * E + 2 * i + 1]);

    // Softmax state of ONE head, that of the lane: the dot products of an octet's lanes are added up in a tree that leaves
    // each lane with a head of its own (for fewer heads than lanes, several with the same).
    constexpr int HB = GH == 8 ? 3 : GH == 4 ? 2 : 1;      // bits of a lane's number that say its head
    int my_head = 0;
#pragma unroll
    for (int i = 0; i < HB; i++) my_head |= ((t >> i) & 1) << (HB - 1 - i);
    auto lane_of = [&](int h) {   // a lane of this octet with head h
        int r = lane & 24;
#pragma unroll
        for (int i = 0; i < HB; i++) r |= ((h >> (HB - 1 - i)) & 1) << i;
        return r;
    };
    float m_run = -INFINITY, l_run = 0.f;
#pragma unroll
    for (int h = 0; h < GH; h++)
#pragma unroll
        for (int i = 0; i < EP; i++) acc[h][i] = pk2(0.f, 0.f);
    // centroids of the lane's code pair `pair`
    const uint32_t col = (lane & 15) * 8;
    auto look_up = [&](int at, uint32_t index) { return *reinterpret_cast<const u64*>(smem_raw + at + (index | col)); };

    // ---- main loop over 64-token tiles, a page per warp
    for (int ti0 = 0; ti0 < n_tiles; ti0 += kTileRing) {
#pragma unroll
      for (int buf = 0; buf < kTileRing; buf++) {     // (buffer numbers known to the compiler: `norm` stays in registers)
        const int ti = ti0 + buf;
        if (ti >= n_tiles) break;
        issue_page(ti + kTileRing - 1, (buf + kTileRing - 1) % kTileRing);
        cp_async_wait<kTileRing - 1>();
        uint8_t* page = tiles + buf * TILE_BYTES + warp * PAGE_BYTES;
        if constexpr (!PAGED)
            reinterpret_cast<uint16_t*>(page + (lane >= kPageTokens ? OFF_VN : OFF_KN))[lane & (kPageTokens - 1)] = norm[buf];
        __syncwarp();

        const int ts = t0 + ti * (kTilePages * kPageTokens) + warp * kPageTokens;
        if (ts < t1) {  // warp-uniform
            const int ntok = min(kPageTokens, t1 - ts);

            float sc[4];
#pragma unroll
            for (int step = 0; step < 4; step++) {
                const int tk = step * 4 + o;
                uint32_t w[(NBK + 3) / 4];
                load_code_bytes<NBK>(page + tk * PDK + t * NBK, w);
                const float kn =
                    __half2float(reinterpret_cast<const __half*>(page + OFF_KN)[tk]);
                u64 kv[EP];
#pragma unroll
                for (int i = 0; i < EP; i++) kv[i] = look_up(TAB_K, pair_index<2 * BK>(w, i));
                float d[GH];
#pragma unroll
                for (int h = 0; h < GH; h++) {
                    u64 d2 = pk2(0.f, 0.f);
#pragma unroll
                    for (int i = 0; i < EP; i++) d2 = fma2(qr[h][i], kv[i], d2);
                    float d0, d1;
                    upk2(d2, d0, d1);
                    d[h] = d0 + d1;
                }
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const int n = GH >> (i + 1);
                    if (n > 0) {
                        const bool up = (t >> i) & 1;   // this lane keeps the upper half of the heads
#pragma unroll
                        for (int k = 0; k < (n > 0 ? n : 1); k++) {
                            const float give = up ? d[k] : d[k + n], keep = up ? d[k + n] : d[k];
                            d[k] = keep + __shfl_xor_sync(0xffffffffu, give, 1 << i);
                        }
                    } else {
                        d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1 << i);
                    }
                }
                sc[step] = tk < ntok ? d[0] * kn : -INFINITY;
            }

            float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            // (a maximum that stays leaves the accumulators as they are: the factor is one)
            if (__any_sync(0xffffffffu, !(mx <= m_run))) {
                const float m_new = fmaxf(m_run, mx);  // finite: token 0 of the page is valid
                const float corr = m_run == -INFINITY ? 0.f : __expf(m_run - m_new);
                m_run = m_new;
                l_run *= corr;
#pragma unroll
                for (int h = 0; h < GH; h++) {
                    const float c = __shfl_sync(0xffffffffu, corr, lane_of(h));
                    const u64 corr2 = pk2(c, c);
#pragma unroll
                    for (int i = 0; i < EP; i++) acc[h][i] = mul2(acc[h][i], corr2);
                }
            }
            float wp[4], ls = 0.f;
#pragma unroll
            for (int step = 0; step < 4; step++) {
                wp[step] = sc[step] == -INFINITY ? 0.f : __expf(sc[step] - m_run);
                ls += wp[step];
            }
            l_run += ls;

#pragma unroll
            for (int step = 0; step < 4; step++) {
                const int tk = step * 4 + o;
                uint32_t w[(NBV + 3) / 4];
                // pool pages store a V row with its halves exchanged for tokens with bit 1 set
                const int vt = PAGED ? (t ^ ((tk & 2) << 1)) : t;
                load_code_bytes<NBV>(page + OFF_VC + tk * PDV + vt * NBV, w);
                const float vn = __half2float(reinterpret_cast<const __half*>(page + OFF_VN)[tk]);
                const float wgt = tk < ntok ? wp[step] * vn : 0.f;
                u64 vv[EP];
#pragma unroll
                for (int i = 0; i < EP; i++) vv[i] = look_up(tab_v, pair_index<2 * BV>(w, i));
#pragma unroll
                for (int h = 0; h < GH; h++) {
                    const float wh = __shfl_sync(0xffffffffu, wgt, lane_of(h));
                    const u64 wgt2 = pk2(wh, wh);
#pragma unroll
                    for (int i = 0; i < EP; i++) acc[h][i] = fma2(wgt2, vv[i], acc[h][i]);
                }
            }
        }
        __syncwarp();   // (the buffer is requested again in the next round)
      }
    }

    // ---- combine the 4 octets of each warp, then the 4 warps through shared memory
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 8);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 16);
#pragma unroll
    for (int h = 0; h < GH; h++) {
#pragma unroll
        for (int i = 0; i < EP; i++) {
            acc[h][i] = add2(acc[h][i], __shfl_xor_sync(0xffffffffu, acc[h][i], 8));
            acc[h][i] = add2(acc[h][i], __shfl_xor_sync(0xffffffffu, acc[h][i], 16));
        }
    }
    bad_block = __syncthreads_or(bad_block) != 0;    // (nobody reads the tiles any more)
    float* wacc = reinterpret_cast<float*>(tiles);   // [4][GH][D]
    float* wm = wacc + 4 * GH * D;                   // [4][GH]
    float* wl = wm + 4 * GH;                         // [4][GH]
    if (o == 0) {
#pragma unroll
        for (int h = 0; h < GH; h++) {
#pragma unroll
            for (int i = 0; i < EP; i++)
                *reinterpret_cast<u64*>(wacc + (warp * GH + h) * D + t * E + 2 * i) = acc[h][i];
        }
        if (t < GH) {   // (the lanes with the heads' first copies)
            // (a score that is not a number is in the sum of the weights, but no maximum knows it)
            wm[warp * GH + my_head] = l_run != l_run ? l_run : m_run;
            wl[warp * GH + my_head] = l_run;
        }
    }
    __syncthreads();
    for (int idx = tid; idx < nh * D; idx += kAttnThreads) {
        const int h = idx / D, d = idx - h * D;
        float M = -INFINITY;
#pragma unroll
        for (int w2 = 0; w2 < 4; w2++) M = fmaxf(M, wm[w2 * GH + h]);
        float a = 0.f, l = 0.f;
#pragma unroll
        for (int w2 = 0; w2 < 4; w2++) {
            const float mw = wm[w2 * GH + h];
            if (mw != -INFINITY) {
                const float f = __expf(mw - M);
                a = fmaf(wacc[(w2 * GH + h) * D + d], f, a);
                l = fmaf(wl[w2 * GH + h], f, l);
            }
        }
        prow[h * prow_head_stride + d] = a;
        if (d == 0) {
            if (bad_block && h == 0 && p.work_counter) atomicOr(p.work_counter + kStatusWord, kStatusBadBlock);
            if (bad_block || l != l) M = __int_as_float(0x7fc00000);
            prow[h * prow_head_stride + D] = M;
            prow[h * prow_head_stride + D + 1] = l;
        }
    }
}

// Merge the chunk partials of one (layer, sequence, query head), normalise,
// rotate back to the original space (inverse_randomized_hadamard,
// core/hadamard.py:93-100) and store.  OCTETS octets per output vector: each takes every OCTETS-th
// chunk's row, and their sums are added up with shuffles.  What bounds it is the latency of the
// rows' loads, so the loop has nothing that keeps the next row's loads from being issued.  (An octet
// per vector with a branch per row took 23 us of the 65 us of a call with 128 vectors of 32 chunks.)
// `st` (optional): the error words of the kernel before (their epoch: unique per launch) become the call's status word.
struct MergeStatus {
    int* status;
    unsigned long long* errors;   // [2]: expired waits, bad block ids
    unsigned long long epoch;
};
template <int D, typename OT, int OCTETS>
__global__ void __launch_bounds__(128)
attn_merge_kernel(const float* partials, OT* __restrict__ out,   // (only the output is restrict: see load8)
                  const int32_t* seq_lens, int S, int B, int Hq, int n_chunks,
                  int chunk_tokens, int64_t n_vec, SignBits signs, float rsqrt_d, MergeStatus st) {
    constexpr int E = D / kOctet;
    constexpr int ROW = D + 4;
    const int lane = threadIdx.x & 31;
    const int t = lane & 7, o = (lane >> 3) & (OCTETS - 1);
    after_previous_kernel();   // the rows are complete
    if (st.status && blockIdx.x == 0 && threadIdx.x == 0) {
        *st.status = (__ldcg(st.errors) == st.epoch ? kStatusWaitExpired : 0) | (__ldcg(st.errors + 1) == st.epoch ? kStatusBadBlock : 0);
        st.errors[0] = st.errors[1] = 0ull;   // (a replayed launch has the same epoch)
    }
    const int64_t at = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / (8 * OCTETS);
    const int64_t v = at < n_vec ? at : n_vec - 1;   // (octets left over repeat the last vector)
    const int b = static_cast<int>((v / Hq) % B);
    const int len = seq_lens ? (S > 0 ? min(seq_lens[b], S) : seq_lens[b]) : S;
    const int nc = min(n_chunks, (len + chunk_tokens - 1) / chunk_tokens);
    const float* rows = partials + v * n_chunks * ROW;
    float M = -INFINITY;
    for (int c = 8 * o + t; c < nc; c += 8 * OCTETS) M = fmaxf(M, rows[static_cast<int64_t>(c) * ROW + D]);
#pragma unroll
    for (int m = 1; m < 8 * OCTETS; m <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, m));
    float a[E];
#pragma unroll
    for (int r = 0; r < E; r++) a[r] = 0.f;
    float L = 0.f;
#pragma unroll 2
    for (int c = o; c < nc; c += OCTETS) {
        const float* row = rows + static_cast<int64_t>(c) * ROW;
        const float mc = row[D];
        const bool live = mc != -INFINITY;   // (the vector of a dead chunk's row was never written)
        const float f = live ? __expf(mc - M) : 0.f;
        L = live ? fmaf(row[D + 1], f, L) : L;
#pragma unroll
        for (int i = 0; i < E / 8; i++) {
            float tmp[8];
            load8<float>(row + 8 * (t + 8 * i), tmp);
#pragma unroll
            for (int cc = 0; cc < 8; cc++) a[8 * i + cc] = live ? fmaf(tmp[cc], f, a[8 * i + cc]) : a[8 * i + cc];
        }
    }
#pragma unroll
    for (int m = 8; m < 8 * OCTETS; m <<= 1) {
        L += __shfl_xor_sync(0xffffffffu, L, m);
#pragma unroll
        for (int r = 0; r < E; r++) a[r] += __shfl_xor_sync(0xffffffffu, a[r], m);
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll
    for (int r = 0; r < E; r++) a[r] *= inv;
    octet_fwht<E>(a, lane);
#pragma unroll
    for (int k = 0; k < E; k++) {
        if (at >= n_vec || (k & (OCTETS - 1)) != o) continue;   // (every octet of the vector holds the result and stores its part)
        const float r = a[k] * rsqrt_d;
        out[v * D + t + 8 * k] =
            from_float<OT>(__uint_as_float(__float_as_uint(r) ^ sign_mask(signs, t + 8 * k)));
    }
}

}  // namespace ftq
