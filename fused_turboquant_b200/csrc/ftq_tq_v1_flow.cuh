// vLLM-v1 slot format, decode stage 1: every CTA streams an equal share of the batch's pages, all KV
// heads of a page at once.
//
// Same result as tq_split_kernel (ftq_tq_v1.cuh), i.e. the reference's `_tq_decode_stage1_offset`
// (src/fused_turboquant/vllm_plugin/triton_decode_offset.py:42-444), partials in the same
// [B, Hq, splits, D + 1] layout.
//
// The slots of one head start on 2-byte boundaries and no bulk copy can fetch them, but the 16 tokens of
// ALL heads of a page are one contiguous, 16-byte aligned span of a [block, position, head, slot] cache.  So a CTA
// works on whole pages: warp 16 (the producer) fetches them by 1-D bulk copies (TMA) into a ring in
// shared memory, and of the other sixteen warps warp w works on KV head w % Hkv of every (16 / Hkv)-th
// page, with an online-softmax state of its own.  The warps of a head fold their states at the end of a
// piece; nothing synchronises the whole CTA after the set-up.  (A warp that copied the slots of its own
// pages word by word through registers spent 722 instructions a page and head on it: 32 x 8192 tokens of
// 8 heads, 4-bit keys and values, took 182 us; this way 113.)
//
// Work: the pages of a layer's (sequence, split) units lie in one line, each unit's behind piece_cost places without a page
// (what a piece costs beside its pages: queries, the fold, the rows), and the line is cut into equal shares, at most one per
// SM; a share's part of a unit that holds no page is no piece.  (Shares of pages alone gave the CTAs with the short contexts
// of a ragged batch many times the pieces of the others: 64 sequences of 62 to 16000 tokens, 8 heads of 128, 4-bit codes, 242 us
// and now 120 in this kernel.)  And the CTAs of the persistent grid take the shares of all layers in turn.  (Shares of single layers: a layer's
// result does not depend on which others are in the call.)  A piece of a unit that a share's end cuts leaves its rows in the
// workspace (two row blocks per share: its first and its last piece can be parts of units) and the merge kernel
// puts them together; a whole unit's rows go to mid_o.  Splits keep their borders in tokens, pages the
// cache's: the page that a border runs through belongs to both units.
//
// Page i of a piece is the work of the (i mod 16 / Hkv)-th warp of each head, and these warps have a part of the ring to
// themselves: every waiter sees each phase of its barriers.
//
// Every wait is bounded; a wait that runs out sets the workspace's share to 0, which makes the merge kernel
// return NaN.  Block ids outside the
// cache are never dereferenced (block 0 stands in, the unit's lse becomes NaN).
#pragma once

#include "ftq_attn_mma.cuh"
#include "ftq_tq_v1.cuh"

namespace ftq {

// mbar_wait for the producer, with a pause between polls: it has time, the ring is some pages ahead, and its polls without one
// were a tenth of the kernel's instructions.  (For the warps that compute a pause made no difference: 122.3 us with, 122.2
// without for 32 x 8192 tokens.)
__device__ __forceinline__ bool mbar_wait_idle(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kMbarSpinLimit; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        __nanosleep(32);
    }
    return false;
}
// A constant that stays in its register (an instruction has room for one immediate).
__device__ __forceinline__ uint32_t in_register(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}

// What the warps of a CTA hear about a piece.
struct TqPiece {
    int n;              // pages (0: no more pieces)
    int row, sid;       // (layer, sequence) row, split
    int lo, hi;         // tokens attended, relative to the piece's first page
    int block;          // row block of the workspace, or -1: the whole unit, rows of mid_o
};

// ---- arithmetic of one warp on one head of a page, Lloyd-Max key codes and uniform value codes of 2 to 4
// bits.  Fragment maps (lane = 4 g + tg):
//   S: A rows g, g + 8 = tokens g, g + 8; 4-bit codes: k-blocks 2 j, 2 j + 1 are the bytes of word tg + 4 j of the
//      row, so that the eight rows of a load fall into distinct banks; else slices of D / 4 coordinates
//   O^T: A rows = coordinates, k = (token, parity) for at most four heads, tokens for five to eight; the lane's tokens
//      are 2 tg, 2 tg + 1, 2 tg + 8, 2 tg + 9; 4-bit codes: words g and g + 8 of the rows, else slices of
//      D / 8 coordinates
// A head's slots start 0 or 2 bytes behind a word boundary, all alike (a token's bytes are a multiple of 4).  4-bit rows are not
// realigned: the codes are read as the aligned words hold them, the two halves of the words at the ends put together, and the coordinates of the query
// fragments and of the output follow.
// Values are code * scale + zero, codes centred (see ftq_tq_v1_mma.cuh).
// Precision: a rotated query is the sum of two fp16 numbers, hi + lo / 2^11, the lo parts in the columns that hold each of at
// most four heads a second time, or by an MMA more for five to eight heads.  A warp has four times the pages of an item
// kernel's warp under one reference maximum, and the weight of the token that sets it is the one that fp16 does not round; with
// queries of one fp16 number the mean error against 64 bits was 1.03 to 1.08 of the item kernels' (splits of 128 to 1250 tokens),
// with both it is 0.57 to 0.72 (32 x 2000 tokens 50.4 us and now 51.5).
template <int D_, int KB, int VB, int NH_>
struct TqCodes {
    static constexpr int D = D_, NH = NH_, HL = NH_, NKB = D / 16;
    static constexpr int PDK = D * KB / 8, PDV = D * VB / 8;
    static constexpr int KSB = PDK / 4, VSB = PDV / 8, KW = (KSB + 3) / 4, VW = (VSB + 3) / 4;
    static constexpr int IWK = 2 * KB, IWV = 2 * VB;
    static constexpr int OFF_VC = PDK + 2, OFF_SC = PDK + 2 + PDV, USED = OFF_SC + 4;
    static constexpr bool WINDOW = KB == 4;                      // 64 KB byte table of the key centroids
    static constexpr int TKS = KB == 4 ? 0 : (1 << IWK) * 128;   // small tables, aligned to their size (keys: two)
    static constexpr int TVS = VB == 4 ? 0 : (1 << IWV) * 128;
    static constexpr int OL = NH == 1 ? D / 8 : D / 4;           // output floats of a lane
    static constexpr float kCtr = VB == 4 ? 8.f : 0.5f * ((1 << VB) - 1);

    static constexpr int FLUSH = 0;
    static constexpr float kLo = 2048.f, kInvLo = 1.f / 2048.f;
    uint32_t qb[NKB][2];
    uint32_t q_lo;        // NH = 2: where the lane's lo parts are
    float m_run[HL], l_run[HL], z_run[HL], oacc[OL / 4][4];
    float s_ref, up;    // largest value scale so far as a power of two; weights are rounded times up
    uint32_t lk_lane, lv_lane;
    uint32_t magic, c_sub, c_mul, c_add;   // of centred()
    int mis;        // the head's slots start 2 * mis bytes behind a word boundary

    // Key tables: 32 copies of the fp16 centroids of two adjacent codes, and of the sum of their squares (byte-indexed: the
    // halves of rows of 256 bytes).
    static __device__ __forceinline__ void init_tables(const TqDecodeParams& p, uint32_t* window, uint32_t* tk,
                                                       uint32_t* tv, int tid, int threads) {
        auto pack = [](float lo, float hi) {
            const __half2 h = __floats2half2_rn(lo, hi);
            return *reinterpret_cast<const uint32_t*>(&h);
        };
        for (int i = tid; i < (1 << IWK) * 32; i += threads) {
            const int e = i >> 5;
            const uint32_t two = pack(p.centroids.v[e & ((1 << KB) - 1)], p.centroids.v[e >> KB]);
            const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&two));
            const uint32_t squares = __float_as_uint(fmaf(c.x, c.x, c.y * c.y));
            if constexpr (KB == 4) {
                window[e * 64 + (i & 31)] = two;
                window[e * 64 + 32 + (i & 31)] = squares;
            } else {
                tk[i] = two;
                tk[TKS / 4 + i] = squares;
            }
        }
        for (int i = tid; i < TVS / 4; i += threads) {
            const int e = i >> 5;
            tv[i] = pack(static_cast<float>(e & ((1 << VB) - 1)) - kCtr, static_cast<float>(e >> VB) - kCtr);
        }
    }
    __device__ __forceinline__ void init(uint32_t window, uint32_t tk, uint32_t tv, int lane, int mis_) {
        lk_lane = (KB == 4 ? window : tk) | (lane * 4);
        lv_lane = tv | (lane * 4);
        mis = mis_;
        auto twice = [](float x) {
            const __half2 h = __floats2half2_rn(x, x);
            return in_register(*reinterpret_cast<const uint32_t*>(&h));
        };
        magic = in_register(0x64006400u);
        c_sub = twice(1024.f + kCtr);
        c_mul = twice(0.0625f);
        c_add = twice(-(64.f + kCtr));
    }

    // queries of the head's group, rotated and pre-scaled, in qs[4 * NH][D + 4]
    __device__ __forceinline__ void rotate(const TqDecodeParams& p, float* qs, int64_t head0, int group, int lane) {
        constexpr int E = D / kOctet;
        const int t8 = lane & 7;
#pragma unroll
        for (int x = 0; x < NH; x++) {
            const int hh = 4 * x + (lane >> 3);
            const bool hv = hh < group;
            const int64_t qoff = (head0 + (hv ? hh : 0)) * D;
            float a[E];
#pragma unroll
            for (int i = 0; i < E / 8; i++) {
                float tmp[8];
                const int64_t eo = qoff + 8 * (t8 + 8 * i);
                if (p.q_dtype == kBF16) load8<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(p.q) + eo, tmp);
                else load8<__half>(static_cast<const __half*>(p.q) + eo, tmp);
#pragma unroll
                for (int c = 0; c < 8; c++) a[8 * i + c] = tmp[c];
            }
            octet_fwht<E>(a, lane);
#pragma unroll
            for (int k = 0; k < E; k++)
                qs[hh * (D + 4) + t8 + 8 * k] = hv ? a[k] * p.rsqrt_d * (p.scale * kLog2e) : 0.f;
        }
    }
    // (for five to eight heads the lo parts take the queries' place in qs)
    __device__ __forceinline__ void begin(float* qs, int lane) {
        const int g = lane >> 2, tg = lane & 3;
        const int head = NH == 1 ? g >> 1 : g;
        auto pack = [](float lo, float hi) {
            const __half2 h = __floats2half2_rn(lo, hi);
            return *reinterpret_cast<const uint32_t*>(&h);
        };
        auto residual = [](float x) { return (x - __half2float(__float2half_rn(x))) * kLo; };
        uint32_t lo[NKB][2];
#pragma unroll
        for (int kb = 0; kb < NKB; kb++) {
            int coord = (D / 4) * tg + 4 * kb;
            if constexpr (KB == 4) {
                coord = (8 * (tg + 4 * (kb >> 1)) + 4 * (kb & 1) - 4 * mis) & (D - 1);
            }
            const float4 q4 = *reinterpret_cast<const float4*>(qs + head * (D + 4) + coord);
            qb[kb][0] = pack(q4.x, q4.y);
            qb[kb][1] = pack(q4.z, q4.w);
            lo[kb][0] = pack(residual(q4.x), residual(q4.y));
            lo[kb][1] = pack(residual(q4.z), residual(q4.w));
            if (NH == 1 && (g & 1)) {
                qb[kb][0] = lo[kb][0];
                qb[kb][1] = lo[kb][1];
            }
        }
        if constexpr (NH == 2) {
            __syncwarp();
            uint2* const at = reinterpret_cast<uint2*>(qs) + lane;
#pragma unroll
            for (int kb = 0; kb < NKB; kb++) at[32 * kb] = make_uint2(lo[kb][0], lo[kb][1]);
            q_lo = static_cast<uint32_t>(__cvta_generic_to_shared(at));
        }
#pragma unroll
        for (int h = 0; h < HL; h++) {
            m_run[h] = -INFINITY;
            l_run[h] = z_run[h] = 0.f;
        }
        s_ref = 0.f;
        up = 1.f;
#pragma unroll
        for (int i = 0; i < OL / 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) oacc[i][j] = 0.f;
    }

    // SB bytes at the (2-byte aligned) shared address `at` -> ceil(SB / 4) words
    template <int SB>
    static __device__ __forceinline__ void load_bytes(uint32_t at, uint32_t (&out)[(SB + 3) / 4]) {
        constexpr int NW = (SB + 3) / 4;
        const uint32_t base = at & ~3u, sh = 8u * (at & 3u);
        uint32_t w[NW + 1];
#pragma unroll
        for (int j = 0; j <= NW; j++) w[j] = lds32(base + 4 * j);
#pragma unroll
        for (int j = 0; j < NW; j++) out[j] = __funnelshift_r(w[j], w[j + 1], sh);
    }
    // The head's slots of a page: token 0 at `page`, ts bytes (a multiple of 4) apart; tokens [lo, hi) count.
    __device__ __forceinline__ void page(uint32_t page, uint32_t ts, int lo, int hi, bool norm_correction, int lane) {
        const int g = lane >> 2, tg = lane & 3;
        uint32_t ka[KW], kb_[KW];
        float kna, knb;
        uint32_t sca, scb;     // scale | zero of the lane's two tokens
        const uint32_t rowa = (page & ~3u) + g * ts, rowb = rowa + 8 * ts;
        if constexpr (KB == 4) {
            // words as they lie; word 0 gets the row's last two bytes in its lower half where the row starts in its
            // middle.  The word behind the codes holds those bytes and the norm, or the norm first.
            const uint32_t sel = mis && tg == 0 ? 0x3254u : 0x3210u, sel_n = mis ? 0x4432u : 0x4410u;
#pragma unroll
            for (int j = 0; j < KW; j++) {
                ka[j] = lds32(rowa + 4 * tg + 16 * j);
                kb_[j] = lds32(rowb + 4 * tg + 16 * j);
            }
            const uint32_t xa = lds32(rowa + PDK), xb = lds32(rowb + PDK);
            ka[0] = __byte_perm(ka[0], xa, sel);
            kb_[0] = __byte_perm(kb_[0], xb, sel);
            kna = half_bits_to_float(__byte_perm(xa, 0u, sel_n));
            knb = half_bits_to_float(__byte_perm(xb, 0u, sel_n));
        } else {
            const uint32_t ra = rowa + 2 * mis, rb = rowb + 2 * mis;
            load_bytes<KSB>(ra + KSB * tg, ka);
            load_bytes<KSB>(rb + KSB * tg, kb_);
            unsigned short na, nb;
            asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(na) : "r"(ra + PDK));
            asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(nb) : "r"(rb + PDK));
            kna = half_bits_to_float(na);
            knb = half_bits_to_float(nb);
        }
        const uint32_t at = OFF_SC - 2 + 4 * mis, sh = mis ? 0u : 16u;
        sca = __funnelshift_r(lds32(rowa + at), lds32(rowa + at + 4), sh);
        scb = __funnelshift_r(lds32(rowb + at), lds32(rowb + at + 4), sh);

        // ---- S = K.Q^T; with norm correction the sum of the squared centroids of the two tokens.  (From a second look-up per
        // pair of codes: the key tile times itself, whose diagonal holds the sums, kept the tensor pipe as busy as the
        // issue slots.)
        float c[NH + 1][4];   // (NH = 2: two chains of the hi parts and one of the lo parts)
        if (norm_correction) {   // (uniform)
            u64 n2 = pk2(0.f, 0.f);
            scores<true>(ka, kb_, c, n2);
            n2 = add2(n2, __shfl_xor_sync(0xffffffffu, n2, 1));
            n2 = add2(n2, __shfl_xor_sync(0xffffffffu, n2, 2));
            float na, nb;
            upk2(n2, na, nb);
            kna *= rsqrtf(na + 1e-16f);
            knb *= rsqrtf(nb + 1e-16f);
        } else {
            u64 n2 = 0;
            scores<false>(ka, kb_, c, n2);
        }

        if (lo <= 0 && hi >= kPageTokens) attend<true>(page, ts, lo, hi, lane, c, kna, knb, sca, scb);
        else attend<false>(page, ts, lo, hi, lane, c, kna, knb, sca, scb);
    }

    template <bool NC>
    __device__ __forceinline__ void scores(const uint32_t (&ka)[KW], const uint32_t (&kb_)[KW], float (&c)[NH + 1][4], u64& n2) const {
        constexpr uint32_t SQ = KB == 4 ? 128u : TKS;   // from an entry to its squares
        u64 other = pk2(0.f, 0.f);
#pragma unroll
        for (int kb = 0; kb < NKB; kb++) {
            const uint32_t e0 = entry_addr<IWK>(ka, 2 * kb, lk_lane), e1 = entry_addr<IWK>(kb_, 2 * kb, lk_lane);
            const uint32_t e2 = entry_addr<IWK>(ka, 2 * kb + 1, lk_lane), e3 = entry_addr<IWK>(kb_, 2 * kb + 1, lk_lane);
            const uint32_t a0 = lut32(e0), a1 = lut32(e1), a2 = lut32(e2), a3 = lut32(e3);
            if (kb < 2) mma_16816_z(c[kb & 1], a0, a1, a2, a3, qb[kb][0], qb[kb][1]);
            else mma_16816(c[kb & 1], a0, a1, a2, a3, qb[kb][0], qb[kb][1]);
            if constexpr (NH == 2) {
                const uint2 lo = lds64(q_lo + 256 * kb);
                if (kb == 0) mma_16816_z(c[NH], a0, a1, a2, a3, lo.x, lo.y);
                else mma_16816(c[NH], a0, a1, a2, a3, lo.x, lo.y);
            }
            if constexpr (NC) {
                n2 = add2(n2, pk2(__uint_as_float(lut32(e0 + SQ)), __uint_as_float(lut32(e1 + SQ))));
                other = add2(other, pk2(__uint_as_float(lut32(e2 + SQ)), __uint_as_float(lut32(e3 + SQ))));
            }
        }
        if constexpr (NC) n2 = add2(n2, other);
    }

    template <bool FULL>
    __device__ __forceinline__ void attend(uint32_t page, uint32_t ts, int lo, int hi, int lane, const float (&c)[NH + 1][4],
                                           float kna, float knb, uint32_t sca, uint32_t scb) {
        const int g = lane >> 2, tg = lane & 3;
        // ---- online softmax (base-2 exponents), the lane's tokens g and g + 8
        const bool okA = FULL || (g >= lo && g < hi), okB = FULL || (g + 8 >= lo && g + 8 < hi);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&sca));
        const float2 fb = __half22float2(*reinterpret_cast<const __half2*>(&scb));
        const float vsa = okA ? fa.x : 0.f, vsb = okB ? fb.x : 0.f;
        const float vza = okA ? fmaf(kCtr, fa.x, fa.y) : 0.f, vzb = okB ? fmaf(kCtr, fb.x, fb.y) : 0.f;
        float sa[HL], sb[HL];
        const float s_max = fmaxf(fabsf(vsa), fabsf(vsb));
        bool above = s_max > s_ref;
#pragma unroll
        for (int h = 0; h < HL; h++) {
            const float la = NH == 1 ? c[0][1] + c[1][1] : c[NH][h], lb = NH == 1 ? c[0][3] + c[1][3] : c[NH][2 + h];
            sa[h] = okA ? fmaf(la, kInvLo, c[0][h] + c[1][h]) * kna : -INFINITY;
            sb[h] = okB ? fmaf(lb, kInvLo, c[0][2 + h] + c[1][2 + h]) * knb : -INFINITY;
            above |= fmaxf(sa[h], sb[h]) > m_run[h];
        }
        if (__any_sync(0xffffffffu, above)) {
            // the largest value scale, rounded up to a power of two, brought to 2^14: fp16 holds weights down to 2^-28 of the
            // largest at full precision (a warp meets many pages under one reference maximum)
            float top = s_max;
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            float shift = 1.f;
            if (top > s_ref) {   // (warp-uniform)
                s_ref = __uint_as_float((__float_as_uint(top) + 0x007fffffu) & 0x7f800000u);
                const float was = up;
                up = 16384.f / s_ref;
                shift = up / was;
            }
            float corr[HL];
#pragma unroll
            for (int h = 0; h < HL; h++) {
                float m = fmaxf(sa[h], sb[h]);
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
                const float m_new = fmaxf(m_run[h], m);   // finite: a page has a token that counts
                corr[h] = fast_exp2(m_run[h] - m_new);
                l_run[h] *= corr[h];
                z_run[h] *= corr[h];
                m_run[h] = m_new;
            }
#pragma unroll
            for (int i = 0; i < OL / 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) oacc[i][j] *= corr[j % HL] * shift;
        }
        float wa[HL], wb[HL];
        const float sua = vsa * up, sub = vsb * up;   // (exact)
#pragma unroll
        for (int h = 0; h < HL; h++) {
            const float pa = fast_exp2(sa[h] - m_run[h]), pb = fast_exp2(sb[h] - m_run[h]);
            l_run[h] += pa + pb;
            z_run[h] = fmaf(pa, vza, fmaf(pb, vzb, z_run[h]));
            wa[h] = pa * sua;
            wb[h] = pb * sub;
        }

        // ---- O^T += V^T.P^T
        uint32_t v[4][VW];
        const uint32_t vrow = (page & ~3u) + 2 * tg * ts;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t row = vrow + ((j & 1) + 8 * (j >> 1)) * ts;
            if constexpr (VB == 4) {   // (as the keys; the values start OFF_VC = 2 mod 4 bytes into the slot)
                const uint32_t at = row + OFF_VC - 2 + 4 * mis;
#pragma unroll
                for (int u = 0; u < VW; u++) v[j][u] = lds32(at + 4 * g + 32 * u);
                v[j][0] = __byte_perm(v[j][0], lds32(at + PDV), !mis && g == 0 ? 0x3254u : 0x3210u);
            } else {
                load_bytes<VSB>(row + 2 * mis + OFF_VC + VSB * g, v[j]);
            }
        }
        auto pack = [](float lo, float hi) {
            const __half2 h = __floats2half2_rn(lo, hi);
            return *reinterpret_cast<const uint32_t*>(&h);
        };
        if constexpr (NH == 1) {
            // transposed, lane (g, tg) holds the weights of head g >> 1 for its tokens; a column is (head, parity):
            // the weight stands in the half that its parity selects
            const uint32_t t0 = movmatrix_trans(pack(wa[0], wa[0])), t1 = movmatrix_trans(pack(wb[0], wb[0]));
            const uint32_t sel_lo = (g & 1) ? 0x1044u : 0x4410u, sel_hi = (g & 1) ? 0x3244u : 0x4432u;
            const uint32_t pb[2][2] = {{__byte_perm(t0, 0u, sel_lo), __byte_perm(t0, 0u, sel_hi)},
                                       {__byte_perm(t1, 0u, sel_lo), __byte_perm(t1, 0u, sel_hi)}};
#pragma unroll
            for (int ks = 0; ks < 2; ks++) {
                if constexpr (VB == 4) {
#pragma unroll
                    for (int u = 0; u < VW; u++) {
                        uint32_t x[4], y[4];
                        centred(v[2 * ks][u], x);
                        centred(v[2 * ks + 1][u], y);
                        mma_16816(oacc[2 * u], x[0], x[1], y[0], y[1], pb[ks][0], pb[ks][1]);
                        mma_16816(oacc[2 * u + 1], x[2], x[3], y[2], y[3], pb[ks][0], pb[ks][1]);
                    }
                } else {
#pragma unroll
                    for (int mt = 0; mt < D / 32; mt++)
                        mma_16816(oacc[mt], lut32(entry_addr<IWV>(v[2 * ks], 2 * mt, lv_lane)),
                                  lut32(entry_addr<IWV>(v[2 * ks], 2 * mt + 1, lv_lane)),
                                  lut32(entry_addr<IWV>(v[2 * ks + 1], 2 * mt, lv_lane)),
                                  lut32(entry_addr<IWV>(v[2 * ks + 1], 2 * mt + 1, lv_lane)), pb[ks][0], pb[ks][1]);
                }
            }
        } else {
            const uint32_t b0 = movmatrix_trans(pack(wa[0], wa[HL - 1])), b1 = movmatrix_trans(pack(wb[0], wb[HL - 1]));
            if constexpr (VB == 4) {
#pragma unroll
                for (int u = 0; u < VW; u++)
#pragma unroll
                    for (int z = 0; z < 2; z++) {   // 16-bit halves of the words: the same codes of two tokens
                        uint32_t x[4], y[4];
                        centred(__byte_perm(v[0][u], v[1][u], z ? 0x7632u : 0x5410u), x);
                        centred(__byte_perm(v[2][u], v[3][u], z ? 0x7632u : 0x5410u), y);
                        mma_16816(oacc[4 * u + 2 * z], x[0], x[1], y[0], y[1], b0, b1);
                        mma_16816(oacc[4 * u + 2 * z + 1], x[2], x[3], y[2], y[3], b0, b1);
                    }
            } else {
#pragma unroll
                for (int pr = 0; pr < D / 16; pr++) {
                    uint32_t x[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) x[j] = lut32(entry_addr<IWV>(v[j], pr, lv_lane));
                    mma_16816(oacc[pr], __byte_perm(x[0], x[1], 0x5410u), __byte_perm(x[0], x[1], 0x7632u),
                              __byte_perm(x[2], x[3], 0x5410u), __byte_perm(x[2], x[3], 0x7632u), b0, b1);
                }
            }
        }
    }
    // The codes at bits 0, 4, 8, 12 of each 16-bit half of w, centred, as fp16 pairs: a nibble or-ed into the
    // mantissa of 1024 is 1024 + code (or 1024 + 16 code one nibble up), one packed subtraction or
    // multiply-add centres it exactly.
    __device__ __forceinline__ void centred(uint32_t w, uint32_t (&t)[4]) const {
        const uint32_t w8 = w >> 8;
        const uint32_t x[4] = {(w & 0x000F000Fu) | magic, (w & 0x00F000F0u) | magic,
                               (w8 & 0x000F000Fu) | magic, (w8 & 0x00F000F0u) | magic};
        const __half2 sub = *reinterpret_cast<const __half2*>(&c_sub), mul = *reinterpret_cast<const __half2*>(&c_mul),
                      add = *reinterpret_cast<const __half2*>(&c_add);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const __half2 h = *reinterpret_cast<const __half2*>(&x[i]);
            const __half2 r = (i & 1) ? __hfma2(h, mul, add) : __hsub2(h, sub);
            t[i] = *reinterpret_cast<const uint32_t*>(&r);
        }
    }

    // the lane's state: OL floats at xo[f * 32 + lane], (m, l, z) of its heads at xml[0..2][8]
    __device__ __forceinline__ void publish(float* xo, float* xml, int lane, bool poison) {
#pragma unroll
        for (int h = 0; h < HL; h++)
#pragma unroll
            for (int m = 4; m < 32; m <<= 1) {
                l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], m);
                z_run[h] += __shfl_xor_sync(0xffffffffu, z_run[h], m);
            }
#pragma unroll
        for (int f = 0; f < OL; f++) xo[f * 32 + lane] = oacc[f >> 2][f & 3] * (1.f / up);
        if (lane < 4) {
#pragma unroll
            for (int h = 0; h < HL; h++) {
                xml[HL * lane + h] = poison ? __int_as_float(0x7fc00000) : m_run[h];
                xml[8 + HL * lane + h] = l_run[h];
                xml[16 + HL * lane + h] = z_run[h];
            }
        }
    }
    // head and coordinate of output float f of lane ln
    static __device__ __forceinline__ int head_of(int f, int ln) { return NH == 1 ? ln & 3 : 2 * (ln & 3) + (f & 1); }
    __device__ __forceinline__ int coord_of(int f, int ln) const {
        const int g = ln >> 2, tile = f >> 2, i = f & 3;
        if constexpr (VB == 4) {
            const int u = NH == 1 ? tile >> 1 : tile >> 2;
            const int nib = NH == 1 ? 2 * (tile & 1) + (i >> 1) + 4 * (i & 1) : 2 * (tile & 3) + (i >> 1);
            return (8 * (g + 8 * u) + nib - (mis ? 0 : 4)) & (D - 1);
        } else {
            return (D / 8) * g + (NH == 1 ? 4 * tile + i : 2 * tile + (i >> 1));
        }
    }
};

template <class E>
__global__ void __launch_bounds__(kTqFlowThreads, 1)
tq_flow_kernel(const __grid_constant__ TqFlowParams f) {
    const TqDecodeParams& p = f.d;
    constexpr int D = E::D;
    constexpr int XSLOT = tq_flow_xslot(D, E::NH);   // (an exchange slot holds a warp's queries first)
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    auto gptr = [&](uint32_t saddr) { return smem_raw + (saddr - sbase); };

    // ---- shared memory: the table window (64 KB aligned), small objects first-fit before / behind it, ring
    const uint32_t window = E::WINDOW ? (sbase + 65535u) & ~65535u : sbase;
    uint32_t free0 = sbase, free1 = E::WINDOW ? window + 65536u : sbase;
    const uint32_t end0 = window, end1 = sbase + kTqFlowSmem - 16;   // (a load may reach 2 bytes past a slot)
    auto take = [&](uint32_t bytes, uint32_t align) {
        uint32_t a = (free0 + align - 1) & ~(align - 1);
        if (a + bytes <= end0) { free0 = a + bytes; return a; }
        a = (free1 + align - 1) & ~(align - 1);
        free1 = a + bytes;
        return a;
    };
    const uint32_t tk = E::TKS > 0 ? take(2 * E::TKS, E::TKS) : 0, tv = E::TVS > 0 ? take(E::TVS, E::TVS) : 0;
    const uint32_t full = take(kTqFlowBarriers * 8, 128), empty = full + kTqFlowSlots * 8,
                   pfull = empty + kTqFlowSlots * 8, pempty = pfull + kTqFlowPieces * 8, folded = pempty + kTqFlowPieces * 8;
    TqPiece* pieces = reinterpret_cast<TqPiece*>(gptr(take(kTqFlowPieces * sizeof(TqPiece), 128)));
    // where a ring slot lies, and what the producer knows of the page in it: its turn * 2 + (block id out of range), -1: never
    // used
    const uint32_t slot_table = take(kTqFlowSlots * 8, 128);
    volatile int2* slot_info = reinterpret_cast<volatile int2*>(gptr(slot_table));
    float* xml = reinterpret_cast<float*>(gptr(take(kTqFlowWarps * 24 * 4, 128)));
    int* prefix = reinterpret_cast<int*>(gptr(take((kFlowMaxSeqs + 4) * 4, 128)));
    const uint32_t xarea = take(kTqFlowWarps * XSLOT, 128);
    const uint32_t ts = static_cast<uint32_t>(p.stride_pos), bytes = f.page_bytes;
    const uint32_t pitch = (kPageTokens * ts + 127) & ~127u;
    free0 = (free0 + 127u) & ~127u;
    free1 = (free1 + 127u) & ~127u;
    const int n0 = end0 > free0 ? (end0 - free0) / pitch : 0;
    const int subs = kTqFlowWarps / p.Hkv;      // warps of a head
    const int n_slots = min(kTqFlowSlots, n0 + static_cast<int>((end1 - free1) / pitch)) / subs * subs;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    E::init_tables(p, reinterpret_cast<uint32_t*>(gptr(window)), reinterpret_cast<uint32_t*>(gptr(tk ? tk : sbase)),
                   reinterpret_cast<uint32_t*>(gptr(tv ? tv : sbase)), tid, kTqFlowThreads);
    if (tid < n_slots) {
        mbar_init(full + tid * 8, 1);
        mbar_init(empty + tid * 8, p.Hkv);
        slot_info[tid].x = tid < n0 ? free0 + tid * pitch : free1 + (tid - n0) * pitch;
        slot_info[tid].y = -1;
    }
    if (tid < p.Hkv) mbar_init(folded + tid * 8, subs);
    if (tid < kTqFlowPieces) {
        mbar_init(pfull + tid * 8, 1);
        mbar_init(pempty + tid * 8, kTqFlowWarps);
    }
    mbar_fence_init();
    after_previous_kernel();

    // ---- prefix sums of the sequences' places over all splits (also for the merge kernel)
    const int cost = f.piece_cost;
    auto kv_start_of = [&](int b) { return p.kv_start ? p.kv_start[b] : 0; };
    if (warp == 0) {
        int carry = 0;
        for (int b0 = 0; b0 < p.B_seq; b0 += 32) {
            const int b = b0 + lane;
            int x = 0;
            if (b < p.B_seq) {
                const int len = p.seq_lens[b], start = kv_start_of(b);
                for (int s = 0; s < p.splits; s++) {
                    const int n = tq_range_pages(tq_split_range(len, start, p.splits, s));
                    x += n > 0 ? n + cost : 0;
                }
            }
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            if (b < p.B_seq) prefix[b + 1] = carry + x;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) prefix[0] = 0;
    }
    __syncthreads();
    const uint32_t per_layer = prefix[p.B_seq];   // (the host bounds it by 2^30)
    const uint32_t share = max((per_layer + gridDim.x - 1) / gridDim.x, f.min_share);
    const uint32_t n_shares = (per_layer + share - 1) / share, all_shares = n_shares * (p.B / p.B_seq);
    if (blockIdx.x == 0) {
        if (tid == 0) {
            f.share[0] = share;
            f.share[1] = n_shares;
        }
        for (int i = tid; i <= p.B_seq; i += kTqFlowThreads) f.prefix[i] = prefix[i];
    }
    // splits without tokens: no CTA meets them; neutral partials (zeros, lse = -inf)
    for (int i = blockIdx.x; i < p.B * p.splits; i += gridDim.x) {
        const int row = i / p.splits, sid = i - row * p.splits;
        const int b = row - static_cast<int>(fast_div(static_cast<uint32_t>(row), p.div_bseq)) * p.B_seq;
        const TqRange r = tq_split_range(p.seq_lens[b], kv_start_of(b), p.splits, sid);
        if (r.t1 > r.t0) continue;
        for (int j = tid; j < p.Hq * (D + 1); j += kTqFlowThreads) {
            const int h = j / (D + 1), d = j - h * (D + 1);
            p.mid_o[((static_cast<int64_t>(row) * p.Hq + h) * p.splits + sid) * (D + 1) + d] = d == D ? -INFINITY : 0.f;
        }
    }

    if (warp >= kTqFlowWarps) {
        // ================================================================ producer
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kTqFetchRegs));
        if (warp > kTqFlowWarps) return;
        const uint64_t policy = l2_evict_first_policy();   // (pages are read once per step)
        const int per_sub = n_slots / subs;
        bool ok = true;
        int pi = 0;              // pieces announced
        int sub_pages = 0;       // lane s: pages requested for the s-th warps of the heads
        // the CTA's shares [at, last), position in the layer's line
        const uint32_t each = (all_shares + gridDim.x - 1) / gridDim.x;
        uint32_t at = min(each * blockIdx.x, all_shares), pos = 0;
        const uint32_t last = min(at + each, all_shares);
        if (at < last) pos = at % n_shares * share;
        for (;;) {
            const int ps = pi % kTqFlowPieces;
            if (pi >= kTqFlowPieces) ok = mbar_wait_idle(pempty + ps * 8, ((pi / kTqFlowPieces) - 1) & 1) && ok;
            TqPiece pc{};
            int b = 0, layer = 0, page0 = 0;
            while (ok && at < last) {   // (until a part with pages)
                layer = at / n_shares;
                const uint32_t first = (at - layer * n_shares) * share, end = min(first + share, per_layer);
                int r = pos;
                int lo = 0, hi = p.B_seq;    // prefix[lo] <= r < prefix[hi]
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (prefix[mid] <= r) lo = mid; else hi = mid;
                }
                b = lo;
                r -= prefix[b];
                const int len = p.seq_lens[b], start = kv_start_of(b);
                TqRange rg{};
                int n = 0;
                for (pc.sid = 0; pc.sid < p.splits; pc.sid++) {
                    rg = tq_split_range(len, start, p.splits, pc.sid);
                    n = tq_range_pages(rg);
                    const int places = n > 0 ? n + cost : 0;
                    if (r < places) break;
                    r -= places;
                }
                const int stop = min(n + cost, r + static_cast<int>(end - pos));   // places [r, stop) of the unit
                const int from = max(r - cost, 0);
                pc.n = max(stop - cost, 0) - from;
                pc.row = layer * p.B_seq + b;
                pc.block = pc.n == n ? -1 : 2 * static_cast<int>(at) + (pos == first && r >= cost ? 0 : 1);
                page0 = rg.t0 / kPageTokens + from;
                pc.lo = rg.t0 - page0 * kPageTokens;
                pc.hi = rg.t1 - page0 * kPageTokens;
                pos += stop - r;
                if (pos == end) {
                    at++;
                    pos = at % n_shares * share;
                }
                if (pc.n > 0) break;
            }
            if (lane == 0) {
                pieces[ps] = pc;
                mbar_arrive(pfull + ps * 8);
            }
            __syncwarp();
            pi++;
            if (pc.n == 0) break;
            // the piece's pages, one for each of the heads' warps at a time (lane s: the s-th warps'); block ids by
            // batches of 32, one batch ahead
            const int32_t* btab = p.block_table + static_cast<int64_t>(b) * p.max_blocks;
            const uint8_t* const kv_layer = p.kv_cache + layer * p.cache_layer_stride;
            auto load_id = [&](int i) {
                if (i >= pc.n) return 0;
                return btab[fast_div(static_cast<uint32_t>(page0 + i) * kPageTokens, p.div_block)];
            };
            int ids = 0, ids_next = load_id(lane);
            for (int i0 = 0; i0 < pc.n && ok; i0 += subs) {
                if ((i0 & 31) == 0) {
                    ids = ids_next;
                    ids_next = load_id(i0 + 32 + lane);
                }
                int64_t id = __shfl_sync(0xffffffffu, ids, (i0 + lane) & 31);
                const int i = i0 + lane;
                const int k = sub_pages + i0 / subs, turn = k / per_sub, s = (k - turn * per_sub) * subs + lane;
                const uint32_t tok = static_cast<uint32_t>(page0 + i) * kPageTokens;
                const uint32_t off = tok - fast_div(tok, p.div_block) * p.block_size;
                const bool bad = p.num_blocks > 0 && static_cast<uint64_t>(id) >= static_cast<uint64_t>(p.num_blocks);
                if (bad) id = 0;
                const uint8_t* const src = kv_layer + id * p.stride_block + static_cast<int64_t>(off) * ts;
                // one after the other (polls of all of them at once were a quarter of the kernel's instructions)
                for (int u = 0; u < subs && ok; u++) {
                    const int s_u = __shfl_sync(0xffffffffu, s, u), turn_u = __shfl_sync(0xffffffffu, turn, u);
                    if (i0 + u >= pc.n) break;
                    // (a slot whose last copy has not arrived is not armed again)
                    if (turn_u > 0)
                        ok = mbar_wait_idle(empty + s_u * 8, (turn_u - 1) & 1) && mbar_wait(full + s_u * 8, (turn_u - 1) & 1);
                    ok = __all_sync(0xffffffffu, ok);
                    if (ok && lane == u) {
                        slot_info[s].y = 2 * turn + (bad ? 1 : 0);
                        mbar_expect_tx(full + s * 8, bytes);
#ifdef FTQ_TEST_WAIT_EXPIRY
                        if (blockIdx.x == 0 && sub_pages == 0 && i == 0) continue;   // (see kMbarSpinLimit)
#endif
                        bulk_g2s_hint(slot_info[s].x, src, bytes, full + s * 8, policy);
                    }
                }
                __syncwarp();
            }
            sub_pages += (pc.n + subs - 1 - lane) / subs;   // (lanes from `subs` on are not read)
        }
        // nobody leaves with copies in flight
        __syncwarp();
        for (int s = lane; s < n_slots; s += 32)
            if (slot_info[s].y >= 0) ok = mbar_wait(full + s * 8, (slot_info[s].y >> 1) & 1) && ok;
        if (!ok) *f.share = 0u;
        return;
    }

    // ==================================================================== consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kTqFlowRegs));
    const int head = warp % p.Hkv, sub = warp / p.Hkv;
    const int group = p.Hq / p.Hkv;
    const uint32_t my_off = static_cast<uint32_t>(p.stride_head) * head;
    auto xchg = [&](int w) { return reinterpret_cast<float*>(gptr(xarea + w * XSLOT)); };
    bool stalled = false;
    uint32_t fold_par = 0;
    // barrier of the head's warps (an mbarrier: a warp that never comes does not hang the others)
    auto head_sync = [&]() {
        __syncwarp();
        if (subs == 1) return;
        if (lane == 0) mbar_arrive(folded + head * 8);
        if (!stalled && !mbar_wait(folded + head * 8, fold_par)) stalled = true;
        fold_par ^= 1u;
    };
    E e;
    e.init(window, tk, tv, lane, (my_off >> 1) & 1);
    int s = sub;             // ring slot of the warp's next page, and the parity of its turn
    uint32_t par = 0;
    for (int pi = 0;; pi++) {
        const int ps = pi % kTqFlowPieces;
        if (!mbar_wait(pfull + ps * 8, (pi / kTqFlowPieces) & 1)) {
            stalled = true;
            break;
        }
        const volatile TqPiece& pc = pieces[ps];
        const int n = pc.n;
        int lo = pc.lo - sub * kPageTokens, hi = pc.hi - sub * kPageTokens;
        if (n == 0) break;
        int64_t head0 = static_cast<int64_t>(pc.row) * p.Hq + head * group;
        float* qs = xchg(warp);
        e.rotate(p, qs, head0, group, lane);
        __syncwarp();
        e.begin(qs, lane);
        __syncwarp();
        bool poison = false;
        int seen = 0;
        (void)seen;
        for (int i = sub; i < n; i += subs) {
            if (!stalled && !mbar_wait(full + s * 8, par)) stalled = true;
            const uint2 slot = lds64(slot_table + s * 8);
            poison |= (slot.y & 1u) != 0u;
            const uint32_t page = slot.x + my_off;
            e.page(page, ts, lo, hi, p.norm_correction != 0, lane);
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + s * 8);
            if constexpr (E::FLUSH > 0)
                if (++seen % E::FLUSH == 0) e.flush(xchg(warp), lane);
            s += subs;
            if (s >= n_slots) { s = sub; par ^= 1u; }
            lo -= subs * kPageTokens;
            hi -= subs * kPageTokens;
        }

        // ---- the warps of the head put their states together
        head0 = static_cast<int64_t>(pc.row) * p.Hq + head * group;
        const int sid = pc.sid, block = pc.block;
        __syncwarp();
        if (lane == 0) mbar_arrive(pempty + ps * 8);
        e.publish(xchg(warp), xml + warp * 24, lane, poison || stalled);
        head_sync();
        for (int j = sub * 32 + lane; j < E::OL * 32; j += subs * 32) {
            const int ln = j & 31, fo = j >> 5, h = E::head_of(fo, ln);
            if (h >= group) continue;
            float M = -INFINITY;
            bool nan = stalled;
            for (int w = head; w < kTqFlowWarps; w += p.Hkv) {
                const float mw = xml[w * 24 + h];
                nan |= mw != mw;
                M = fmaxf(M, mw);
            }
            float o = 0.f, l = 0.f, z = 0.f;
            for (int w = head; w < kTqFlowWarps; w += p.Hkv) {
                const float sc = fast_exp2(xml[w * 24 + h] - M);   // (a warp without pages: 0)
                o = fmaf(xchg(w)[j], sc, o);
                l = fmaf(xml[w * 24 + 8 + h], sc, l);
                z = fmaf(xml[w * 24 + 16 + h], sc, z);
            }
            const int coord = e.coord_of(fo, ln);
            if (block < 0) {
                float* dst = p.mid_o + ((head0 + h) * p.splits + sid) * (D + 1);
                dst[coord] = (o + z) / l;
                if (coord == 0) dst[D] = nan ? __int_as_float(0x7fc00000) : M * kLn2 + logf(l);
            } else {   // (sums, reference maximum and weight sum: nothing is rounded into a logarithm before the merge)
                float* dst = f.rows + (static_cast<int64_t>(block) * p.Hq + head * group + h) * (D + 2);
                dst[coord] = o + z;
                if (coord == 0) {
                    dst[D] = M;
                    dst[D + 1] = nan ? __int_as_float(0x7fc00000) : l;
                }
            }
        }
        head_sync();
    }
    if (stalled && lane == 0) *f.share = 0u;
}

// What is left of a row once its partials are summed up (weights relative to M, their sum l): normalise, rotate back,
// merge the prefix in, store.  Every octet of the row holds the sums and stores its part.  (As the end of
// tq_merge_kernel, which has it in its body and its registers' number from that.)
template <int D, typename OT, int OCTETS>
__device__ __forceinline__ void tq_finish_row(const TqMergeParams& p, OT* __restrict__ out, float* __restrict__ lse_out,
                                              int64_t row, float (&a)[D / kOctet], float l, float M, int lane, bool store) {
    constexpr int E = D / kOctet;
    const int t = lane & 7, o = (lane >> 3) & (OCTETS - 1);
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int r = 0; r < E; r++) a[r] *= inv;
    if (p.rotate) {
        octet_fwht<E>(a, lane);
#pragma unroll
        for (int k = 0; k < E; k++) a[k] *= p.rsqrt_d;
    }
    float lse = l > 0.f ? M + logf(l) : -INFINITY;
    float w_own = 1.f, w_pre = 0.f;
    const bool prefix = p.prefix_out != nullptr;
    if (prefix) {
        const float lp = p.prefix_lse[row];
        const float lmax = fmaxf(lp, lse);
        if (lmax == -INFINITY) {  // nothing attended on either side
            w_own = 0.f;
        } else {
            const float ep = __expf(lp - lmax), eq = __expf(lse - lmax);
            const float total = fmaxf(ep + eq, 1e-20f);
            w_pre = ep / total;
            w_own = eq / total;
            lse = lmax + logf(ep + eq);
        }
    }
    OT* orow = out + row * D;
#pragma unroll
    for (int r = 0; r < E; r++) {
        if (!store || (r & (OCTETS - 1)) != o) continue;
        const int coord = p.rotate ? t + 8 * r : load_coord(t, r);
        float v = a[r];
        if (prefix) {
            const int64_t at = row * D + coord;
            const float pv = p.prefix_dtype == kF32 ? static_cast<const float*>(p.prefix_out)[at]
                             : p.prefix_dtype == kF16
                                 ? __half2float(static_cast<const __half*>(p.prefix_out)[at])
                                 : __bfloat162float(static_cast<const __nv_bfloat16*>(p.prefix_out)[at]);
            v = pv * w_pre + v * w_own;
        }
        if constexpr (sizeof(OT) == 4) orow[coord] = v;
        else if constexpr (std::is_same<OT, __half>::value) orow[coord] = __float2half_rn(v);
        else orow[coord] = __float2bfloat16_rn(v);
    }
    if (lse_out && t == 0 && o == 0 && store) lse_out[row] = lse;
}

// Stage 2 (tq_merge_kernel, ftq_tq_v1.cuh) where a split that a share's end cut lies in the workspace in pieces: they
// are put together, written to mid_o and merged.  Two warps per row, an octet per split, the eight octets side by side; the
// pieces of a split kPieceBatch at a time (four took more registers: 4096 whole rows 23 us, 18 with two).  The latency of the
// loads bounds it.  (While the octets of a warp took turns -- each looked through all splits for its own -- 64 rows of 64 splits
// took 134 us, now 13; 512 rows of which 8 splits had 14 pieces each 74 us, now 12.)
// Stage 1 does not let it start early: this kernel's CTAs would fill the first SMs that stage 1 leaves, many to an SM, and
// wait there, and the few SMs then do all of its work (with one long context among short ones 55 us for the whole
// call, 32 so).
template <int D, typename OT>
__global__ void __launch_bounds__(128)
tq_join_kernel(const __grid_constant__ TqJoinParams p) {
    constexpr int E = D / kOctet, kPieceBatch = 2;
    __shared__ float part[2][kOctet][E + 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 7;
    const int which = warp >> 1, oct = 4 * (warp & 1) + (lane >> 3);
    const int64_t at = static_cast<int64_t>(blockIdx.x) * 2 + which;
    const int64_t row = at < p.m.n_rows ? at : p.m.n_rows - 1;
    const uint32_t r = fast_div(static_cast<uint32_t>(row), p.div_hq);   // (layer, sequence)
    const int h = static_cast<int>(static_cast<uint32_t>(row) - r * p.Hq);
    const uint32_t layer = fast_div(r, p.div_bseq);
    const int b = static_cast<int>(r - layer * p.B_seq);
    let_next_kernel_start();
    after_previous_kernel();   // stage 1 is complete
    const uint32_t share = __ldcg(p.share);
    const int64_t shares0 = static_cast<int64_t>(layer) * __ldcg(p.share + 1);
    const int len = p.seq_lens[b], start = p.kv_start ? p.kv_start[b] : 0;
    uint32_t pos = static_cast<uint32_t>(__ldcg(p.page_prefix + b));
    float M = -INFINITY, l = 0.f, a[E];
#pragma unroll
    for (int i = 0; i < E; i++) a[i] = 0.f;
    for (int s0 = 0; s0 < p.m.splits; s0 += kOctet) {
        // lane t: pages of split s0 + t; its place in the line
        const uint32_t pages = s0 + t < p.m.splits ? tq_range_pages(tq_split_range(len, start, p.m.splits, s0 + t)) : 0;
        uint32_t upto = pages > 0 ? pages + p.piece_cost : 0;
#pragma unroll
        for (int m = 1; m < kOctet; m <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, upto, m, kOctet);
            if (t >= m) upto += y;
        }
        const uint32_t n = __shfl_sync(0xffffffffu, pages, oct, kOctet);
        const uint32_t first = pos + __shfl_sync(0xffffffffu, upto, oct, kOctet) - n;
        pos += __shfl_sync(0xffffffffu, upto, kOctet - 1, kOctet);
        if (n == 0 || share == 0) continue;
        const uint32_t c0 = first / share, c1 = (first + n - 1) / share;
        const bool cut = c0 != c1;
        float* const mid = p.mid_out + (row * p.m.splits + s0 + oct) * (D + 1);
        // (row block 0 is the piece the share starts with, 1 its last one)
        auto source = [&](uint32_t c) {
            return cut ? p.rows + ((2 * (shares0 + c) + (c * share >= first ? 0 : 1)) * p.Hq + h) * (D + 2) : mid;
        };
        const float* src = source(c0);
        float x[E], ms = __ldcg(src + D), ls = cut ? __ldcg(src + D + 1) : 1.f;   // (a NaN stays one)
#pragma unroll
        for (int i = 0; i < E; i++) x[i] = __ldcg(src + load_coord(t, i));
        for (uint32_t c = c0 + 1; c <= c1; c += kPieceBatch) {
            float y[kPieceBatch][E], my[kPieceBatch], ly[kPieceBatch];
#pragma unroll
            for (int k = 0; k < kPieceBatch; k++) {
                my[k] = -INFINITY;
                ly[k] = 0.f;
#pragma unroll
                for (int i = 0; i < E; i++) y[k][i] = 0.f;
                if (c + k <= c1) {
                    src = source(c + k);
                    my[k] = __ldcg(src + D);
                    ly[k] = __ldcg(src + D + 1);
#pragma unroll
                    for (int i = 0; i < E; i++) y[k][i] = __ldcg(src + load_coord(t, i));
                }
            }
            float top = ms;
#pragma unroll
            for (int k = 0; k < kPieceBatch; k++) top = fmaxf(top, my[k]);
            const float f0 = fast_exp2(ms - top);
            ls *= f0;
#pragma unroll
            for (int i = 0; i < E; i++) x[i] *= f0;
#pragma unroll
            for (int k = 0; k < kPieceBatch; k++) {
                const float f = fast_exp2(my[k] - top);
                ls = fmaf(ly[k], f, ls);
#pragma unroll
                for (int i = 0; i < E; i++) x[i] = fmaf(y[k][i], f, x[i]);
            }
            ms = top;
        }
        if (cut) {
            const float inv = 1.f / ls;
            ms = ms * kLn2 + logf(ls);
#pragma unroll
            for (int i = 0; i < E; i++) {
                x[i] *= inv;
                mid[load_coord(t, i)] = x[i];
            }
            if (t == 0) mid[D] = ms;
        }
        const float m_new = fmaxf(M, ms);
        const float f0 = __expf(M - m_new), f = __expf(ms - m_new);
        l = fmaf(l, f0, f);
#pragma unroll
        for (int i = 0; i < E; i++) a[i] = fmaf(a[i], f0, x[i] * f);
        M = m_new;
    }
    if (share == 0) {
        l = __int_as_float(0x7fc00000);
#pragma unroll
        for (int i = 0; i < E; i++) a[i] = l;
    }
    // the octets of a warp, then the two warps
    auto join = [&](float m_o, float l_o, auto other) {
        const float m_new = fmaxf(M, m_o);
        const float f0 = M == -INFINITY && l == 0.f ? 0.f : __expf(M - m_new);
        const float f1 = m_o == -INFINITY && l_o == 0.f ? 0.f : __expf(m_o - m_new);
        l = l * f0 + l_o * f1;
#pragma unroll
        for (int i = 0; i < E; i++) a[i] = a[i] * f0 + other(i) * f1;
        M = m_new;
    };
#pragma unroll
    for (int m = 8; m < 32; m <<= 1) {
        const float m_o = __shfl_xor_sync(0xffffffffu, M, m), l_o = __shfl_xor_sync(0xffffffffu, l, m);
        join(m_o, l_o, [&](int i) { return __shfl_xor_sync(0xffffffffu, a[i], m); });
    }
    if ((warp & 1) && lane < kOctet) {
#pragma unroll
        for (int i = 0; i < E; i++) part[which][t][i] = a[i];
        part[which][t][E] = M;
        part[which][t][E + 1] = l;
    }
    __syncthreads();
    if (warp & 1) return;
    join(part[which][t][E], part[which][t][E + 1], [&](int i) { return part[which][t][i]; });
    tq_finish_row<D, OT, 4>(p.m, static_cast<OT*>(p.m.out), p.m.lse, row, a, l, M, lane, at < p.m.n_rows);
}

}  // namespace ftq
