// vLLM-v1 slot format with FP8 keys, decode stage 1 on the tensor cores at fp32 precision.
//
// Same result as tq_split_kernel (ftq_tq_v1.cuh), i.e. the reference's
// `_tq_decode_stage1_offset` (src/fused_turboquant/vllm_plugin/triton_decode_offset.py:42-444), partials
// in the same [B, Hq, splits, D + 1] layout.  That kernel spends 1500 instructions on a 16-token page
// (fp32 FMAs per query head, shuffles per score) and was issue bound at 137 us for 16 x 4096 tokens of
// 8 heads; here both products are m16n8k16 MMAs (73 us):
//   * e4m3 keys and 2- to 4-bit value codes are exact in fp16.  The code nearest to the value 0 is taken off
//     a token's codes and what it is off by goes through fp32 sums: the sums of code * scale and of the zero
//     points would be large numbers of opposite sign otherwise;
//   * a rotated query is the sum of two fp16 numbers, hi + lo / 2^11, after scaling by a power of two that
//     puts the head's largest coordinate in [2^10, 2^11): 23 bits of that coordinate's magnitude;
//   * a softmax weight (times the value scale) is split the same way, times the power of two that puts the
//     largest value scale seen so far at 2^14.
// An MMA truncates its sums where FMAs round, so chains are short (two k-blocks of a score, one page of the
// output) and added up in fp32.  Error against 64-bit arithmetic over 72 configurations (64 / 128, 300 to
// 30000 tokens, values times 1 to 1e-4, shifted by 10, channels ten times larger), mean per vector: 0.57 to
// 1.02 of the fp32 kernel's, 0.87 in the middle.  With chains over all of a warp's pages, unscaled
// weights and codes centred at 7.5 it was 0.55 to 4.1 of it, 1.16 in the middle, in 70 us.
// With at most four heads the eight columns of an MMA are (head, hi / lo), so the split costs no MMA; with
// five to eight heads hi and lo are one MMA each.
//
// Fragment maps for a page of 16 tokens (lane = 4 g + tg):
//   S: A rows g, g + 8 = tokens, k-block kb = coordinates (D/4) tg + 4 kb + {0..3} (word kb of the lane's
//      key slice), C columns 2tg, 2tg + 1 = (head tg, hi / lo) or heads 2tg, 2tg + 1
//   O^T: A rows g, g + 8 of m-tile mt = coordinates (D/8) g + 2 mt, + 1, k = tokens; B = the weights,
//      packed per token and transposed by movmatrix
//
// Work: persistent CTAs over (split, KV head, sequence) items, the pages of an item dealt to the warps.
// A warp's copies (cp.async, 4 bytes: slots are only 4-byte aligned; eight lanes per slot) run STAGES - 1
// pages ahead of its arithmetic and across items.
#pragma once

#include <cuda_fp8.h>

#include "ftq_attn_mma.cuh"
#include "ftq_tq_v1.cuh"

namespace ftq {

// ---- arithmetic of one warp on the pages of one head.  Used by the kernel below, whose pages lie in rows of whole 16-byte
// units (WIDE), and by the one that streams whole pages of all heads (ftq_tq_v1_flow.cuh), where a slot is only
// 4-byte aligned and the k-block kb of the scores is word tg + 4 kb of a row instead of word kb of the lane's
// quarter (neighbouring lanes on neighbouring banks).
template <int D_, int VB, int NH_, bool WIDE>
struct TqFp8 {
    static constexpr int D = D_, NH = NH_, HL = NH_, NKB = D / 16, NMT = D / 16, E = D / kOctet;
    static constexpr int PDV = D * VB / 8, VSB = PDV / 8, VW = (VSB + 3) / 4;
    static constexpr int CHAINS = 4;                             // independent sums of a score
    static constexpr int OL = NMT * 2 * HL;                      // output floats of a lane
    static constexpr float kLo = 2048.f, kInvLo = 1.f / 2048.f;
    // A head's rotated query and its factor: WIDE in quarters four floats apart (the lanes of a load read different quarters; in
    // one row, four of them on one bank, 19 x 429 tokens of 4 heads took 19.2 us instead of 17.7)
    static constexpr int QROW = WIDE ? D + 16 : D + 4, QMUL = QROW - 4;
    static __device__ __forceinline__ constexpr int q_at(int head, int coord) {
        return head * QROW + (WIDE ? coord / (D / 4) * (D / 4 + 4) + coord % (D / 4) : coord);
    }
    // (tq_flow_kernel: no tables)
    static constexpr bool WINDOW = false;
    static constexpr int TKS = 0, TVS = 0;
    static __device__ __forceinline__ void init_tables(const TqDecodeParams&, uint32_t*, uint32_t*, uint32_t*, int, int) {}
    __device__ __forceinline__ void init(uint32_t, uint32_t, uint32_t, int, int) {}

    uint32_t qb[NH][NKB][2];
    float mul[HL], m_run[HL], l_run[HL], z_run[HL], oacc[NMT][2 * HL];   // [m-tile][row g or g + 8, head]
    float s_ref, up;   // largest value scale so far as a power of two; weights are split times up
    // Sums over many pages in fp32 lose digits: a warp that goes through more than FLUSH of them adds up its sums of
    // FLUSH pages in shared memory.  l_sum, z_sum, m_sum, up_sum: the other sums, and what the ones there are relative to.
    static constexpr int FLUSH = WIDE ? 0 : 4;
    float l_sum[HL], z_sum[HL], m_sum[HL], up_sum;

    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    static __device__ __forceinline__ float residual(float x) { return (x - __half2float(__float2half_rn(x))) * kLo; }

    // rotate (no signs) and normalise the queries of heads 4 x .. 4 x + 3, an octet per head
    static __device__ __forceinline__ void rotate_four(const TqDecodeParams& p, float* qs, int64_t head0, int group, int lane, int x) {
        const int t8 = lane & 7, hh = 4 * x + (lane >> 3);
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
        float mx = 0.f;
#pragma unroll
        for (int k = 0; k < E; k++) mx = fmaxf(mx, fabsf(a[k]));
#pragma unroll
        for (int m = 1; m < 8; m <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
        // power of two that brings mx into [2^10, 2^11) (1 for zero, infinite or NaN rows)
        int e = static_cast<int>((__float_as_uint(mx) >> 23) & 255u);
        e = e == 255 || mx == 0.f ? 0 : min(120, 127 + 10 - e);
        const float scale_up = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
        const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
#pragma unroll
        for (int k = 0; k < E; k++) qs[q_at(hh, t8 + 8 * k)] = hv ? a[k] * scale_up : 0.f;
        // (the transform's factor goes here, not into the coordinates: one rounding for all factors)
        constexpr double kRotate = D == 64 ? 0.125 : 0.08838834764831845;   // 1 / sqrt(D)
        if (t8 == 0) qs[hh * QROW + QMUL] = static_cast<float>(p.scale * (1.4426950408889634 * kRotate)) * down;
    }
    __device__ __forceinline__ void rotate(const TqDecodeParams& p, float* qs, int64_t head0, int group, int lane) {
#pragma unroll
        for (int x = 0; x < NH; x++) rotate_four(p, qs, head0, group, lane, x);
    }
    // B fragments: column g = (head g >> 1, hi for an even g, lo for an odd one), or head g (hi, lo)
    __device__ __forceinline__ void begin(const float* qs, int lane) {
        const int g = lane >> 2, tg = lane & 3;
#pragma unroll
        for (int kb = 0; kb < NKB; kb++) {
            const int coord = WIDE ? (D / 4) * tg + 4 * kb : 4 * (tg + 4 * kb);
            const float4 q4 = *reinterpret_cast<const float4*>(qs + q_at(NH == 1 ? g >> 1 : g, coord));
            const uint32_t h0 = pack(q4.x, q4.y), h1 = pack(q4.z, q4.w);
            const uint32_t l0 = pack(residual(q4.x), residual(q4.y)), l1 = pack(residual(q4.z), residual(q4.w));
            if constexpr (NH == 1) {
                qb[0][kb][0] = (g & 1) ? l0 : h0;
                qb[0][kb][1] = (g & 1) ? l1 : h1;
            } else {
                qb[0][kb][0] = h0; qb[0][kb][1] = h1;
                qb[NH - 1][kb][0] = l0; qb[NH - 1][kb][1] = l1;
            }
        }
#pragma unroll
        for (int h = 0; h < HL; h++) {
            mul[h] = qs[(HL * tg + h) * QROW + QMUL];
            m_run[h] = -INFINITY;
            l_run[h] = z_run[h] = l_sum[h] = z_sum[h] = 0.f;
            m_sum[h] = -INFINITY;
        }
#pragma unroll
        for (int mt = 0; mt < NMT; mt++)
#pragma unroll
            for (int i = 0; i < 2 * HL; i++) oacc[mt][i] = 0.f;
        s_ref = 0.f;
        up = 1.f;
        up_sum = 0.f;   // (nothing there yet)
    }
    // adds the sums since the last time to those at xo[f * 32 + lane] (the lane's own)
    __device__ __forceinline__ void flush(float* xo, int lane) {
        const float ratio = up_sum > 0.f ? up / up_sum : 0.f;
#pragma unroll
        for (int h = 0; h < HL; h++) {
            const float f = up_sum > 0.f ? fast_exp2(m_sum[h] - m_run[h]) : 0.f;
            l_sum[h] = fmaf(l_sum[h], f, l_run[h]);
            z_sum[h] = fmaf(z_sum[h], f, z_run[h]);
            l_run[h] = z_run[h] = 0.f;
            m_sum[h] = m_run[h];
#pragma unroll
            for (int mt = 0; mt < NMT; mt++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    float* at = xo + (mt * 2 * HL + j * HL + h) * 32 + lane;
                    *at = up_sum > 0.f ? fmaf(*at, f * ratio, oacc[mt][j * HL + h]) : oacc[mt][j * HL + h];
                    oacc[mt][j * HL + h] = 0.f;
                }
        }
        up_sum = up;
    }
    // a lane's value slice (at the 4-byte aligned `at`, `sh` = 8 * the bytes it starts behind it)
    static __device__ __forceinline__ void load_slice(uint32_t at, uint32_t sh, uint32_t (&w)[VW]) {
        if constexpr (WIDE || VSB % 8 != 0) {
            lds_slice<VSB>(at, sh, w);
        } else {
#pragma unroll
            for (int i = 0; i < VW; i++) w[i] = lds32(at + 4 * i);
        }
    }

    // token 0 at `page`, `row` bytes apart; tokens [lo, hi) count
    __device__ __forceinline__ void page(uint32_t page, uint32_t row, int lo, int hi, bool, int lane) {
        const int g = lane >> 2, tg = lane & 3;
        // ---- scores: chains of NKB / CH MMAs (an MMA's sum is truncated, the sums of the chains'
        // results are rounded)
        constexpr int CH = CHAINS;
        float c[NH][CH][4];
        const uint32_t rowa = page + g * row, rowb = rowa + 8 * row;
#pragma unroll
        for (int q = 0; q < NKB / 4; q++) {
            uint32_t wa[4], wb[4];
            if constexpr (WIDE) {
                const uint4 ka = lds128(rowa + (D / 4) * tg + 16 * q), kb4 = lds128(rowb + (D / 4) * tg + 16 * q);
                wa[0] = ka.x; wa[1] = ka.y; wa[2] = ka.z; wa[3] = ka.w;
                wb[0] = kb4.x; wb[1] = kb4.y; wb[2] = kb4.z; wb[3] = kb4.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    wa[j] = lds32(rowa + 4 * tg + 16 * (4 * q + j));
                    wb[j] = lds32(rowb + 4 * tg + 16 * (4 * q + j));
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                auto half2_of = [](uint32_t two) {
                    const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(two), __NV_E4M3);
                    return static_cast<uint32_t>(r.x) | (static_cast<uint32_t>(r.y) << 16);
                };
                const uint32_t a0 = half2_of(wa[j] & 0xffffu), a2 = half2_of(wa[j] >> 16);
                const uint32_t a1 = half2_of(wb[j] & 0xffffu), a3 = half2_of(wb[j] >> 16);
#pragma unroll
                for (int x = 0; x < NH; x++) {
                    const int kb = 4 * q + j;
                    if (kb < CH) mma_16816_z(c[x][kb % CH], a0, a1, a2, a3, qb[x][kb][0], qb[x][kb][1]);
                    else mma_16816(c[x][kb % CH], a0, a1, a2, a3, qb[x][kb][0], qb[x][kb][1]);
                }
            }
        }

        // ---- online softmax (base-2 exponents), the lane's tokens g and g + 8
        const bool okA = g >= lo && g < hi, okB = g + 8 >= lo && g + 8 < hi;
        const uint32_t ma = lds32(rowa + D + PDV), mb = lds32(rowb + D + PDV);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&ma));
        const float2 fb = __half22float2(*reinterpret_cast<const __half2*>(&mb));
        const float vsa = okA ? fa.x : 0.f, vsb = okB ? fb.x : 0.f;
        // the code nearest to the value 0 and what it is off by
        auto code0 = [](float2 m) { return fminf(fmaxf(rintf(__fdividef(-m.y, m.x)), 0.f), static_cast<float>((1 << VB) - 1)); };
        const float ca = code0(fa), cb = code0(fb);
        const float vza = okA ? fmaf(ca, fa.x, fa.y) : 0.f;
        const float vzb = okB ? fmaf(cb, fb.x, fb.y) : 0.f;
        float ra[HL], rb[HL], sa[HL], sb[HL];   // products; scaled scores
        const float s_max = fmaxf(fabsf(vsa), fabsf(vsb));
        bool above = s_max > s_ref;
#pragma unroll
        for (int h = 0; h < HL; h++) {
            // sum of a column over the chains
            auto total = [&](const float (&x)[CH][4], int i) {
                float t[CH];
#pragma unroll
                for (int z = 0; z < CH; z++) t[z] = x[z][i];
#pragma unroll
                for (int w = CH / 2; w > 0; w /= 2)
#pragma unroll
                    for (int z = 0; z < w; z++) t[z] += t[z + w];
                return t[0];
            };
            constexpr int LO = NH - 1;   // where the lo parts are: the next column, or the second MMA
            ra[h] = fmaf(total(c[LO], NH == 1 ? 1 : h), kInvLo, total(c[0], h));
            rb[h] = fmaf(total(c[LO], NH == 1 ? 3 : 2 + h), kInvLo, total(c[0], 2 + h));
            sa[h] = okA ? ra[h] * mul[h] : -INFINITY;
            sb[h] = okB ? rb[h] * mul[h] : -INFINITY;
            above |= fmaxf(sa[h], sb[h]) > m_run[h];   // (no slack: a weight is at most the value scale)
        }
        if (__any_sync(0xffffffffu, above)) {
            // the page's largest value scale, rounded up to a power of two, brought to 2^14: no weight
            // leaves fp16's range, and one below its normal numbers is 2^-28 of the largest possible
            float top = s_max;
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            float shift = 1.f;
            if (top > s_ref) {   // (warp-uniform; a power of two >= 2^-24)
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
                const float m_new = fmaxf(m_run[h], m);   // finite: the page's first token is valid
                corr[h] = fast_exp2(m_run[h] - m_new);
                l_run[h] *= corr[h];
                z_run[h] *= corr[h];
                m_run[h] = m_new;
            }
#pragma unroll
            for (int mt = 0; mt < NMT; mt++)
#pragma unroll
                for (int i = 0; i < 2 * HL; i++) oacc[mt][i] *= corr[i % HL] * shift;
        }
        uint32_t pb[NH][2];
        {
            float wa[HL], wb[HL];
            const float sua = vsa * up, sub = vsb * up;   // (exact)
#pragma unroll
            for (int h = 0; h < HL; h++) {
                // (the exponent in one rounding)
                const float pa = okA ? fast_exp2(fmaf(ra[h], mul[h], -m_run[h])) : 0.f;
                const float pbv = okB ? fast_exp2(fmaf(rb[h], mul[h], -m_run[h])) : 0.f;
                l_run[h] += pa + pbv;
                z_run[h] = fmaf(pa, vza, fmaf(pbv, vzb, z_run[h]));
                wa[h] = pa * sua;
                wb[h] = pbv * sub;
            }
            if constexpr (NH == 1) {
                pb[0][0] = movmatrix_trans(pack(wa[0], residual(wa[0])));
                pb[0][1] = movmatrix_trans(pack(wb[0], residual(wb[0])));
            } else {
                pb[0][0] = movmatrix_trans(pack(wa[0], wa[HL - 1]));
                pb[0][1] = movmatrix_trans(pack(wb[0], wb[HL - 1]));
                pb[NH - 1][0] = movmatrix_trans(pack(residual(wa[0]), residual(wa[HL - 1])));
                pb[NH - 1][1] = movmatrix_trans(pack(residual(wb[0]), residual(wb[HL - 1])));
            }
        }

        // ---- O^T += V^T.P^T.  Codes become fp16 arithmetically: or-ed into the mantissa of 1024 a
        // code at bit s is 1024 + 2^s * code, and one packed FMA scales it and takes the token's code of
        // zero off exactly (s >= 1: 2^(10 - s) + code is then an fp16 number).  A 16-bit half of x holds
        // the next codes of one token, the other half those of its neighbour.
        const uint32_t czero = pack(ca, cb);   // tokens g, g + 8
        const uint32_t c_even = __shfl_sync(0xffffffffu, czero, 9 * tg), c_odd = __shfl_sync(0xffffffffu, czero, 9 * tg + 4);
        const uint32_t c01 = __byte_perm(c_even, c_odd, 0x5410u), c23 = __byte_perm(c_even, c_odd, 0x7632u);
        uint32_t v[4][VW];
        const uint32_t vrow = page + D + slice_word<VSB>(g) + 2 * tg * row;
        const uint32_t vsh = slice_shift<VSB>(g);
        load_slice(vrow, vsh, v[0]);
        load_slice(vrow + row, vsh, v[1]);
        load_slice(vrow + 8 * row, vsh, v[2]);
        load_slice(vrow + 9 * row, vsh, v[3]);
        constexpr int CPW = VB == 3 ? 5 : 16 / VB;     // whole codes in 16 bits
        constexpr int CLO = VB == 3 ? 3 : CPW / 2;     // ... of which the first CLO are read from x << 1
        constexpr int DOWN = VB * CLO - 1;             // the others from x >> DOWN
        uint32_t h01[D / 8], h23[D / 8];               // [coordinate] tokens 2tg, 2tg + 1 / 2tg + 8, 2tg + 9
        auto window = [&](const uint32_t (&a)[VW], const uint32_t (&b)[VW], int bit) {
            const int j = bit >> 5, sh = bit & 31;
            const uint32_t hi_a = a[j + 1 < VW ? j + 1 : j], hi_b = b[j + 1 < VW ? j + 1 : j];
            const uint32_t x = sh == 0 ? a[j] : sh + 16 <= 32 ? a[j] >> sh : __funnelshift_r(a[j], hi_a, sh);
            const uint32_t y = sh == 0 ? b[j] : sh + 16 <= 32 ? b[j] >> sh : __funnelshift_r(b[j], hi_b, sh);
            return __byte_perm(x, y, 0x5410u);
        };
        auto code_half2 = [&](uint32_t above1, uint32_t below, int i, uint32_t zero) {
            const int sh = i < CLO ? VB * i + 1 : VB * i - DOWN;
            const uint32_t w = ((i < CLO ? above1 : below) & (((1u << VB) - 1u) * 0x00010001u << sh)) | 0x64006400u;
            const float inv = 1.f / static_cast<float>(1 << sh), off = -1024.f * inv;
            const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&w), __floats2half2_rn(inv, inv),
                                      __hsub2(__floats2half2_rn(off, off), *reinterpret_cast<const __half2*>(&zero)));
            return *reinterpret_cast<const uint32_t*>(&r);
        };
#pragma unroll
        for (int w = 0; w < (D / 8 + CPW - 1) / CPW; w++) {
            const uint32_t x = window(v[0], v[1], w * CPW * VB), y = window(v[2], v[3], w * CPW * VB);
#pragma unroll
            for (int i = 0; i < CPW; i++) {
                if (w * CPW + i >= D / 8) break;
                h01[w * CPW + i] = code_half2(x << 1, x >> DOWN, i, c01);
                h23[w * CPW + i] = code_half2(y << 1, y >> DOWN, i, c23);
            }
        }
        // (a page's sum is a new MMA chain, added in fp32: sums over many pages stay rounded, not truncated)
#pragma unroll
        for (int mt = 0; mt < NMT; mt++) {
            float o[NH][4];
#pragma unroll
            for (int x = 0; x < NH; x++)
                mma_16816_z(o[x], h01[2 * mt], h01[2 * mt + 1], h23[2 * mt], h23[2 * mt + 1], pb[x][0], pb[x][1]);
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int h = 0; h < HL; h++)
                    oacc[mt][j * HL + h] += fmaf(NH == 1 ? o[0][2 * j + 1] : o[NH - 1][2 * j + h], kInvLo, o[0][2 * j + h]);
        }
    }
    // the lane's state: OL floats at xo[f * 32 + lane], (m, l, z) of its heads at xml[0..2][8]
    __device__ __forceinline__ void publish(float* xo, float* xml, int lane, bool poison) {
        if constexpr (FLUSH > 0) {
            flush(xo, lane);
#pragma unroll
            for (int h = 0; h < HL; h++) {
                l_run[h] = l_sum[h];
                z_run[h] = z_sum[h];
            }
#pragma unroll
            for (int f = 0; f < OL; f++) xo[f * 32 + lane] *= 1.f / up;
        } else {
#pragma unroll
            for (int mt = 0; mt < NMT; mt++)
#pragma unroll
                for (int i = 0; i < 2 * HL; i++) xo[(mt * 2 * HL + i) * 32 + lane] = oacc[mt][i] * (1.f / up);
        }
#pragma unroll
        for (int h = 0; h < HL; h++)
#pragma unroll
            for (int m = 4; m < 32; m <<= 1) {
                l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], m);
                z_run[h] += __shfl_xor_sync(0xffffffffu, z_run[h], m);
            }
        if (lane < 4) {
#pragma unroll
            for (int h = 0; h < HL; h++) {
                xml[HL * lane + h] = poison ? __int_as_float(0x7fc00000) : m_run[h];
                xml[8 + HL * lane + h] = l_run[h];
                xml[16 + HL * lane + h] = z_run[h];
            }
        }
    }
    // head and coordinate of output float f = (m-tile, row g or g + 8, head) of lane ln
    static __device__ __forceinline__ int head_of(int f, int ln) { return HL * (ln & 3) + f % HL; }
    __device__ __forceinline__ int coord_of(int f, int ln) const { return (D / 8) * (ln >> 2) + f / HL; }
};

template <int D, int VB, int NH>
struct TqFp8Cfg {
    using Engine = TqFp8<D, VB, NH, true>;
    static constexpr int WARPS = 8, THREADS = 32 * WARPS;
    static constexpr int USED = D + D * VB / 8 + 4, NW = USED / 4;      // bytes and words of a slot
    // an odd number of 16-byte units: the rows g, g + 1 of a 16-byte load fall into distinct banks
    static constexpr int ROWB = ((USED + 15) / 16 | 1) * 16;
    static constexpr int PAGE = kPageTokens * ROWB;
    static constexpr int STAGES = NH == 1 ? 3 : 2;
    static constexpr int OL = Engine::OL;
    static constexpr int QS = 4 * NH * Engine::QROW * 4;
    static constexpr int XO = WARPS * 32 * OL * 4, XML = WARPS * 3 * 8 * 4;
    static constexpr int SMEM_BYTES = WARPS * STAGES * PAGE + QS + XO + XML + 64;
    static_assert(USED % 4 == 0 && 2 * SMEM_BYTES <= 226 * 1024, "two CTAs per SM");
};

template <int D, int VB, int NH>
__global__ void __launch_bounds__(TqFp8Cfg<D, VB, NH>::THREADS, 2)
tq_fp8_kernel(const TqDecodeParams p, int n_items) {
    using C = TqFp8Cfg<D, VB, NH>;
    using Engine = typename C::Engine;
    constexpr int WARPS = C::WARPS;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) + warp * C::STAGES * C::PAGE;
    float* qs = reinterpret_cast<float*>(smem_raw + WARPS * C::STAGES * C::PAGE);   // [4 * NH][QROW]
    float* xo = qs + C::QS / 4;                                                    // [WARPS][OL][32]
    float* xml = xo + C::XO / 4;                                                   // [WARPS][3][8]
    const int group = p.Hq / p.Hkv;

    struct Item { int sid, hkv, b, bs, layer, t0, t1, n_pages; };
    auto item_info = [&](int item) {
        Item it;
        it.sid = item % p.splits;
        const int r = item / p.splits;
        it.hkv = r % p.Hkv;
        it.b = r / p.Hkv;   // (layer, sequence) row
        it.layer = static_cast<int>(fast_div(static_cast<uint32_t>(it.b), p.div_bseq));
        it.bs = it.b - it.layer * p.B_seq;
        const int seq_len = p.seq_lens[it.bs];
        const int kv_start = p.kv_start ? p.kv_start[it.bs] : 0;
        const int split_len = (seq_len - kv_start + p.splits - 1) / p.splits;
        it.t0 = kv_start + split_len * it.sid;
        it.t1 = min(it.t0 + split_len, seq_len);
        it.n_pages = it.t1 > it.t0 ? (it.t1 - it.t0 + kPageTokens - 1) / kPageTokens : 0;
        return it;
    };
    auto mid_row = [&](const Item& it, int h) {
        return p.mid_o + ((static_cast<int64_t>(it.b) * p.Hq + it.hkv * group + h) * p.splits + it.sid) * (D + 1);
    };

    // ---- copies: the warp's pages of all its items, in the order of the arithmetic below
    int c_item = blockIdx.x, c_page = warp, c_stage = 0;
    uint32_t stage_bad = 0;   // bit s: a block id of the page in ring buffer s was out of range
    Item c_it = item_info(c_item < n_items ? c_item : 0);
    auto copy_next = [&]() {
        while (c_item < n_items && c_page >= c_it.n_pages) {
            c_item += gridDim.x;
            c_page = warp;
            if (c_item < n_items) c_it = item_info(c_item);
        }
        if (c_item < n_items) {   // (warp-uniform)
            // tokens past the end of the range re-read the last valid slot (their weight is zero)
            const int pos = min(c_it.t0 + c_page * kPageTokens + (lane & 15), c_it.t1 - 1);
            const uint32_t blk = fast_div(static_cast<uint32_t>(pos), p.div_block);
            const uint32_t off = static_cast<uint32_t>(pos) - blk * p.block_size;
            int64_t id = p.block_table[static_cast<int64_t>(c_it.bs) * p.max_blocks + blk];
            const bool bad = p.num_blocks > 0 && static_cast<uint64_t>(id) >= static_cast<uint64_t>(p.num_blocks);
            if (bad) id = 0;
            const bool any_bad = __any_sync(0xffffffffu, bad);
            stage_bad = (stage_bad & ~(1u << c_stage)) | (static_cast<uint32_t>(any_bad) << c_stage);
            const uint8_t* sp = p.kv_cache + c_it.layer * p.cache_layer_stride + id * p.stride_block +
                                off * p.stride_pos + c_it.hkv * p.stride_head;
            const uint32_t dst = ring + c_stage * C::PAGE + 4 * (lane & 7);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int tk = (lane >> 3) + 4 * k;
                const uint8_t* src = reinterpret_cast<const uint8_t*>(__shfl_sync(
                                         0xffffffffu, reinterpret_cast<unsigned long long>(sp), tk)) + 4 * (lane & 7);
#pragma unroll
                for (int j = 0; j < (C::NW + 7) / 8; j++)
                    if (8 * j + 7 < C::NW || 8 * j + (lane & 7) < C::NW)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst + tk * C::ROWB + 32 * j),
                                     "l"(src + 32 * j));
            }
            c_page += WARPS;
        }
        cp_async_commit();
        c_stage = c_stage + 1 == C::STAGES ? 0 : c_stage + 1;
    };
#pragma unroll
    for (int i = 0; i < C::STAGES - 1; i++) copy_next();
    int stage = 0;

    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        const Item it = item_info(item);
        if (it.n_pages == 0) {   // neutral partial (CTA-uniform): zeros and lse = -inf
            for (int idx = tid; idx < group * (D + 1); idx += C::THREADS) {
                const int h = idx / (D + 1), d = idx - h * (D + 1);
                mid_row(it, h)[d] = d == D ? -INFINITY : 0.f;
            }
            continue;
        }
        __syncthreads();   // (the item before has been folded)
        if (warp < NH)
            Engine::rotate_four(p, qs, static_cast<int64_t>(it.b) * p.Hq + it.hkv * group, group, lane, warp);
        __syncthreads();
        Engine e;
        e.begin(qs, lane);
        bool bad_block = false;

        for (int pg = warp; pg < it.n_pages; pg += WARPS) {
            cp_async_wait<C::STAGES - 2>();
            __syncwarp();   // the page is there for every lane; everybody is done with the one before
            const uint32_t page = ring + stage * C::PAGE;
            bad_block |= ((stage_bad >> stage) & 1u) != 0u;
            copy_next();
            stage = stage + 1 == C::STAGES ? 0 : stage + 1;

            e.page(page, C::ROWB, 0, it.t1 - it.t0 - pg * kPageTokens, false, lane);
        }

        // ---- fold the warps' states
        e.publish(xo + warp * C::OL * 32, xml + warp * 24, lane, false);
        const bool any_bad = __syncthreads_or(bad_block) != 0;
        for (int i = tid; i < C::OL * 32; i += C::THREADS) {
            const int ln = i & 31, f = i >> 5, h = Engine::head_of(f, ln);
            if (h >= group) continue;
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < WARPS; w++) M = fmaxf(M, xml[(w * 3 + 0) * 8 + h]);
            float o = 0.f, l = 0.f, z = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; w++) {
                const float s = fast_exp2(xml[(w * 3 + 0) * 8 + h] - M);   // (a warp without pages: 0)
                o = fmaf(xo[(w * C::OL + f) * 32 + ln], s, o);
                l = fmaf(xml[(w * 3 + 1) * 8 + h], s, l);
                z = fmaf(xml[(w * 3 + 2) * 8 + h], s, z);
            }
            float* dst = mid_row(it, h);
            const int coord = e.coord_of(f, ln);
            dst[coord] = (o + z) / l;
            if (coord == 0) dst[D] = any_bad ? __int_as_float(0x7fc00000) : M * kLn2 + logf(l);
        }
    }
    cp_async_wait<0>();
}

}  // namespace ftq
