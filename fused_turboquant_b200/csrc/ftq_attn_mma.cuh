// Arithmetic of the tensor-core kernel of paged decode attention (ftq_attn_flow.cuh); its look-ups, MMAs and
// copies serve the slot-format and chunk kernels too.  Whole 16-token pages arrive in a per-warp ring by 1-D bulk copies (TMA), every lane
// copies its slices to registers, the codes are dequantised through a
// bank-conflict-free shared-memory table and feed warp-level m16n8k16 fp16 MMAs
// (fp32 accumulate).  With a GQA
// group of G query heads the products are skinny GEMMs (G x D x tokens), so the
// per-element work no longer grows with G and every packed byte is dequantised
// exactly once per KV head.
//
// Same mathematics as attn_split_kernel (ftq_attn.cuh), i.e. the fused
// formulation of src/fused_turboquant/kernels/triton_flash_decode.py:33-324 in the
// reference; centroids, the rotated query and the softmax weights are rounded
// to fp16 before the MMAs, accumulation is fp32.  The V centroids are multiplied
// by a host-chosen factor in [1, 2) before the rounding (and the weights divided
// by it): a common rounding bias of the centroids would otherwise add up over
// all coordinates into one output element through the inverse rotation.
//
// Tables: an entry holds the fp16 centroids of two adjacent codes, replicated for the 32 lanes so that
// bank = lane (no conflicts whatever the codes are); struct Window below says how codes of 4, 3 and 2 bits find
// their entry.  (The slot-format kernels' 3- and 2-bit codes use 128-byte rows in a table aligned to its own
// size: shift + and/or, entry_addr.)
//
// Fragment maps for one 16-token page (lane = 4*g + tg), GQA group <= 4 (NH = 1):
//   S = K.Q^T :  A = K [16 tokens x 16 coords]: rows g / g+8 = page tokens rho(g) / rho(g)+2,
//                    k-block kb covers coordinates (D/4)*tg + 4*kb + {0..3}
//                B = Q^T[16 coords x 8]: column n = head n>>1 (each head twice)
//                C[token][head tg]  (columns 2tg and 2tg+1 are the same head)
//   the weights p*vnorm are rounded to fp16 and transposed with movmatrix, which
//   hands lane (g, tg) the weights of head g>>1 for page tokens 4tg .. 4tg+3;
//   O^T = V^T.P^T with reduction index k = (token, parity of d), so that the fp16
//   pair a table lookup returns, (V[t,d], V[t,d+1]), is directly an A register:
//                A[row = d-pair][k = (token, parity)] = V[token][2*pair + parity]
//                B[k = (token, parity)][n = (head n>>1, parity n&1)] = p or 0
//                C[d-pair][(head tg, parity)]: lane (g,tg) owns O[head tg][(D/8)g .. +D/8)
// GQA group 5 .. 8 (NH = 2): the eight columns are eight heads,
//   S:  B column n = head n;  C[token][heads 2tg, 2tg + 1]; the two weights of a token are packed
//                into one fp16 pair, and movmatrix turns the packed scores of tokens rho(0..7)
//                (rho(0..7) + 2) straight into the B registers of P.V: head g, tokens 4tg, 4tg + 1
//                (4tg + 2, 4tg + 3);
//   O^T += V^T.P^T with k = token:  A[row g / g+8 = coordinate (D/8)g + 2mt / + 1][k = token]: the
//                codes of two tokens are merged into pairs before the look-up (Window::merge);
//                C[coordinate pair][heads 2tg, 2tg + 1].
//   Against two passes of the 4-head map this halves the MMAs and the softmax bookkeeping.
// In both maps a lane dequantises the K slices (D/4 coordinates) of two tokens and the V
// slices (D/8 coordinates) of four tokens per page, all contiguous bytes, every
//   code exactly once per KV head.
#pragma once

#include <type_traits>

#include "ftq_attn.cuh"

namespace ftq {

constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

// (not volatile: a pure function of its operands, so the compiler may interleave the MMAs
// with the table lookups of later k-blocks)
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
// Lookup in a dequantisation table: the tables never change after the CTA-wide barrier that
// follows their construction and every address derives from page data read after that barrier,
// so the load may be scheduled freely (not volatile).
template <int OFFSET = 0>
__device__ __forceinline__ uint32_t lut32(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1+%2];\n" : "=r"(v) : "r"(addr), "n"(OFFSET));
    return v;
}

__device__ __forceinline__ uint2 lut64(uint32_t addr) {
    uint2 v;
    asm("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

#ifndef FTQ_LAZY_SLACK
#define FTQ_LAZY_SLACK 3
#endif
// slack of the lazy reference maximum of the online softmax (base-2 exponent units)
constexpr float kLazyMaxSlack = static_cast<float>(FTQ_LAZY_SLACK);
// m16n8k16 with a zero accumulator input (saves clearing the accumulators of every page)
__device__ __forceinline__ void mma_16816_z(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                            uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};\n"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t f2h_sat(float x) {
    unsigned short h;
    asm("cvt.rn.satfinite.f16.f32 %0, %1;\n" : "=h"(h) : "f"(x));
    return h;
}

__device__ __forceinline__ uint32_t f2h2_sat(float lo, float hi) {
    uint32_t h;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;\n" : "=r"(h) : "f"(hi), "f"(lo));
    return h;
}

// ---- mbarrier + bulk-copy (TMA, 1-D, no multicast) helpers; all addresses are shared-window
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// Bulk copy with an L2 policy: KV pages are read once per decode step, so L2 is told to drop
// them first (measured on B200: +1.5 % on the Llama-shaped K4V4 batch).
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void bulk_g2s_hint(uint32_t dst, const void* src, uint32_t bytes,
                                              uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::
            "r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
        : "memory");
}
// Bounded wait: gives up after kMbarSpinLimit polls (each poll may itself block for a
// hardware-defined slice) and reports failure instead of hanging the SM.
// FTQ_TEST_WAIT_EXPIRY (only the test library of build.py defines it): warp 5 of CTA 0 announces its
// first page copy to the mbarrier but does not issue it, and the poll limit is small -- the wait
// runs out, which is the one way to execute the give-up path (NaN rows, status word) on purpose.
#ifdef FTQ_TEST_WAIT_EXPIRY
constexpr int kMbarSpinLimit = 1 << 6;
#else
constexpr int kMbarSpinLimit = 1 << 20;
#endif
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {   // one poll
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kMbarSpinLimit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// A lane's slice of SB packed bytes into ceil(SB/4) words.  `addr` is the 4-byte aligned address at
// or below the slice's start and `sh` 8 * the bytes between the two (both are lane constants, see
// slice_word / slice_shift; whole-word slices ignore `sh`).  Slices of 6 and 3 bytes come out of
// two words with funnel shifts; bits beyond the slice are junk that pair_index masks (the second
// word of a row's last slice may lie behind the row, never behind the page).
template <int SB>
__device__ __forceinline__ constexpr uint32_t slice_word(int idx) { return (SB * idx) & ~3; }
template <int SB>
__device__ __forceinline__ constexpr uint32_t slice_shift(int idx) { return 8 * ((SB * idx) & 3); }
template <int SB>
__device__ __forceinline__ void lds_slice(uint32_t addr, uint32_t sh, uint32_t (&w)[(SB + 3) / 4]) {
    if constexpr (SB % 16 == 0) {
#pragma unroll
        for (int i = 0; i < SB / 16; i++) {
            const uint4 v = lds128(addr + 16 * i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    } else if constexpr (SB % 8 == 0) {
#pragma unroll
        for (int i = 0; i < SB / 8; i++) {
            const uint2 v = lds64(addr + 8 * i);
            w[2 * i] = v.x; w[2 * i + 1] = v.y;
        }
    } else if constexpr (SB % 4 == 0) {
#pragma unroll
        for (int i = 0; i < SB / 4; i++) w[i] = lds32(addr + 4 * i);
    } else if constexpr (SB == 6) {
        const uint32_t x0 = lds32(addr), x1 = lds32(addr + 4);
        w[0] = __funnelshift_r(x0, x1, sh);
        w[1] = x1 >> sh;
    } else if constexpr (SB == 3) {
        const uint32_t x0 = lds32(addr), x1 = lds32(addr + 4);
        w[0] = __funnelshift_r(x0, x1, sh);
    } else {
        static_assert(SB == 2, "unsupported slice size");
        w[0] = lds32(addr) >> sh;
    }
}

// Shared-memory address of the table entry for code pair `pair` of a slice.
//   IW == 8 (4-bit): lane_base = window | table half | lane*4; the code byte becomes byte 1.
//   IW  < 8        : lane_base = table | lane*4; entry * 128 is or-ed in.
template <int IW, int NW>
__device__ __forceinline__ uint32_t entry_addr(const uint32_t (&w)[NW], int pair, uint32_t lane_base) {
    if constexpr (IW == 8) {
        const int j = pair >> 2, k = pair & 3;
        return __byte_perm(w[j], lane_base, 0x7604u | (static_cast<uint32_t>(k) << 4));
    } else {
        return lane_base | pair_index<IW>(w, pair);
    }
}

// A dequantisation window: 256 rows of 256 bytes, each row the 32-fold copies of two entries ("columns" of 128
// bytes), indexed by a whole byte of the packed codes: the address of a look-up is ONE byte-permute, the byte dropped
// into bits 8..15 of the lane's base address.
//   4-bit codes: a byte is a pair of codes.
//   2-bit codes: a byte is four codes, an entry eight bytes (sixteen copies).
//   3-bit codes: a pair is six of a byte's bits.  Of the four pairs in 24 bits, the first is the low six bits of byte 0
//     and the last the high six of byte 2; of the codes shifted right by four, the second is the high six of byte 0
//     and the third the low six of byte 1.  With both columns (BOTH: one codebook for keys and values; column 0 by the
//     low six bits, column 1 by the high six) that is one shift and four byte-permutes for four look-ups, with
//     the low six bits alone three shifts.
// The ALU pipe bounds the 3-bit page loop (64 % busy when a shift and an and-or, three instructions where a pair
// straddles words, made an index): 24 layers of 32 x 4096 tokens, 14 / 2 heads of 64, 152 -> 139 us, 4 x 131072, 64 / 8
// heads of 128, 159 -> 138 us by these tables and `merge` alone.
template <int BITS, bool BOTH>
struct Window {
    static constexpr int NS = BITS != 3 ? 0 : BOTH ? 1 : 3;   // shifted copies of the codes
    template <int NW>
    struct Run {              // consecutive codes of a lane: NW words
        uint32_t w[NW];
        uint32_t s[NS > 0 ? NS : 1][NW];
    };
    template <int NW>
    static __device__ __forceinline__ void shift(Run<NW>& r) {
#pragma unroll
        for (int k = 0; k < NS; k++)
#pragma unroll
            for (int j = 0; j < NW; j++) {
                const int sh = BOTH ? 4 : 6 - 2 * k;
                r.s[k][j] = j + 1 < NW ? __funnelshift_r(r.w[j], r.w[j + 1], sh) : r.w[j] >> sh;
            }
    }
    // centroids of the code pairs 2i and 2i + 1
    template <int NW>
    static __device__ __forceinline__ void pairs(const Run<NW>& r, int i, uint32_t base, uint32_t& x, uint32_t& y) {
        auto at = [&](const uint32_t (&w)[NW], int byte) {
            return __byte_perm(w[byte >> 2], base, 0x7604u | (static_cast<uint32_t>(byte & 3) << 4));
        };
        if constexpr (BITS == 4) {
            x = lut32(at(r.w, 2 * i));
            y = lut32(at(r.w, 2 * i + 1));
        } else if constexpr (BITS == 2) {
            const uint2 e = lut64(at(r.w, i));
            x = e.x; y = e.y;
        } else if (i % 2 == 0) {
            const int b = 3 * (i / 2);
            x = lut32(at(r.w, b));
            y = BOTH ? lut32<128>(at(r.s[0], b)) : lut32(at(r.s[0], b));
        } else {
            const int b = 3 * (i / 2);
            x = lut32(at(r.s[BOTH ? 0 : 1], b + 1));
            y = BOTH ? lut32<128>(at(r.w, b + 2)) : lut32(at(r.s[BOTH ? 0 : 2], b + 2));
        }
    }
    // codes of two tokens, a and b, merged into the pairs (a[2f], b[2f]) and (a[2f + 1], b[2f + 1])
    template <int NW>
    static __device__ __forceinline__ void merge(const uint32_t (&a)[NW], const uint32_t (&b)[NW], Run<NW>& even, Run<NW>& odd) {
#pragma unroll
        for (int j = 0; j < NW; j++) {
            uint32_t m = 0;      // the bits of the even codes
#pragma unroll
            for (int i = 0; i < 32; i++) m |= (32 * j + i) % (2 * BITS) < BITS ? 1u << i : 0u;
            const uint32_t up = j > 0 && BITS == 3 ? __funnelshift_l(b[j > 0 ? j - 1 : 0], b[j], BITS) : b[j] << BITS;
            const uint32_t down = j + 1 < NW && BITS == 3 ? __funnelshift_r(a[j], a[j + 1 < NW ? j + 1 : j], BITS) : a[j] >> BITS;
            even.w[j] = (a[j] & m) | (up & ~m);
            odd.w[j] = (down & m) | (b[j] & ~m);
        }
    }
};

template <int D, int BK, int BV, int NH>
struct MmaCfg {
    static constexpr int NKB = D / 16;                  // k-blocks of K.Q^T
    static constexpr int NMT = D / 32;                  // m-tiles of O^T
    static constexpr int PDK = packed_dim(D, BK), PDV = packed_dim(D, BV);
    static constexpr int KSB = PDK / 4, VSB = PDV / 8;  // slice bytes per lane
    static constexpr int KW = (KSB + 3) / 4, VW = (VSB + 3) / 4;   // ... in words
    static constexpr int OFF_KN = kPageTokens * PDK;
    static constexpr int OFF_VC = OFF_KN + 2 * kPageTokens;
    static constexpr int OFF_VN = OFF_VC + kPageTokens * PDV;
    static constexpr int PAGE_BYTES = OFF_VN + 2 * kPageTokens;
    static constexpr int STATE_F4 = NH * NMT;                    // float4 items per lane
};

// One page worth of packed data in registers (per lane).
template <int KSB, int VSB>
struct PageRegs {
    uint32_t k[2][(KSB + 3) / 4];  // K slice tg of page tokens rho(g), rho(g) + 2
    uint32_t v[4][(VSB + 3) / 4];  // V slice g of page tokens 4tg .. 4tg+3
    uint2 kn, vn;                  // fp16 norms of page tokens 4(g>>1) .. 4(g>>1)+3
};

__device__ __forceinline__ float half_bits_to_float(uint32_t h16) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h16)));
}

__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}

}  // namespace ftq
