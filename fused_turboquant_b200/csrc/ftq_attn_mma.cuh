// What the tensor-core kernels of paged decode attention share (ftq_attn_flow.cuh: equal
// shares of pages per CTA; ftq_attn_stream.cuh: streaming warps): whole
// 16-token pages arrive in a per-warp ring by 1-D bulk copies (TMA), every lane
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
// Tables: an entry holds the fp16 centroids of two adjacent codes, replicated
// for the 32 lanes so that bank = lane (no conflicts whatever the codes are).
// 4-bit codes index by byte: the table occupies a 64 KB-aligned window with
// 256-byte rows, so that the address is one byte-permute -- the code byte
// dropped into bits 8..15 of the lane's base address.  3- and 2-bit codes use
// 128-byte rows in a table aligned to its own size (shift + and/or).
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
//                pairs of two tokens' look-ups are exchanged with two byte-permutes;
//                C[coordinate pair][heads 2tg, 2tg + 1].
//   Against two passes of the 4-head map this halves the MMAs and the softmax bookkeeping for one
//   byte-permute per value look-up.
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
__device__ __forceinline__ uint32_t lut32(uint32_t addr) {
    uint32_t v;
    asm("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
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

// The sixteen 2-bit codes c0 .. c15 of a word as fp16 centroid pairs, without a table: a byte-permute picks
// the two bytes of a centroid out of the eight of all four (`lo` = centroids 0 and 1, `hi` = 2 and 3).  Its
// selector is 2c, 2c + 1, i.e. 0x22 * c + 0x10, for four codes at a time.  x[2i] = (c[i], c[i + 4]),
// x[2i + 1] = (c[i + 8], c[i + 12]).
__device__ __forceinline__ void select_pairs2(uint32_t w, uint32_t lo, uint32_t hi, uint32_t (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t m = (w >> (2 * i)) & 0x03030303u;
        x[2 * i] = __byte_perm(lo, hi, m * 0x22u + 0x10101010u);
        x[2 * i + 1] = __byte_perm(lo, hi, (m * 0x22u + 0x10101010u) >> 16);
    }
}

template <int D, int BK, int BV, int NH>
struct MmaCfg {
    static constexpr int NKB = D / 16;                  // k-blocks of K.Q^T
    static constexpr int NMT = D / 32;                  // m-tiles of O^T
    static constexpr int PDK = packed_dim(D, BK), PDV = packed_dim(D, BV);
    static constexpr int KSB = PDK / 4, VSB = PDV / 8;  // slice bytes per lane
    static constexpr int KW = (KSB + 3) / 4, VW = (VSB + 3) / 4;   // ... in words
    static constexpr int IWK = 2 * BK, IWV = 2 * BV;    // table index width (two codes)
    static constexpr bool BYTE = BK == 4 || BV == 4;    // a 64 KB byte-indexed window is used
    static constexpr int OFF_KN = kPageTokens * PDK;
    static constexpr int OFF_VC = OFF_KN + 2 * kPageTokens;
    static constexpr int OFF_VN = OFF_VC + kPageTokens * PDV;
    static constexpr int PAGE_BYTES = OFF_VN + 2 * kPageTokens;
    // small (non-byte) tables, each aligned to its own size
    static constexpr int TKS = BK == 4 ? 0 : (1 << IWK) * 128;
    // 2-bit values next to 4-bit keys: the upper half of every row of the key's byte window holds,
    // 16 times, the FOUR centroids of a value byte (8 bytes), so one byte-permute + one 8-byte
    // load dequantise four codes (instead of shift/and + two 4-byte loads)
    static constexpr bool V2BYTE = BK == 4 && BV == 2;
    static constexpr int TVS = (BV == 4 || V2BYTE) ? 0 : (1 << IWV) * 128;
    static constexpr int SMALL_ALIGN = TKS > TVS ? TKS : TVS;
    static constexpr int SMALL_BYTES = TKS + TVS + SMALL_ALIGN;  // incl. alignment slack
    static constexpr int STATE_F4 = NH * NMT;                    // float4 items per lane
    static constexpr bool H8 = NH == 2;       // eight heads in the N dimension (see the fragment maps)
    static constexpr int HL = H8 ? 2 : 1;     // heads whose softmax state a lane keeps: HL * tg + {0 ..}
    static constexpr int NPB = H8 ? 1 : 2;    // P.V steps per page
    // Lane (g, tg) reads slice g of page tokens 4tg .. 4tg + 3, one row per instruction.  Rows of whole
    // power-of-two sizes put the quad's four rows (4 rows apart) on the same banks: each lane then
    // starts at another of its four tokens.  24- and 48-byte rows (3 bits, head_dim 64 / 128) are
    // apart as they are -- rotated they collide (20 extra wavefronts per page at head_dim 64).
    static constexpr bool ROT = !(BV == 3 && D <= 128);
    // per-warp ring of stages filled by bulk copies (TMA), one mbarrier per stage; a stage holds the
    // NP consecutive pages a warp works on at a time
    static constexpr int RING = 2;
    // tables, queries, the folded piece, prefix sums, mbarriers, ring addresses
    static constexpr int MISC_BYTES = SMALL_BYTES + 8 * (D + 16) * 4 + 4 * NH * (D + 4) * 4 +
                                      (kFlowMaxSeqs + 4) * 4 + 16 * RING * 8 + 16 * 4 + 64;
    // a warp's share of the merge exchange area: its (O, m, l)
    static constexpr int XSLOT = 32 * STATE_F4 * 16, XML = NH * 2 * 4 * 4;
    // Objects are placed first-fit before / after the 64 KB-aligned table window: the misc block, the
    // exchange area where it has its own space (`sep`: the first pages of the NEXT item can then
    // already be copied into the rings while the merge runs; else a warp's share lies in its ring,
    // which is idle during the merge), and every warp's ring.  Bytes needed from `base`.
    __host__ __device__ static constexpr int ring_bytes(int np, bool sep) {
        const int ring = RING * np * PAGE_BYTES;
        return ((sep || ring > XSLOT ? ring : XSLOT) + 127) / 128 * 128;
    }
    __host__ __device__ static constexpr int plan(int warps, int np, bool sep, int base) {
        int free0 = base, end0 = base, free1 = base;
        if (BYTE) {
            end0 = (base + 65535) / 65536 * 65536;
            free1 = end0 + 65536;
        }
        const int n = warps + (sep ? 2 : 1);
        for (int i = 0; i < n; i++) {
            const int bytes = i == 0 ? MISC_BYTES + warps * XML : (sep && i == 1) ? warps * XSLOT : ring_bytes(np, sep);
            const int a0 = (free0 + 127) / 128 * 128;
            if (a0 + bytes <= end0) free0 = a0 + bytes;
            else free1 = (free1 + 127) / 128 * 128 + bytes;
        }
        return (free1 > free0 ? free1 : free0) - base;
    }
    __host__ __device__ static constexpr int need(int warps, int np, bool sep) {
        int worst = 0;
        const int bases[5] = {0, 16, 1024, 2048, 4096};
        for (int i = 0; i < 5; i++) {
            const int n = plan(warps, np, sep, bases[i]);
            worst = n > worst ? n : worst;
        }
        return worst + 128;
    }
    static constexpr int CTAS_PER_SM = BYTE ? 1 : 2;
    static constexpr int LIMIT = BYTE ? 227 * 1024 : 227 * 1024 / CTAS_PER_SM - 1024;
    // head_dim 256 keeps the query fragments in shared memory (one 8-byte load per k-block and
    // stage) instead of 32 registers, which lets it run 16 warps per SM like head_dim 128
    // wherever 16 page rings fit next to the byte table
    static constexpr int WARPS = (BYTE && D <= 128 && need(16, 1, false) <= LIMIT) ? 16 : 8;
    // two pages per stage wherever their rings leave the warp count alone
    static constexpr int NP = need(WARPS, 2, false) <= LIMIT ? 2 : 1;
    static constexpr int STAGE_BYTES = NP * PAGE_BYTES;
    // (an 8-warp CTA that owns its SM has 255 registers per thread and keeps them in registers)
    static constexpr bool QSMEM = D == 256 && !(BYTE && WARPS == 8);
    static constexpr int THREADS = 32 * WARPS;
    static constexpr bool SEP = need(WARPS, NP, true) <= LIMIT;
    static constexpr int SMEM_BYTES = need(WARPS, NP, SEP);
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
