// Paged decode attention on the tensor cores: every CTA owns an equal share of the batch's pages.
//
// Arithmetic, tables, page layout and fragment maps: ftq_attn_mma.cuh (the fused formulation of
// src/fused_turboquant/kernels/triton_flash_decode.py:33-324 of the reference, with the query
// rotation of hf/fused_cache.py:579-581 and the page-table walk of vllm_plugin/cache_ops.py:151-205
// folded in).  This file: how the work is split and put together again.
//
// One CTA per SM holds the dequantisation tables; its threads are two halves, each of which walks a share of the work
// on its own (own queries, page rings, barriers): while one half folds, merges or waits for a piece's first pages, the
// other one computes.  "CTA" below means such a half.
//
// The (layer, sequence, KV head) units lie in one line of places, unit after unit, a place for each page and PIECE more
// for each unit, and CTA c of the persistent grid takes places [c * share, (c + 1) * share): all CTAs have the same amount
// of work whatever the lengths of the sequences are, and a unit is cut only where a share ends.  PIECE is what a piece
// costs on its own (rotate the queries, fold the warps' states, the first pages' latency).  Without it the CTAs whose
// shares held many short sequences were the last by far: 40 sequences log-uniform up to 4000 tokens, 32 / 8 heads of 128,
// K3V3, 59 -> 25 us; 100 up to 1000, 64 / 8 heads, K4V4, 85 -> 33.  (20 to 40 places measure alike, 8 and 60 up to half as
// much again.)  Batches of short units are not cut at all (WHOLE below).  The partition needs the prefix sums of the
// places, which every CTA computes from seq_lens at its start.
// This kernel took the place of one that streamed pages across work items without CTA-wide barriers, tickets handing
// out the items.  In turn on one device, us there and here: 64 x 8192 tokens of 32 / 8 heads of 128, K4V4, 140 and 135
// (runs of one side differ by 3 %), 24 sequences log-uniform up to 30000 tokens 64 and 35, 4 x 131072, 64 / 8 heads, K3V3,
// 159 and 139, the ragged batch of 256 up to 32768, 16 / 8 heads of 256, K4V2, 877 and 781.
//
// A piece is walked by the CTA's warps in stages of NP consecutive pages, dealt round-robin.  A
// warp keeps RING stages in flight (1-D bulk copies, TMA); block ids are read straight from the
// block table, a batch of 32 per warp, one batch ahead.  The first stages of the next piece are
// requested before this piece's states are folded.
//
// Pieces of a cut unit leave (O, m, l) rows in the workspace (two row blocks per half: a share's first
// and last piece can be parts of units).  When its share is done a half counts them in; whoever arrives last
// merges the rows, rotates back (core/hadamard.py:93-100) and stores.  A unit that one piece covers is
// finished from shared memory.  Nobody waits for anybody.  The counters are cleared by CTA 0 under
// the launch's epoch, as described at AttnParams.
//
// CLUSTER: few units with short contexts.  A cluster of CTAs has one unit, each half a part of its pages; the parts' (O,
// m, l) stay in shared memory, and after a cluster barrier a warp per head merges them from there.
//
// Every wait is bounded and run by whole warps (mbar_wait, the epoch); one that runs out turns the rows of the units that it
// was for into NaN and sets a bit of the status word.  Block ids outside [0, num_blocks) are never dereferenced.
#pragma once

#include "ftq_attn_mma.cuh"

namespace ftq {

#ifdef FTQ_TEST_WAIT_EXPIRY
constexpr int kEpochSpinLimit = 1 << 8;
// Set by a test of the give-up path: CTA 0 does not publish its epoch (and every page copy is issued).
__device__ int test_withhold_epoch = 0;
#else
constexpr int kEpochSpinLimit = 1 << 22;
#endif

// A piece of a CTA's share: pages [page0, page0 + n_pages) of one unit (n_pages = 0: none left).
struct FlowPiece {
    int64_t unit_start;   // first place of the unit on the line of all places
    int64_t next;         // where the next piece starts
    int unit_pages, layer, b, hkv, page0, n_pages, tokens;
    bool first;           // the share starts with it
};

// A half's share: places [first, end) of the line; all shares but the last have `share` places.
struct FlowShare {
    int64_t first, end, share;
    bool whole;           // units are not cut (see FlowCfg::WHOLE): a half has those that start in its share
};

template <int D, int BK, int BV, int NH, bool CLUSTER = false>
struct FlowCfg : MmaCfg<D, BK, BV, NH> {
    using M = MmaCfg<D, BK, BV, NH>;
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
    // what a half (see attn_flow_kernel) has of its own: the queries; the folded piece, the warps' (m, l), mbarriers,
    // ring addresses
    static constexpr int QS_BYTES = 4 * NH * (D + 16) * 4;
    __host__ __device__ static constexpr int misc_bytes(int warps) {
        return 4 * NH * (D + 4) * 4 + warps * XML + warps * RING * 8 + warps * 4 + 64;
    }
    // a warp's share of the merge exchange area: its (O, m, l)
    static constexpr int XSLOT = 32 * M::STATE_F4 * 16, XML = NH * 2 * 4 * 4;
    static constexpr int PREFIX_BYTES = (kFlowMaxSeqs + 4) * 4;
    // Objects are placed first-fit before / after the 64 KB-aligned table window, large ones first: every warp's ring, the
    // exchange areas where they have their own space (`sep`: the first pages of the NEXT item can then
    // already be copied into the rings while the merge runs; else a warp's share lies in its ring,
    // which is idle during the merge), the queries, the misc blocks, the prefix sums.  Bytes needed from `base`.
    __host__ __device__ static constexpr int ring_bytes(int np, bool sep) {
        const int ring = RING * np * M::PAGE_BYTES;
        return ((sep || ring > XSLOT ? ring : XSLOT) + 127) / 128 * 128;
    }
    __host__ __device__ static constexpr int plan(int halves, int warps, int np, bool sep, int base) {
        int free0 = base, free1 = (base + 65535) / 65536 * 65536;
        const int end0 = free1;
        free1 += 65536;
        const int n = halves * (warps + 3) + 1;
        for (int i = 0; i < n; i++) {
            const int k = i - halves * warps;
            const int bytes = k < 0 ? ring_bytes(np, sep) : k < halves ? (sep ? warps * XSLOT : 0) : k < 2 * halves ? QS_BYTES
                              : k < 3 * halves ? misc_bytes(warps) : PREFIX_BYTES;
            const int a0 = (free0 + 127) / 128 * 128;
            if (a0 + bytes <= end0) free0 = a0 + bytes;
            else free1 = (free1 + 127) / 128 * 128 + bytes;
        }
        return (free1 > free0 ? free1 : free0) - base;
    }
    __host__ __device__ static constexpr int need(int halves, int warps, int np, bool sep) {
        // (wherever the dynamic part starts in the first 4 KB: all bases with the same next 128-byte boundary place alike, and
        // the first of them needs the most)
        int worst = plan(halves, warps, np, sep, 0);
        for (int base = 16; base <= 4096; base += 128) {
            const int n = plan(halves, warps, np, sep, base);
            worst = n > worst ? n : worst;
        }
        return worst;
    }
    static constexpr int LIMIT = 226 * 1024;   // (1 KB for the kernel's static shared memory)
    // A CTA per SM, as two halves that share the tables and nothing else: one half's barriers and folds overlap with the
    // other's pages.  Warps of a half: 8 of 128 registers where 3-bit codes or 2-bit keys keep the ALU pipe busy, 6 of 168
    // otherwise (64 x 8192 tokens, two layers of 32 / 8 heads of 128, K4V4: 258 us with 8, 238 with 6; 4 x 131072, 64 / 8
    // heads, K3V3: 134 with 8, 138 with 6); heads of 256: 6 (ragged K4V2 batch of 256 up to 32768 tokens: 802 with 8, 739
    // with 6), in groups of five to eight 4 of 255.  A cluster's CTA at head_dim 256 is one half.
    static constexpr int HALVES = D == 256 && CLUSTER ? 1 : 2;
    static constexpr int WARPS = CLUSTER ? (D == 256 && NH == 1 ? 12 : 8) : D == 256 ? (NH == 1 ? 6 : 4) : BK == 4 && BV != 3 ? 6 : 8;
    // places of the line that a unit takes beyond one for each page (see above)
    static constexpr int PIECE = 28;
    // Where the longest unit has no more pages than this, none is cut: it belongs to the half in whose share it starts.  A
    // half walks them in less time than the merge of a cut unit takes (200 sequences of up to 400 tokens, 32 / 8 heads of
    // 128, K4V4: 31.5 -> 30.1 us; 60 of 300 17.7 -> 15.8; 224 units of 118 11.2 -> 9.5).  At 48 pages 300 units of 600 tokens, a few
    // more than there are halves, take 20.3 us in place of 19.2; heads of 256 at 32 pages 344 of 468 30.0 in place of 27.8.
    static constexpr int WHOLE = D == 256 ? 24 : 32;
    // two pages per stage wherever their rings leave the warp count alone (a cluster's parts are a few pages long)
    static constexpr int NP = !CLUSTER && need(HALVES, WARPS, 2, false) <= LIMIT ? 2 : 1;
    static constexpr int STAGE_BYTES = NP * M::PAGE_BYTES;
    static constexpr int THREADS = 32 * WARPS;
    static constexpr bool SEP = need(HALVES, WARPS, NP, true) <= LIMIT;
    static constexpr int SMEM_BYTES = need(HALVES, WARPS, NP, SEP);
    // the codes' look-ups: keys in column 0 of the window, values in column 1, or both in the same tables
    template <bool SHARED>
    using WinK = Window<BK, SHARED && BK == 3>;
    template <bool SHARED>
    using WinV = Window<BV, SHARED && BV == 3>;
};

__device__ __forceinline__ uint32_t atom_add_acq_rel(int* p, int v) {
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;\n" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ float2 ld_cluster2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

template <int D, int BK, int BV, bool SHARED_LUT, int NH, bool CLUSTER>
__global__ void __launch_bounds__(FlowCfg<D, BK, BV, NH, CLUSTER>::HALVES * FlowCfg<D, BK, BV, NH, CLUSTER>::THREADS, 1)
attn_flow_kernel(const __grid_constant__ AttnParams p) {
    using C = FlowCfg<D, BK, BV, NH, CLUSTER>;
    using WK = typename C::template WinK<SHARED_LUT>;
    using WV = typename C::template WinV<SHARED_LUT>;
    constexpr int NKB = C::NKB, NMT = C::NMT, WARPS = C::WARPS, THREADS = C::THREADS, NP = C::NP;
    constexpr int E = D / kOctet;
    constexpr int ROW = D + 4;
    constexpr int IDS = 32 / NP;   // stages per batch of block ids

    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
    // ---- carve shared memory (addresses in the shared window): the tables need a
    // 64 KB-aligned window; the other objects go first-fit before or after it
    const uint32_t window = (sbase + 65535u) & ~65535u, end0 = window;
    uint32_t free0 = sbase, free1 = window + 65536u;
    auto take = [&](uint32_t bytes) {
        uint32_t a = (free0 + 127u) & ~127u;
        if (a + bytes <= end0) { free0 = a + bytes; return a; }
        a = (free1 + 127u) & ~127u;
        free1 = a + bytes;
        return a;
    };
    auto gptr = [&](uint32_t saddr) { return smem_raw + (saddr - sbase); };
    const int half = C::HALVES > 1 ? static_cast<int>(threadIdx.x) / THREADS : 0;
    uint32_t rings[WARPS], xarea = 0, qs_at = 0, misc_of[C::HALVES];
    auto take_mine = [&](uint32_t& mine, uint32_t bytes) {   // one for each half
#pragma unroll
        for (int h = 0; h < C::HALVES; h++) {
            const uint32_t a = take(bytes);
            if (h == half) mine = a;
        }
    };
#pragma unroll
    for (int w = 0; w < WARPS; w++) take_mine(rings[w], C::ring_bytes(NP, C::SEP));
    if constexpr (C::SEP) take_mine(xarea, WARPS * C::XSLOT);
    take_mine(qs_at, C::QS_BYTES);
#pragma unroll
    for (int h = 0; h < C::HALVES; h++) misc_of[h] = take(C::misc_bytes(WARPS));
    const uint32_t misc = half == 0 ? misc_of[0] : misc_of[C::HALVES - 1];
    int* prefix = reinterpret_cast<int*>(gptr(take(C::PREFIX_BYTES)));   // [B + 1] places, summed up
    float* qs = reinterpret_cast<float*>(gptr(qs_at));                // [4 * NH][D + 16] rotated queries
    float* folded = reinterpret_cast<float*>(gptr(misc));             // [4 * NH][ROW] the piece's (O, m, l)
    float* xml = folded + 4 * NH * ROW;                               // [WARPS][2][4 * NH]
    const uint32_t bars = misc + 4 * NH * ROW * 4 + WARPS * C::XML;   // [WARPS][RING] x 8 bytes
    uint32_t* ring_at = reinterpret_cast<uint32_t*>(gptr(bars + WARPS * C::RING * 8));  // [WARPS]
    const int tid = static_cast<int>(threadIdx.x) - half * THREADS;
    if (tid == 0) {
#pragma unroll
        for (int w = 0; w < WARPS; w++) ring_at[w] = rings[w];
    }
    // warp w's share of the merge exchange area
    auto xchg = [&](int w) {
        return reinterpret_cast<float4*>(gptr(C::SEP ? xarea + w * C::XSLOT : ring_at[w]));
    };
    // the half's barrier, and the cluster's.  (`bar.sync` and `.aligned` want whole warps to arrive together, and lanes that
    // have parted -- one of them asked for the epoch, some wrote rows -- need not have met again by themselves)
    auto sync_half = [&]() {
        if constexpr (C::HALVES == 1) {
            __syncthreads();
        } else {
            __syncwarp();
            asm volatile("bar.sync %0, %1;\n" ::"r"(1 + half), "n"(THREADS) : "memory");
        }
    };
    auto sync_cluster = [&]() {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    };

    // the next kernel of the stream may start its own set-up as soon as every CTA got here
    let_next_kernel_start();
    const int lane = tid & 31, warp = tid >> 5;
    // This half among all halves of the grid.  A cluster: its unit's part `cta` of `ctas`.
    int cta = half * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x), ctas = C::HALVES * static_cast<int>(gridDim.x);
    uint32_t rank = 0, cluster_size = 1;
    if constexpr (CLUSTER) {
        asm("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(cluster_size));
        cta = static_cast<int>(rank) * C::HALVES + half;
        ctas = static_cast<int>(cluster_size) * C::HALVES;
    }
    const int g = lane >> 2, tg = lane & 3;
    const bool odd = g & 1;
    const int group = p.Hq / p.Hkv;  // <= 4 * NH
    constexpr bool H8 = C::H8;
    constexpr int NO = C::STATE_F4;  // accumulator tiles per lane
    constexpr int HL = C::HL;
    // byte selectors (source 4 = a zero byte): a lane's own fp16 of a packed pair, and the
    // placement of a weight in the low (even g) or high (odd g) half of a B register
    uint32_t sel_own = odd ? 0x4432u : 0x4410u;
    uint32_t sel_plo = odd ? 0x1044u : 0x4410u;
    uint32_t sel_phi = odd ? 0x3244u : 0x4432u;
    // Lane constants of the page reads: byte offset of the key row rho(g) and of the norm quad;
    // per value register j the first word of slice g in the row of page token 4tg + ((j + tg) & 3)
    // (halves exchanged for tokens with bit 1 set).
    uint32_t koff = (4 * (g >> 1) + (g & 1)) * C::PDK + slice_word<C::KSB>(tg);
    const uint32_t ksh = slice_shift<C::KSB>(tg);
    uint32_t noff = C::OFF_KN + 8 * (g >> 1);
    uint32_t vrow[4];
    const uint32_t vsh = slice_shift<C::VSB>(g);   // (the same for the exchanged slice g ^ 4)
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int u = C::ROT ? (j + tg) & 3 : j;
        const int slice = g ^ ((u & 2) << 1);
        vrow[j] = C::OFF_VC + (4 * tg + u) * C::PDV + slice_word<C::VSB>(slice);
    }

    // ---- once per CTA: dequantisation tables.  A lane keeps one level of each codebook; a row (32
    // copies of an entry) is two shuffles, a conversion and one store.
    {
        const float lev_k = p.lk.v[lane & 15], lev_v = p.lv_scaled.v[lane & 15];
        auto pair = [&](float lev, int lo, int hi) {
            const __half2 h = __floats2half2_rn(__shfl_sync(0xffffffffu, lev, lo), __shfl_sync(0xffffffffu, lev, hi));
            return *reinterpret_cast<const uint32_t*>(&h);
        };
        uint32_t* tb = reinterpret_cast<uint32_t*>(gptr(window));
        auto entry = [&](float lev, int bits, int column, int e) {   // the lane's copy in row e
            if (bits == 4) return pair(lev, e & 15, e >> 4);
            if (bits == 3) return pair(lev, e >> (2 * column) & 7, e >> (2 * column + 3) & 7);
            const uint32_t x = pair(lev, e & 3, (e >> 2) & 3), y = pair(lev, (e >> 4) & 3, e >> 6);
            return (lane & 1) ? y : x;
        };
#pragma unroll 4
        for (int e = threadIdx.x / 32; e < 256; e += C::HALVES * WARPS) {
            tb[e * 64 + lane] = entry(lev_k, BK, 0, e);
            if constexpr (SHARED_LUT && BK == 3) tb[e * 64 + 32 + lane] = entry(lev_k, 3, 1, e);   // (by the high six bits)
            else if constexpr (!SHARED_LUT) tb[e * 64 + 32 + lane] = entry(lev_v, BV, 0, e);
        }
    }
    const uint32_t lk_lane = window | (BK == 2 ? (lane & 15) * 8 : lane * 4);
    const uint32_t lv_lane = window | (SHARED_LUT ? 0u : 128u) | (BV == 2 ? (lane & 15) * 8 : lane * 4);
    // one mbarrier per ring buffer (a single arrival + the copies' bytes)
    const uint32_t my_bars = bars + warp * C::RING * 8;
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < C::RING; r++) mbar_init(my_bars + r * 8, 1);
    }
    mbar_fence_init();
    __shared__ int s_bads[C::HALVES][3];   // by piece number mod 3: a block id of the piece was out of range
    int* s_bad = s_bads[half];
    if (tid < 3) s_bad[tid] = 0;

    // Everything up to here touched shared memory only.  From here on the kernel reads and writes
    // global memory that the kernel before it in the stream may still be using.
    after_previous_kernel();
    unsigned long long* epoch_word = reinterpret_cast<unsigned long long*>(p.work_counter + 2);
    if (blockIdx.x == 0) {
        if constexpr (!CLUSTER)
            for (int i = threadIdx.x; i < p.n_units; i += C::HALVES * THREADS) p.unit_counter[i] = 0;
        if (threadIdx.x == 0) {
            p.work_counter[1] = 0;
            if (p.b0 == 0) p.work_counter[kStatusWord] = 0;   // (the call's: its later launches add to it)
        }
    }
    // prefix sums of the places (lengths beyond the host's bound are cut to it)
    auto tokens_of = [&](int b) { return max(0, min(p.seq_lens[b], p.max_seq)); };
    if (!CLUSTER && threadIdx.x < 32) {
        int carry = 0, longest = 0;
        for (int b0 = 0; b0 < p.B; b0 += 128) {
            int x[4];      // (their loads do not wait for one another)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int b = b0 + 32 * k + lane;
                x[k] = b < p.B ? (tokens_of(b) + kPageTokens - 1) / kPageTokens : 0;
                longest = max(longest, x[k]);
                if (x[k] > 0) x[k] += C::PIECE;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x[k], d);
                    if (lane >= d) x[k] += y;
                }
                const int b = b0 + 32 * k + lane;
                if (b < p.B) prefix[b + 1] = carry + x[k];
                carry += __shfl_sync(0xffffffffu, x[k], 31);
            }
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        if (lane == 0) {
            prefix[0] = 0;
            prefix[kFlowMaxSeqs + 1] = longest;
        }
    }
    __syncthreads();
#ifdef FTQ_TEST_WAIT_EXPIRY
    const bool publish = test_withhold_epoch == 0;
#else
    constexpr bool publish = true;
#endif
    if (blockIdx.x == 0 && threadIdx.x == 0 && publish) {
        __threadfence();
        asm volatile("st.release.gpu.global.u64 [%0], %1;\n" ::"l"(epoch_word), "l"(p.epoch) : "memory");
    }
    bool stalled = false;   // a wait for a page ran out: no more waiting, the warp's results become NaN
    // The counters and the status word are valid once CTA 0 has published this launch's epoch (by the time anybody asks it
    // has normally been there for long).  Run by a whole warp: its lane 0 asks, and all its lanes learn what came of it.
    auto await_epoch = [&]() {
        bool seen = false;
        if (lane == 0)
            for (int i = 0; i < kEpochSpinLimit && !seen; i++) {
                unsigned long long v;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(epoch_word) : "memory");
                seen = v == p.epoch;
                if (!seen) __nanosleep(100);
            }
        return __any_sync(0xffffffffu, seen) != 0;
    };
    // a half with pieces asks once, by its first warp, before them
    __shared__ bool s_epochs_lost[C::HALVES];
    bool& s_epoch_lost = s_epochs_lost[half];

    // a CTA has left (run by one warp; `asked`: its half has)
    auto leave = [&](bool asked) {
        const bool lost = asked ? s_epoch_lost : !await_epoch();
        if (lane == 0 && lost) atomicOr(p.work_counter + kStatusWord, kStatusWaitExpired);
        if (lane == 0 && atomicAdd(p.work_counter + 1, 1) == static_cast<int>(gridDim.x) - 1) {
            __threadfence();
            asm volatile("st.release.gpu.global.u64 [%0], %1;\n" ::"l"(epoch_word), "l"(0ull) : "memory");
        }
    };

    // ---- this CTA's share of the pages, and the piece that starts at a given page
    // (in shared memory: two threads of a half use it between pieces, and the page loop needs the registers)
    __shared__ FlowShare s_shares[C::HALVES];
    FlowShare& mine = s_shares[half];
    if (!CLUSTER && tid == 0) {
        const int64_t total = static_cast<int64_t>(prefix[p.B] * p.Hkv) * p.n_layers;
        int64_t share = (total + ctas - 1) / ctas;
        const int longest = prefix[kFlowMaxSeqs + 1];
        // (the parts of a unit are walked side by side but merged by one half: the square root is where a few long units
        // balance the two.  One sequence of 131072 tokens, 4 / 1 heads of 128, K4V4, 38.6 -> 25.0 us, in 171 parts in place of
        // 293; two ragged ones of 37397, 14 / 2 heads 32.9 -> 22.5; half of it 29.7 and 27.7)
        constexpr int ROUND = WARPS * NP;      // (a stage of each warp: the share's pages take whole rounds)
        const int least = max(ROUND, static_cast<int>(0.8f * sqrtf(static_cast<float>(longest))) / ROUND * ROUND);
        share = share > least ? share : least;
        mine.whole = longest <= C::WHOLE;
        // all alike: as many to each, unless that is half as much again (400 units of 100 tokens on 296 halves 15.0 -> 13.9 us,
        // 302 of 8 12.4 and 13.4)
        const int each = (p.n_units + ctas - 1) / ctas;
        if (mine.whole && total == static_cast<int64_t>(longest + C::PIECE) * p.n_units &&
            (each == 1 || 2 * each * ctas <= 3 * p.n_units))
            share = static_cast<int64_t>(each) * (longest + C::PIECE);
        mine.share = share;
        mine.first = share * cta;
        mine.end = mine.first + share < total ? mine.first + share : total;
    }
    auto locate = [&](int64_t pos) {
        FlowPiece it{};
        it.next = pos;
        if constexpr (CLUSTER) {   // one piece: part `cta` of the cluster's unit
            if (pos != 0) return it;
            const int unit = static_cast<int>(blockIdx.x / cluster_size), per_lay = p.B * p.Hkv;
            it.layer = unit / per_lay;
            const int r = unit - it.layer * per_lay;
            it.b = r / p.Hkv;
            it.hkv = r - it.b * p.Hkv;
            const int tokens = tokens_of(it.b);
            it.unit_pages = (tokens + kPageTokens - 1) / kPageTokens;
            const int per = (it.unit_pages + ctas - 1) / ctas;
            it.page0 = cta * per;
            it.n_pages = max(0, min(per, it.unit_pages - it.page0));
            it.tokens = min(tokens - it.page0 * kPageTokens, it.n_pages * kPageTokens);
            it.next = 1;
            return it;
        }
        if (pos >= mine.end) return it;
        int r;
        if (p.n_layers == 1) {
            it.layer = 0;
            r = static_cast<int>(pos);
        } else {
            const int per_layer = prefix[p.B] * p.Hkv;
            it.layer = static_cast<int>(pos / per_layer);
            r = static_cast<int>(pos - static_cast<int64_t>(it.layer) * per_layer);
        }
        int lo = 0, hi = p.B;    // prefix[lo] * Hkv <= r < prefix[hi] * Hkv
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (prefix[mid] * p.Hkv <= r) lo = mid; else hi = mid;
        }
        it.b = lo;
        int places = prefix[lo + 1] - prefix[lo];
        r -= prefix[lo] * p.Hkv;
        it.hkv = r / places;
        int at = r - it.hkv * places;
        if (mine.whole && at > 0) {   // (a share that starts inside a unit: with the next one, if that is in it)
            pos += places - at;
            it.next = pos;
            if (pos >= mine.end) return it;
            at = 0;
            if (++it.hkv == p.Hkv) {
                it.hkv = 0;
                do {
                    if (++lo == p.B) { lo = 0; it.layer++; }
                    places = prefix[lo + 1] - prefix[lo];
                } while (places == 0);
                it.b = lo;
            }
        }
        it.unit_pages = places - C::PIECE;
        it.unit_start = pos - at;
        it.first = pos == mine.first;
        const int64_t room = mine.whole ? places : mine.end - pos;
        const int to = places - at > room ? at + static_cast<int>(room) : places;
        // (a share that ends among a unit's extra places has none of its pages: 0, and the share's end)
        it.page0 = max(at - C::PIECE, 0);
        it.n_pages = max(to - C::PIECE, 0) - it.page0;
        it.tokens = min(tokens_of(lo) - it.page0 * kPageTokens, it.n_pages * kPageTokens);
        it.next = pos + (to - at);
        return it;
    };
    // The pieces of the share, by number mod 3: this one, the next one and the one after are known (one
    // thread looks for them, between two barriers).
    __shared__ FlowPiece s_pieces[C::HALVES][3];
    FlowPiece* s_piece = s_pieces[half];
    if (tid == 0) s_piece[0] = locate(CLUSTER ? 0 : mine.first);
    sync_half();

    // ---- pages: block ids and bulk copies
    const uint32_t my_ring = ring_at[warp];
    const uint32_t blk_stride = static_cast<uint32_t>(p.Hkv) * C::PAGE_BYTES;
    const uint64_t page_policy = l2_evict_first_policy();   // (pages are read once per step)
    uint32_t phase = 0;   // bit r = parity the next wait on ring buffer r expects
    int ring_it = 0;      // stages this warp has taken from its ring so far (buffer = ring_it % RING)
#ifdef FTQ_TEST_WAIT_EXPIRY
    bool test_drop = blockIdx.x == 0 && half == 0 && warp == 5 && publish;
#endif
    // stages of a piece that are this warp's: warp, warp + WARPS, ...
    auto my_stages = [&](const FlowPiece& it) {
        const int n = (it.n_pages + NP - 1) / NP - warp;
        return n > 0 ? (n + WARPS - 1) / WARPS : 0;
    };
    // block ids of this warp's stages k0 .. k0 + IDS - 1: lane NP * j + i holds page i of stage k0 + j
    // (an id outside the pool is replaced by 0 and remembered)
    auto load_ids = [&](const FlowPiece& it, int k0, int slot) {
        const int pg = (warp + (k0 + lane / NP) * WARPS) * NP + lane % NP;
        int id = 0;
        if (pg < it.n_pages) {
            id = p.block_table[static_cast<int64_t>(it.b) * p.max_blocks + it.page0 + pg];
            if (static_cast<uint32_t>(id) >= static_cast<uint64_t>(p.num_blocks)) {
                id = 0;
                s_bad[slot] = 1;
            }
        }
        return id;
    };
    auto head_base = [&](const FlowPiece& it) {
        return p.pool + it.layer * p.pool_layer_stride + static_cast<int64_t>(it.hkv) * C::PAGE_BYTES;
    };
    // start the copies of the warp's stage k into ring buffer rb: lane i copies page i, lane 0
    // announces the bytes of all of them
    auto issue_stage = [&](const uint8_t* base, int ids, int n_pages, int k, int rb) {
        const int here = min(NP, n_pages - (warp + k * WARPS) * NP);
        const uint32_t id = __shfl_sync(0xffffffffu, ids, (k % IDS) * NP + lane % NP);
        if (lane == 0) mbar_expect_tx(my_bars + rb * 8, here * C::PAGE_BYTES);
        __syncwarp();
#ifdef FTQ_TEST_WAIT_EXPIRY
        if (test_drop) {   // (see kMbarSpinLimit)
            test_drop = false;
            if (lane == 0) return;
        }
#endif
        if (lane < here)
            bulk_g2s_hint(my_ring + rb * C::STAGE_BYTES + lane * C::PAGE_BYTES,
                          base + static_cast<uint64_t>(id) * blk_stride, C::PAGE_BYTES, my_bars + rb * 8,
                          page_policy);
    };

    // ---- queries: rotated, pre-scaled, in shared memory: head rows of D + 16 floats, each quarter of
    // a row padded by 4, so that the 16 distinct float4 a fragment load touches are 2-way at worst
    auto qs_index = [](int head, int coord) {
        return head * (D + 16) + (coord / (D / 4)) * (D / 4 + 4) + coord % (D / 4);
    };
    auto head_row = [&](const FlowPiece& it) {   // first query head of the piece, as a row of q and out
        return (static_cast<int64_t>(it.layer) * p.B_stride + p.b0 + it.b) * p.Hq + it.hkv * group;
    };
    // run by warps w0 and w0 + 1 (8 octets rotate the at most 8 heads)
    auto rotate_queries = [&](const FlowPiece& it, int w0) {
        if (warp < w0 || warp - w0 >= NH) return;
        const int t8 = lane & 7, o = lane >> 3;
        const int hh = (warp - w0) * 4 + o;
        const bool hv = hh < group;
        const uint8_t* src = static_cast<const uint8_t*>(p.q) + (head_row(it) + (hv ? hh : 0)) * (D * 2);
        float a[E];
#pragma unroll
        for (int i = 0; i < E / 8; i++) {
            float tmp[8];
            const uint8_t* at = src + 16 * (t8 + 8 * i);
            if (p.q_dtype == kBF16) load8<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(at), tmp);
            else load8<__half>(reinterpret_cast<const __half*>(at), tmp);
#pragma unroll
            for (int c = 0; c < 8; c++)
                a[8 * i + c] = __uint_as_float(
                    __float_as_uint(tmp[c]) ^ sign_mask(p.signs, load_coord(t8, 8 * i + c)));
        }
        octet_fwht<E>(a, lane);
#pragma unroll
        for (int k = 0; k < E; k++)
            qs[qs_index(hh, t8 + 8 * k)] = hv ? a[k] * p.rsqrt_d * (p.scale * kLog2e) : 0.f;
    };

    // ---- per-piece arithmetic state of a lane: query fragments, softmax state of heads
    // HL*tg + {0 .. HL-1}, O[head][(D/8)*g .. + D/8)
    uint32_t qb[NKB][2];
    float m_run[HL], l_run[HL], oacc[NO][4];

    // a lane's slices of the staged page at `page`
    auto read_keys = [&](uint32_t (&k)[2][C::KW], uint32_t page) {
        lds_slice<C::KSB>(page + koff, ksh, k[0]);
        lds_slice<C::KSB>(page + koff + 2 * C::PDK, ksh, k[1]);
    };
    auto read_values = [&](uint32_t (&v)[4][C::VW], uint32_t page) {
        // register j holds page token 4tg + ((j + tg) & 3) where ROT is set: the four lanes of a
        // quad then read rows of alternating parity in one instruction; the P.V k-slots of a lane may hold its tokens in any order as long as the weights
        // follow (see the rotation of the transposed weights below).  The pool stores a V row
        // with its two halves exchanged for tokens with bit 1 set, so that the four rows a quad
        // reads in one instruction fall into distinct bank groups.
#pragma unroll
        for (int j = 0; j < 4; j++) lds_slice<C::VSB>(page + vrow[j], vsh, v[j]);
    };

    // S = K.Q^T of NP pages (two accumulator chains each)
    auto qk_scores = [&](const uint32_t (&k)[C::NP][2][C::KW], float (&c)[C::NP][2][4]) {
        typename WK::template Run<C::KW> run[NP][2];
#pragma unroll
        for (int i = 0; i < NP; i++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
#pragma unroll
                for (int j = 0; j < C::KW; j++) run[i][r].w[j] = k[i][r][j];
                WK::shift(run[i][r]);
            }
#pragma unroll
        for (int kb = 0; kb < NKB; kb++) {
#pragma unroll
            for (int i = 0; i < NP; i++) {
                uint32_t a0, a1, a2, a3;
                WK::pairs(run[i][0], kb, lk_lane, a0, a2);
                WK::pairs(run[i][1], kb, lk_lane, a1, a3);
                // (the first MMA of each of the two accumulator chains starts from zero)
                if (kb < 2) mma_16816_z(c[i][kb & 1], a0, a1, a2, a3, qb[kb][0], qb[kb][1]);
                else mma_16816(c[i][kb & 1], a0, a1, a2, a3, qb[kb][0], qb[kb][1]);
            }
        }
    };

    // online softmax per head over the scores of NP pages (base-2 exponent domain: the queries
    // carry log2(e)); the weights p * vnorm are rounded to fp16 and transposed into the B
    // operand of P.V: pb[i][ks] = k-slots {2tg, 2tg+1} and {2tg+8, 2tg+9} of page i's MMA step ks
    // (one step of 16 tokens for NH = 2, two of 8 (token, parity) pairs for NH = 1).
    // FULL = all tokens of the pages are valid.
    auto softmax_update = [&](auto full_tag, const uint2 (&kn)[C::NP], const uint2 (&vn)[C::NP], int st, int tokens,
                              const float (&c)[C::NP][2][4], uint32_t (&pb)[C::NP][C::NPB][2]) {
        constexpr bool FULL = decltype(full_tag)::value;
        // columns 2tg, 2tg + 1: two heads (NH = 2) or one head twice
        float sa[C::NP][HL], sb[C::NP][HL];
        bool okA[C::NP], okB[C::NP];
        float mx[HL];
#pragma unroll
        for (int h = 0; h < HL; h++) mx[h] = -INFINITY;
#pragma unroll
        for (int i = 0; i < NP; i++) {
            if constexpr (!FULL) {
                const int ntok = tokens - (st * NP + i) * kPageTokens;
                const int tokA = 4 * (g >> 1) + (g & 1);  // rows g, g+8 of S: tokens tokA, tokA + 2
                okA[i] = tokA < ntok;
                okB[i] = tokA + 2 < ntok;
            }
            const float kna = half_bits_to_float(__byte_perm(kn[i].x, 0u, sel_own));
            const float knb = half_bits_to_float(__byte_perm(kn[i].y, 0u, sel_own));
#pragma unroll
            for (int h = 0; h < HL; h++) {
                sa[i][h] = (c[i][0][h] + c[i][1][h]) * kna;
                sb[i][h] = (c[i][0][2 + h] + c[i][1][2 + h]) * knb;
                if constexpr (!FULL) {
                    sa[i][h] = okA[i] ? sa[i][h] : -INFINITY;
                    sb[i][h] = okB[i] ? sb[i][h] : -INFINITY;
                }
                mx[h] = fmaxf(mx[h], fmaxf(sa[i][h], sb[i][h]));
            }
        }
        bool above = false;
#pragma unroll
        for (int h = 0; h < HL; h++) above |= mx[h] > m_run[h] + kLazyMaxSlack;
        // Lazy reference maximum: the cross-lane maximum and the rescale run only when a
        // score exceeds the reference by more than kLazyMaxSlack (always on the first
        // stage of an item, where it is -inf); weights stay below 2^kLazyMaxSlack.
        if (__any_sync(0xffffffffu, above)) {
            float corr[HL];
#pragma unroll
            for (int h = 0; h < HL; h++) {
                float m = mx[h];
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
                const float m_new = fmaxf(m_run[h], m);   // finite: the stage's token 0 is valid
                corr[h] = fast_exp2(m_run[h] - m_new);    // 1 if unchanged, 0 from -inf
                l_run[h] *= corr[h];
                m_run[h] = m_new;
            }
#pragma unroll
            for (int mt = 0; mt < NO; mt++)
#pragma unroll
                for (int i = 0; i < 4; i++) oacc[mt][i] *= corr[H8 ? (i & 1) : 0];
        }
#pragma unroll
        for (int i = 0; i < NP; i++) {
        float vna = half_bits_to_float(__byte_perm(vn[i].x, 0u, sel_own));
        float vnb = half_bits_to_float(__byte_perm(vn[i].y, 0u, sel_own));
        if constexpr (!FULL) {
            vna = okA[i] ? vna : 0.f;
            vnb = okB[i] ? vnb : 0.f;
        }
        float wa[HL], wb[HL];
#pragma unroll
        for (int h = 0; h < HL; h++) {
            const float pa = fast_exp2(sa[i][h] - m_run[h]);  // exp2(-inf) = 0 for masked tokens
            const float pbv = fast_exp2(sb[i][h] - m_run[h]);
            l_run[h] += pa + pbv;
            wa[h] = pa * vna;
            wb[h] = pbv * vnb;
        }
        uint32_t t0w, t1w;
        if constexpr (H8) {
            t0w = movmatrix_trans(f2h2_sat(wa[0], wa[1]));
            t1w = movmatrix_trans(f2h2_sat(wb[0], wb[1]));
        } else {
            // M[token row][column n], both columns of a head equal; transposed, lane (g, tg)
            // receives head g>>1, page tokens 4tg, 4tg+1 (first) and 4tg+2, 4tg+3 (second)
            t0w = movmatrix_trans(__byte_perm(f2h_sat(wa[0]), 0u, 0x1010u));
            t1w = movmatrix_trans(__byte_perm(f2h_sat(wb[0]), 0u, 0x1010u));
        }
        // rotate the four 16-bit weights by tg positions to match the V register order
        if constexpr (C::ROT) {
            if (tg & 2) { const uint32_t x = t0w; t0w = t1w; t1w = x; }
            const uint32_t sh = (tg & 1) * 16;
            const uint32_t lo = __funnelshift_r(t0w, t1w, sh);
            const uint32_t hi = __funnelshift_r(t1w, t0w, sh);
            t0w = lo;
            t1w = hi;
        }
        if constexpr (H8) {
            pb[i][0][0] = t0w;
            pb[i][0][1] = t1w;
        } else {
            // column n = (head, parity): an even g keeps the weight in the low half (parity 0
            // rows of the k index), an odd g in the high half; the other half is zero
            pb[i][0][0] = __byte_perm(t0w, 0u, sel_plo);
            pb[i][0][1] = __byte_perm(t0w, 0u, sel_phi);
            pb[i][1][0] = __byte_perm(t1w, 0u, sel_plo);
            pb[i][1][1] = __byte_perm(t1w, 0u, sel_phi);
        }
        }
    };

    auto pv_accum = [&](const uint32_t (&v)[4][C::VW], const uint32_t (&pb)[C::NPB][2]) {
        typename WV::template Run<C::VW> run[4];
        if constexpr (H8) {
            // O^T += V^T.P^T : rows = coordinates (D/8)g + 2f, + 1, k = tokens: the codes of two tokens merged
            // into pairs before the look-up (exchanging the looked-up values took a byte-permute per look-up)
            WV::merge(v[0], v[1], run[0], run[1]);
            WV::merge(v[2], v[3], run[2], run[3]);
#pragma unroll
            for (int j = 0; j < 4; j++) WV::shift(run[j]);
#pragma unroll
            for (int m2 = 0; m2 < NMT; m2++) {
                uint32_t x[4], y[4];
#pragma unroll
                for (int j = 0; j < 4; j++) WV::pairs(run[j], m2, lv_lane, x[j], y[j]);
                mma_16816(oacc[2 * m2], x[0], x[1], x[2], x[3], pb[0][0], pb[0][1]);
                mma_16816(oacc[2 * m2 + 1], y[0], y[1], y[2], y[3], pb[0][0], pb[0][1]);
            }
        } else {
            // rows = d-pairs (D/16)*g + 2*mt + {0,1}, k = (token, parity)
#pragma unroll
            for (int j = 0; j < 4; j++) {
#pragma unroll
                for (int i = 0; i < C::VW; i++) run[j].w[i] = v[j][i];
                WV::shift(run[j]);
            }
#pragma unroll
            for (int ks = 0; ks < 2; ks++)
#pragma unroll
                for (int mt = 0; mt < NMT; mt++) {
                    uint32_t a0, a1, a2, a3;
                    WV::pairs(run[2 * ks], mt, lv_lane, a0, a1);
                    WV::pairs(run[2 * ks + 1], mt, lv_lane, a2, a3);
                    mma_16816(oacc[mt], a0, a1, a2, a3, pb[ks][0], pb[ks][1]);
                }
        }
    };

    // warps that fold the per-warp states; when enough warps are left over they rotate the next
    // piece's queries at the same time
    constexpr int NRED = (NO <= WARPS - 2) ? NO : WARPS;
    // warps that finish a piece (four heads each): the last ones, which have the fewest stages
    constexpr int FIN0 = WARPS - NH;

    // Rows (O, m, l) [group][ROW] of a half's pieces that are parts of units: block 0 the piece its share starts with, 1 its
    // last one.
    auto row_of = [&](int64_t c, int block) { return p.partials + (2 * c + block) * group * ROW; };
    __shared__ FlowPiece s_cuts[C::HALVES][2];
    __shared__ int s_part[C::HALVES][2];      // parts of the unit when this half is the last of them, else 0
    FlowPiece* s_cut = s_cuts[half];
    int* s_parts = s_part[half];
    if (tid < 2) s_cut[tid].n_pages = 0;
    // a finished head's coordinates t + 8 k
    auto store_head = [&](const FlowPiece& it, int h, int t, const float (&a)[E]) {
        const int64_t at = (head_row(it) + h) * D;
#pragma unroll
        for (int k = 0; k < E; k++) {
            const float r = a[k] * p.rsqrt_d;
            const float s = __uint_as_float(__float_as_uint(r) ^ sign_mask(p.signs, t + 8 * k));
            const int64_t idx = at + t + 8 * k;
            if (p.out_dtype == kBF16) static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(s);
            else if (p.out_dtype == kF16) static_cast<__half*>(p.out)[idx] = __float2half_rn(s);
            else static_cast<float*>(p.out)[idx] = s;
        }
    };
    // Finish warp w's heads of a folded piece: normalise, rotate back and store when the piece is the whole unit; else
    // leave its rows in the workspace, for merge_units.
    auto finish_piece = [&](const FlowPiece& it, bool first_of_cta) {
        const int t = lane & 7, h = (warp - FIN0) * 4 + (lane >> 3);
        const bool valid = h < group;
        const float* row0 = folded + (valid ? h : 0) * ROW;
        float a[E];
#pragma unroll
        for (int i = 0; i < E / 8; i++) {
            const float4 u = *reinterpret_cast<const float4*>(row0 + 8 * (t + 8 * i));
            const float4 v = *(reinterpret_cast<const float4*>(row0 + 8 * (t + 8 * i)) + 1);
            a[8 * i] = u.x; a[8 * i + 1] = u.y; a[8 * i + 2] = u.z; a[8 * i + 3] = u.w;
            a[8 * i + 4] = v.x; a[8 * i + 5] = v.y; a[8 * i + 6] = v.z; a[8 * i + 7] = v.w;
        }
        const float m = row0[D], l = row0[D + 1];
        if (it.page0 != 0 || it.n_pages != it.unit_pages) {
            if (valid) {
                float* mine = row_of(cta, first_of_cta ? 0 : 1) + h * ROW;
#pragma unroll
                for (int i = 0; i < E / 8; i++) {
                    float4* dst = reinterpret_cast<float4*>(mine + 8 * (t + 8 * i));
                    __stcg(dst, make_float4(a[8 * i], a[8 * i + 1], a[8 * i + 2], a[8 * i + 3]));
                    __stcg(dst + 1, make_float4(a[8 * i + 4], a[8 * i + 5], a[8 * i + 6], a[8 * i + 7]));
                }
                if (t == 0) __stcg(reinterpret_cast<float2*>(mine + D), make_float2(m, l));
            }
            if (tid == FIN0 * 32) s_cut[first_of_cta ? 0 : 1] = it;
            return;
        }
        float inv = l > 0.f ? 1.f / l : 0.f;
        if (m != m) inv = __int_as_float(0x7fc00000);
#pragma unroll
        for (int r = 0; r < E; r++) a[r] *= inv;
        octet_fwht<E>(a, lane);
        if (valid) store_head(it, h, t, a);
    };

    // A head of a unit from its n parts' rows (O, m, l), by S = 1, 2 or 4 octets of a warp (sub = which of them), each of
    // which adds up parts sub, sub + S, ...: the order of the sums depends on n and S alone.  `row` gives the row of a
    // part, `load2` / `load4` read from it.  All lanes of the warp run it together, with S in common; a lane of an octet
    // without a head has n = 0.
    auto merge_head = [&](const FlowPiece& it, int h, int n, int S, int sub, auto row, auto load2, auto load4) {
        const int t = lane & 7;
        float M = -INFINITY, L = 0.f, a[E];
        bool nan = false;
#pragma unroll
        for (int r = 0; r < E; r++) a[r] = 0.f;
        // AHEAD rows of an octet at a time; the first ones are on their way while the maximum is looked for
        constexpr int AHEAD = D == 256 && NH == 1 ? 2 : 4;      // (as many as the registers hold)
        float4 x[AHEAD][E / 4];
        float2 ml[AHEAD];
        auto load = [&](int i0) {
#pragma unroll
            for (int u = 0; u < AHEAD; u++) {
                const int i = i0 + u * S;
                ml[u] = make_float2(-INFINITY, 0.f);
                if (i < n) {
                    const auto r = row(i);
                    ml[u] = load2(r, D);
#pragma unroll
                    for (int c = 0; c < E / 4; c++) x[u][c] = load4(r, 8 * (t + 8 * (c / 2)) + 4 * (c & 1));
                }
            }
        };
        load(sub);
        for (int i = sub * kOctet + t; i < n; i += 4 * S * kOctet) {
            float m[4];
#pragma unroll
            for (int u = 0; u < 4; u++) m[u] = i + u * S * kOctet < n ? load2(row(i + u * S * kOctet), D).x : -INFINITY;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                nan |= m[u] != m[u];   // (fmaxf drops a NaN operand)
                M = fmaxf(M, m[u]);
            }
        }
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, M, s);
            const bool no = __shfl_xor_sync(0xffffffffu, static_cast<int>(nan), s) != 0;
            if (s < kOctet * S) {
                M = fmaxf(M, mo);
                nan |= no;
            }
        }
        for (int i0 = sub;;) {
#pragma unroll
            for (int u = 0; u < AHEAD; u++) {
                if (ml[u].x == -INFINITY) continue;   // (none, or a part without pages: its O is not written)
                const float f = fast_exp2(ml[u].x - M);
                L = fmaf(ml[u].y, f, L);
#pragma unroll
                for (int c = 0; c < E / 4; c++) {
                    a[4 * c] = fmaf(x[u][c].x, f, a[4 * c]);
                    a[4 * c + 1] = fmaf(x[u][c].y, f, a[4 * c + 1]);
                    a[4 * c + 2] = fmaf(x[u][c].z, f, a[4 * c + 2]);
                    a[4 * c + 3] = fmaf(x[u][c].w, f, a[4 * c + 3]);
                }
            }
            i0 += AHEAD * S;
            if (i0 >= n) break;
            load(i0);
        }
        __syncwarp();
        for (int s = kOctet; s < kOctet * S; s <<= 1) {
            L += __shfl_xor_sync(0xffffffffu, L, s);
#pragma unroll
            for (int r = 0; r < E; r++) a[r] += __shfl_xor_sync(0xffffffffu, a[r], s);
        }
        float inv = L > 0.f ? 1.f / L : 0.f;   // (a sequence without tokens: zero)
        if (nan) inv = __int_as_float(0x7fc00000);
#pragma unroll
        for (int r = 0; r < E; r++) a[r] *= inv;
        octet_fwht<E>(a, lane);
        if (sub == 0 && h < group) store_head(it, h, t, a);
    };

    // The cut units of this share (its first and its last piece), once all its pieces are done: whoever is the last to get
    // here with a unit puts it together, all heads at the same time.  Under load a dependent access to L2 takes 1 to 2 us,
    // so the chain is kept short: rows -> counter (2.4 us) -> rows and maxima together (2.4 us, 6 with a head per warp and
    // the maxima first).  In the loop, by the warps that finish pieces, it held up the half's other warps.
    auto merge_units = [&]() {
        if (tid < 2) {
            const FlowPiece& it = s_cut[tid];
            int n = 0;
            const int64_t share = mine.share;
            if (it.n_pages > 0 && s_epoch_lost) {
                n = -1;   // (not counted: nobody else becomes the last one)
            } else if (it.n_pages > 0) {
                // (release: the rows that the half wrote before the barrier; acquire: those of the others)
                const uint32_t old = atom_add_acq_rel(p.unit_counter + (static_cast<int64_t>(it.layer) * p.B + it.b) * p.Hkv + it.hkv, 1);
                const int parts = static_cast<int>((it.unit_start + C::PIECE + it.unit_pages - 1) / share - (it.unit_start + C::PIECE) / share) + 1;
                if (static_cast<int>(old) == parts - 1) n = parts;
            }
            s_parts[tid] = n;
        }
        sync_half();
#pragma unroll 1
        for (int cut = 0; cut < 2; cut++) {
            if (s_parts[cut] >= 0) continue;
            const int64_t at = head_row(s_cut[cut]) * D;
#pragma unroll 1
            for (int i = tid; i < group * D; i += THREADS) {
                if (p.out_dtype == kF32) static_cast<float*>(p.out)[at + i] = __int_as_float(0x7fc00000);
                else static_cast<uint16_t*>(p.out)[at + i] = 0x7fff;   // (a NaN in fp16 and in bf16)
            }
        }
        // Octets a head: from the number of parts alone, not from whether this half has one unit to merge or both, so that who
        // merges does not change the order of the sums.  Units of few parts together, all heads of both at the same time;
        // one of many (few long sequences) by itself, its rows over all octets.
        constexpr int FEW = 8;
        auto octets = [&](int heads) { return 4 * heads <= 4 * WARPS ? 4 : 2 * heads <= 4 * WARPS ? 2 : 1; };
        int n0 = max(s_parts[0], 0), n1 = max(s_parts[1], 0);
        while (n0 + n1 > 0) {
            const int a0 = n0, a1 = n0 > 0 && max(n0, n1) > FEW ? 0 : n1;
            const int S = octets(max(a0, a1) > FEW ? group : 2 * group);
            const int heads0 = a0 ? group : 0, heads = heads0 + (a1 ? group : 0);
            const int octet = warp * 4 + (lane >> 3), k = octet / S;
            const bool second = k >= heads0;
            const FlowPiece& it = s_cut[second];
            const int h = k >= heads ? group : second ? k - heads0 : k;
            const int64_t share = mine.share, c0 = (it.unit_start + C::PIECE) / share;
            merge_head(it, h, k >= heads ? 0 : second ? a1 : a0, S, octet % S,
                       [&](int i) { return row_of(c0 + i, (c0 + i) * share >= it.unit_start ? 0 : 1) + h * ROW; },
                       // (ordinary loads, behind the acquire and the barrier: a lane's two halves of 32 bytes are one sector, which
                       // L1 keeps from one to the other.  2 x 50554 tokens, 16 / 2 heads of 128, K3V4: 39.5 -> 30.7 us)
                       [](const float* r, int at) { return *reinterpret_cast<const float2*>(r + at); },
                       [](const float* r, int at) { return *reinterpret_cast<const float4*>(r + at); });
            n0 = 0;
            n1 -= a1;
        }
    };

    // sequences without tokens: no CTA meets their units, their outputs are zero (softmax over nothing)
    for (int i = CLUSTER ? p.n_layers * p.B : cta; i < p.n_layers * p.B; i += ctas) {
        const int layer = i / p.B, b = i - layer * p.B;
        if (prefix[b + 1] != prefix[b]) continue;
        const int per_seq = p.Hq * D;
        const int64_t at = (static_cast<int64_t>(layer) * p.B_stride + p.b0 + b) * per_seq;
        for (int d = tid; d < per_seq; d += THREADS) {
            if (p.out_dtype == kF32) static_cast<float*>(p.out)[at + d] = 0.f;
            else static_cast<uint16_t*>(p.out)[at + d] = 0;   // (fp16 and bf16 zero)
        }
    }

    // ---- the pieces of this CTA's share
    int slot = 0;                // piece number mod 3
    int ids = 0, ids_next = 0;   // block ids: the batch the next request takes, and the one after
    bool primed = false;         // the first RING stages of the current piece were requested early
    bool any = false, prev_first = true;   // a folded piece is waiting; it was the CTA's first
    if (s_piece[0].n_pages > 0) {
        ids = load_ids(s_piece[0], 0, 0);
        const int n = my_stages(s_piece[0]);
#pragma unroll
        for (int r = 0; r < C::RING; r++)
            if (r < n) issue_stage(head_base(s_piece[0]), ids, s_piece[0].n_pages, r, r);
        primed = true;
        rotate_queries(s_piece[0], FIN0);
        if (tid == 0) s_piece[1] = locate(s_piece[0].next);
        if (!CLUSTER && warp == 0) {   // (while the first pages are on their way)
            const bool seen = await_epoch();
            if (lane == 0) s_epoch_lost = !seen;
        }
    }
    while (s_piece[slot].n_pages > 0) {
        const FlowPiece& cur = s_piece[slot];
        const int slot1 = slot == 2 ? 0 : slot + 1, slot2 = slot == 0 ? 2 : slot - 1;   // next, after next
        const int n_pages = cur.n_pages, tokens = cur.tokens;
        const int n_mine = my_stages(cur);
        const uint8_t* base = head_base(cur);
        ids_next = load_ids(cur, IDS, slot);
        sync_half();         // C: queries, the next piece visible; `folded` holds the piece before
        int ids_piece = 0;       // first batch of the next piece
        if (s_piece[slot1].n_pages > 0) ids_piece = load_ids(s_piece[slot1], 0, slot1);
        // (a warp whose wait has run out requests nothing any more: the mbarrier of the lost copy
        // never completes its phase, and arriving on it again would be an error)
        if (!primed && !stalled) {
            // (when the exchange area aliases the ring, the fold used it with ordinary accesses)
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
#pragma unroll
            for (int r = 0; r < C::RING; r++)
                if (r < n_mine) issue_stage(base, ids, n_pages, r, (ring_it + r) % C::RING);
        }

        // Q^T fragments: column n = g is head g >> 1 (NH = 1) or g (NH = 2); k-block kb covers
        // coordinates (D/4)*tg + 4*kb + {0,1} (b0) and + {2,3} (b1)
#pragma unroll
        for (int kb = 0; kb < NKB; kb++) {
            const float4 q4 = *reinterpret_cast<const float4*>(
                qs + qs_index(H8 ? g : g >> 1, (D / 4) * tg + 4 * kb));
            const __half2 lo = __floats2half2_rn(q4.x, q4.y);
            const __half2 hi = __floats2half2_rn(q4.z, q4.w);
            qb[kb][0] = *reinterpret_cast<const uint32_t*>(&lo);
            qb[kb][1] = *reinterpret_cast<const uint32_t*>(&hi);
        }
        if (any && warp >= FIN0) finish_piece(s_piece[slot2], prev_first);

#pragma unroll
        for (int i = 0; i < HL; i++) { m_run[i] = -INFINITY; l_run[i] = 0.f; }
#pragma unroll
        for (int mt = 0; mt < NO; mt++)
#pragma unroll
            for (int i = 0; i < 4; i++) oacc[mt][i] = 0.f;

        // ---- the warp's stages.  NP pages at a time share the wait, the hand-over of the buffer, the
        // query fragments and the look at the reference maximum, and their chains of look-ups and
        // MMAs overlap.
        for (int k = 0; k < n_mine; k++) {
            const int rb = ring_it % C::RING;
            ring_it++;
            // (every lane polls; the vote brings them together again for the MMAs and makes one answer of theirs)
            if (!stalled) stalled = !__all_sync(0xffffffffu, mbar_wait(my_bars + rb * 8, (phase >> rb) & 1u));
            phase ^= 1u << rb;
            const uint32_t page = my_ring + rb * C::STAGE_BYTES;
            uint32_t kw[C::NP][2][C::KW], v[4][C::VW], pb[C::NP][C::NPB][2];
            uint2 kn[C::NP], vn[C::NP];
            float c[C::NP][2][4];
#pragma unroll
            for (int i = 0; i < NP; i++) {
                read_keys(kw[i], page + i * C::PAGE_BYTES);
                kn[i] = lds64(page + i * C::PAGE_BYTES + noff);
                vn[i] = lds64(page + i * C::PAGE_BYTES + noff + (C::OFF_VN - C::OFF_KN));
            }
            qk_scores(kw, c);
            // all stages but possibly the piece's last one are full (warp-uniform branch)
            const int st = warp + k * WARPS;
            if ((st + 1) * NP * kPageTokens <= tokens) softmax_update(std::true_type{}, kn, vn, st, tokens, c, pb);
            else softmax_update(std::false_type{}, kn, vn, st, tokens, c, pb);
#pragma unroll
            for (int i = 0; i < NP; i++) {
                read_values(v, page + i * C::PAGE_BYTES);
                pv_accum(v, pb[i]);
            }
            __syncwarp();  // every lane has its slices: the buffer may be refilled
            const int req = k + C::RING;
            if (req < n_mine && !stalled) {
                if (req % IDS == 0) {
                    ids = ids_next;
                    ids_next = load_ids(cur, req + IDS, slot);
                }
                issue_stage(base, ids, n_pages, req, rb);
            }
        }

        // ---- this warp's ring is drained: request the first stages of the next piece now, so that
        // they arrive while this one is folded (when the fold has its own exchange area)
        ids = ids_piece;
        primed = false;
        if constexpr (C::SEP) {
            const FlowPiece& nx = s_piece[slot1];
            if (nx.n_pages > 0) {
                primed = true;
                const int n = my_stages(nx);
                if (!stalled) {
#pragma unroll
                    for (int r = 0; r < C::RING; r++)
                        if (r < n) issue_stage(head_base(nx), ids, nx.n_pages, r, (ring_it + r) % C::RING);
                }
            }
        }

        // ---- fold the warps' states: every warp publishes (m, l, O), NRED warps reduce
#pragma unroll
        for (int i = 0; i < HL; i++) {
            l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 4);
            l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 8);
            l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 16);
        }
        // A warp whose copy never arrived poisons its state (NaN propagates to the output), and so does a score that is not
        // a number: it is in the sum of the weights, but no maximum knows it, and a warp without any other looks empty.
#pragma unroll
        for (int i = 0; i < HL; i++)
            if (stalled || l_run[i] != l_run[i]) m_run[i] = __int_as_float(0x7fc00000);
        sync_half();  // A: every warp is done with the ring, the queries and `folded`
#pragma unroll
        for (int mt = 0; mt < NO; mt++)
            // (the factor that undoes the scaling of the value centroids is applied once per piece)
            xchg(warp)[mt * 32 + lane] =
                make_float4(oacc[mt][0] * p.inv_v_scale, oacc[mt][1] * p.inv_v_scale,
                            oacc[mt][2] * p.inv_v_scale, oacc[mt][3] * p.inv_v_scale);
        if (g == 0) {
#pragma unroll
            for (int i = 0; i < HL; i++) {
                xml[(warp * 2 + 0) * (4 * NH) + HL * tg + i] = m_run[i];
                xml[(warp * 2 + 1) * (4 * NH) + HL * tg + i] = l_run[i];
            }
        }
        sync_half();  // B: all states are published
        if (warp < NRED) {
            const bool bad = s_bad[slot] != 0;
            for (int j = tid; j < NO * 32; j += NRED * 32) {
                const int ln = j & 31, mt = j >> 5;
                const int tg_ = ln & 3, g_ = ln >> 2;
                float M[HL], l[HL];
                bool nan[HL];
#pragma unroll
                for (int i = 0; i < HL; i++) {
                    M[i] = -INFINITY;
                    l[i] = 0.f;
                    nan[i] = bad;
#pragma unroll
                    for (int w2 = 0; w2 < WARPS; w2++) {
                        const float mw = xml[(w2 * 2 + 0) * (4 * NH) + HL * tg_ + i];
                        nan[i] |= mw != mw;   // (fmaxf drops a NaN operand)
                        M[i] = fmaxf(M[i], mw);
                    }
                }
                float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int w2 = 0; w2 < WARPS; w2++) {
                    float f[HL];
                    bool some = false;
#pragma unroll
                    for (int i = 0; i < HL; i++) {
                        const float mw = xml[(w2 * 2 + 0) * (4 * NH) + HL * tg_ + i];
                        const bool has = mw != -INFINITY;  // (NaN compares unequal: poison goes through)
                        f[i] = has ? fast_exp2(mw - M[i]) : 0.f;
                        some |= has;
                        l[i] = fmaf(has ? xml[(w2 * 2 + 1) * (4 * NH) + HL * tg_ + i] : 0.f, f[i], l[i]);
                    }
                    if (some) {
                        const float4 o = xchg(w2)[mt * 32 + ln];
                        o4.x = fmaf(o.x, f[0], o4.x);
                        o4.y = fmaf(o.y, f[HL - 1], o4.y);
                        o4.z = fmaf(o.z, f[0], o4.z);
                        o4.w = fmaf(o.w, f[HL - 1], o4.w);
                    }
                }
#pragma unroll
                for (int i = 0; i < HL; i++) {
                    float* dst = folded + (HL * tg_ + i) * ROW;
                    if constexpr (H8)
                        *reinterpret_cast<float2*>(dst + (D / 8) * g_ + 2 * mt) =
                            i == 0 ? make_float2(o4.x, o4.z) : make_float2(o4.y, o4.w);
                    else
                        *reinterpret_cast<float4*>(dst + (D / 8) * g_ + 4 * mt) = o4;
                    if (g_ == 0 && mt == 0) {
                        dst[D] = nan[i] ? __int_as_float(0x7fc00000) : M[i];   // NaN marks a poisoned piece
                        dst[D + 1] = l[i];
                    }
                }
            }
            if (!CLUSTER && bad && tid == 0) atomicOr(p.work_counter + kStatusWord, kStatusBadBlock);
        }
        if (s_piece[slot1].n_pages > 0) rotate_queries(s_piece[slot1], NRED < WARPS ? NRED : 0);
        if (tid == THREADS - 1) {
            s_piece[slot2] = locate(s_piece[slot1].next);
            s_bad[slot2] = 0;
        }
        any = true;
        prev_first = cur.first;
        slot = slot1;
        __syncwarp();
        if (s_piece[slot].n_pages == 0) break;
    }
    if constexpr (CLUSTER) {
        // every part's (O, m, l) lies in its CTA's `folded`: a warp per head adds them up over distributed shared memory
        if (!any && tid < 4 * NH) {   // a part without pages
            folded[tid * ROW + D] = -INFINITY;
            folded[tid * ROW + D + 1] = 0.f;
        }
        if (stalled || (warp == 0 && s_bad[0])) {
            await_epoch();
            if (lane == 0) atomicOr(p.work_counter + kStatusWord, (stalled ? kStatusWaitExpired : 0) | (s_bad[0] ? kStatusBadBlock : 0));
        }
        sync_cluster();
        const int all = static_cast<int>(threadIdx.x) / 32;      // warp of the CTA
        const int h = static_cast<int>(rank) + all * static_cast<int>(cluster_size);
        if (h < group) {
            merge_head(s_piece[0], h, ctas, 4, lane >> 3,
                       [&](int i) {
                           const int r = i / C::HALVES, hf = i - r * C::HALVES;
                           uint32_t at;
                           asm("mapa.shared::cluster.u32 %0, %1, %2;\n"
                               : "=r"(at) : "r"((hf == 0 ? misc_of[0] : misc_of[C::HALVES - 1]) + h * ROW * 4), "r"(r));
                           return at;
                       },
                       [](uint32_t r, int at) { return ld_cluster2(r + at * 4); },
                       [](uint32_t r, int at) { return ld_cluster4(r + at * 4); });
        }
        // the last CTA takes the epoch out, see below; nobody leaves while its rows are being read
        if (threadIdx.x / 32 == C::HALVES * WARPS - 1) leave(false);
        sync_cluster();
        return;
    }
    sync_half();
    if (any && warp >= FIN0) {
        finish_piece(s_piece[slot == 0 ? 2 : slot - 1], prev_first);
    }
    sync_half();
    merge_units();
    if (lane == 0 && (stalled || (any && warp == 0 && s_epoch_lost))) atomicOr(p.work_counter + kStatusWord, kStatusWaitExpired);
    // the last CTA to leave takes the epoch out of the workspace: a replay of this very launch (a
    // captured graph) must not find its own epoch there before CTA 0 has cleared the counters
    __syncthreads();
    if (threadIdx.x < 32) leave(any);
}

}  // namespace ftq
