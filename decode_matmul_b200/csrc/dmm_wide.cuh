// Wide decode-matmul kernel of the fp16 family: fp16 operands, up to 128 batch columns per pass over
// the codes.  (The kernels of dmm_umma.cuh split the activations into four fp8 planes, which is the
// better trade while the product is a weight stream; from some ten batch rows on the planes cost more
// tensor-core time and shared-memory traffic than the fp16 operands cost in the decode.)
//
// Data path.  A decoder thread turns its codes into fp16 weights in registers -- two table look-ups, two
// XORs and four byte-permutes per eight weights, no arithmetic: the table holds the HIGH byte of the half
// q * 2^-17 (kFmtHalf in dmm_common.cuh) -- and writes them into tensor memory as the A operand of
// tcgen05.mma kind::f16 (M = 128, K = 16).  The activations are the B operand: TMA copies 64 k of every
// batch row into shared memory with the 128-byte swizzle and the MMA reads them as they lie there.
// Accumulators are fp32 in TMEM; the epilogue multiplies by 2^15 (2^17, and 1/4 for quarter units) and scale.
//
// Why 256 output rows x up to 128 columns per CTA.  One 16-byte piece of the code stream holds the codes of
// rows g and g + 8, so a thread decodes for two MMA tiles (256 rows).  Per 2 KiB tile of codes (256 rows x
// 32 k) and NB columns an SM needs
//   tensor pipe      4 MMAs of NB / 2 cycles
//   shared memory    96 table look-ups + 32 codes in and out + 1.5 NB
//   integer ALU      9 operations per code and some 40 around them: 180 cycles
// Measured in the steady state (37888 x 8192 .. 32768, one tile per CTA, by the clock seen meanwhile): 270 cycles per tile
// up to 32 columns (the decoders: latency of their waits and look-ups, ALU 70 % busy), 278 at 64, 330 at 112, 370 at 128, where
// only one accumulator set fits and the tensor core waits while the sums are read.  28672 x 8192 with programmatic launches:
// 36.9 us at 17 rows, 37.5 at 32 (the fp8 planes: 42.3, 49), 43 at 64, 62 at 128; 2048 x 8192 x 28672 746 us as a
// single launch and 852 (1.13 PFLOP/s) back to back, when the power cap holds the clock at 1.4 GHz (3455 as passes of 32 rows).
// 112- and 96-column tiles: 783 and 824 single, 886 and 939 back to back.
//
// Accuracy.  kind::f16 truncates when it adds to the accumulator: over a chain of n MMAs the sums shrink by a part
// in 2^24 or so per MMA (measured against 64 bits, random terms: 4.2e-7 after 64, 9.7e-7 after 128, 2.6e-5 after 1792).
// The fp8 planes stay at 7.5e-7 whatever the length.  So a chain is cut after at most kWChain units of 128 k (88
// MMAs, 6.2e-7): the decoder warps add the accumulators to fp32 sums in registers (rounded to nearest) and the
// next chain starts from zero.  (Terms of one sign, activations and weights both, are the worst case: up to 1.3e-6, uncut 1.2e-4;
// the planes 2e-7.)  That is why a column tile ends at 128: its sums are 64 registers per thread.
// Up to 64 columns there are two accumulator sets, so the next chain starts while the last one is read.
//
// Registers.  The compiler allocates 96 per thread, whatever setmaxnreg adds later, and the sums do not leave enough: -Xptxas -v
// shows 144 bytes of spill stores and 48 of loads at 64 columns, 348 and 176 at 128 (fast layout 360 and 152), none at 32.  ncu
// counts some five local loads and as many stores per warp and half unit at 128 columns (from 28672 x 8192 against x 16384),
// those of the chains and epilogues included.
//
// Work split.  A tile of output is (256 rows, NB columns); its reduction is cut into units of 128 k.  While
// there are more tiles than CTAs every CTA computes whole tiles; the units of the tiles that remain are
// split evenly and contiguously over the CTAs (stream-K), partial tiles go through the workspace and
// the last CTA to arrive (ticket), or all of them together (share_fixup), sum them in a fixed order, or straight into
// `out` with atomic adds (DMM_FLAG_ATOMIC).  No CTA depends on another being resident.  With too little workspace for the partials the remaining
// tiles are computed whole.
//
// Warp roles (20 warps, 24 with kConv):
//   0..15  decoders, four groups; group q decodes the half units (64 k) whose CTA-wide number is q mod 4 into
//          its weight slot in TMEM.  Warp wq of a group owns TMEM lanes 32wq..32wq+31.  They also build the
//          look-up table, keep the sums and run the epilogue.  A chain is read, and a segment written out,
//          only after the first units of the next one are decoded, so that the tensor core always has work.
//   16,17  MMA issuers, one per MMA tile (each accumulator has one issuer: the summation order is fixed);
//          warp 16 allocates the tensor memory
//   18     TMA producer of the codes (one thread), 19 of the activations (the only thread whose loads
//          depend on the previous kernel of the stream); warp 19 also clears zero_ptr.
//   kConv (fp32 activations, plain or silu(gate) * up, up to 16 batch rows): warps 19..22 load the activations
//          of every fourth half unit each, round them to fp16 and store them as the TMA would have; warp 23 clears
//          zero_ptr.  A kernel that converts them beforehand costs a launch per product, more than this.
// Every wait is bounded (mbar_wait).
#pragma once
#include "dmm_choice.h"
#include "dmm_umma.cuh"

namespace dmm {

constexpr int kWDecWarps = 16, kWMmaWarp = 16, kWCodeWarp = 18, kWXWarp = 19;
constexpr int kWThreads = 20 * 32;
constexpr int kWConvThreads = 24 * 32, kWLoaders = 4, kWClearWarp = 23;
constexpr int kWConvRows = 16;                  // batch rows up to which the kernel converts fp32 activations itself
                                                // (one piece per lane and quarter; with 32 rows the loaders fall behind)
constexpr int kWMaxCols = 128;
constexpr int kWChain = 11;                     // units (of eight MMAs per accumulator) before the sums leave the tensor core
constexpr int kWDone = 16;                      // ring of "half unit done" barriers
constexpr uint32_t kWUnitBytes = 16 * 4 * 128;  // codes of a unit: 128 k of 16 strips, 512 contiguous bytes of each
constexpr int kWRingPre = 6;                    // ring slots below the table
constexpr uint32_t kWBarBytes = 2048;
constexpr uint32_t kWPreBytes = kWBarBytes + kWRingPre * kWUnitBytes;
constexpr uint32_t kWPostBytes = 100 * 1024;    // behind the table: activation stages and further ring slots
constexpr int kWMaxStages = 16;
constexpr uint32_t kWDynBytes = 0x10000u - 0x400u + kLutBytes + kWPostBytes;
static_assert(kWPreBytes <= 0x10000u - 0x400u, "the code ring does not fit below the table");
static_assert(kWDynBytes <= 232448u, "shared memory plan exceeds the per-CTA limit");

struct WideParams {
    const void *cb;     // fp16 [256, 8]
    float *out;         // [M, N]
    float *partials;    // workspace [grid][2][NB * 256]
    unsigned *tickets;  // workspace, see ticket_bytes in dmm_api.cu, zero between launches
    long long M, N;
    float scale;
    int accumulate, atomic_reduce, sign_convention;
    int nb;             // batch columns per tile: a multiple of 16, at most kWMaxCols
    int units;          // units of 128 k per tile
    int sst;            // super-tiles (256 output rows)
    int whole;          // whole tiles per CTA before the split ones
    int split_grid;     // CTAs that share the split tiles (0: none are left)
    int share_fixup;    // 64-column build: the contributors of a split tile add up its parts together
    Part32 part;        // split units per CTA
    int stages;         // activation stages
    float *zero_ptr;    // optional: buffer this kernel clears on its way
    long long zero_count;
    const void *x;      // kConv: fp32 activations as in UmmaParams
    int x_mode;
    long long x_ld, x_gap, K;
    unsigned dyn_smem_bytes;
};
struct WideArgs {
    WideParams p;
    CUtensorMap codes_map, x_map;
};

// kCols: columns the variant is built for (32, 64 or 128).  Two accumulator sets while the sums leave room.
template <int kCols>
struct WidePlan {
    static constexpr int kSets = kCols <= 64 ? 2 : 1;
    // Code units in flight.  The stream needs some 96 KiB in flight per SM; 128 columns leave room for half of
    // that beside the activations, and stream at less than half the rate.
    static constexpr int kRing = kCols <= 64 ? 2 * kWRingPre : kWRingPre;
    static constexpr uint32_t kXBytes = kWPostBytes - (kRing - kWRingPre) * kWUnitBytes;  // activation stages
    static_assert(kRing % 2 == 0 && kXBytes / (kCols * 128u) >= 4, "too few activation stages");
    static constexpr uint32_t kSetCols = 2 * kCols;
    static constexpr uint32_t kSlotCols = 64;  // [k-tile][MMA tile][16 columns = 32 k x 2 bytes]
    static constexpr uint32_t kACol = kUTmemCols - 4 * kSlotCols;
    static_assert(kSets * kSetCols <= kACol, "TMEM plan exceeds 512 columns");
    static constexpr int kBarCode = 0;                            // [kRing] TMA completion
    static constexpr int kBarEmpty = kBarCode + kRing;            // [kRing] the eight warps that read the unit
    static constexpr int kBarFull = kBarEmpty + kRing;            // [4] the group's four warps
    static constexpr int kBarXFull = kBarFull + 4;                // [kWMaxStages] TMA completion
    static constexpr int kBarDone = kBarXFull + kWMaxStages;      // [kWDone] both issuers' commits: half unit h (mod kWDone) has
                                                                  // been multiplied, its weight slot and activation stage are free
    static constexpr int kBarDReady = kBarDone + kWDone;          // [2 kSets] by MMA tile: its issuer's commit, the chain is complete
    static constexpr int kBarDFree = kBarDReady + 2 * kSets;      // [2 kSets] the eight decoder warps that read it
    static constexpr int kBarCount = kBarDFree + 2 * kSets;
    static_assert(kWDone >= kWMaxStages && kWDone % 4 == 0, "a Done barrier must not be reused before it is waited for");
    static_assert(kBarCount * 8 + 64 <= kWBarBytes && kBarCount <= 96, "barrier block too small");
};

__device__ __forceinline__ void tma_load_2d_plain(uint32_t dst, const void *tmap, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem descriptor], kind::f16, the descriptor as two 32-bit words
__device__ __forceinline__ void mma_ts_f16_lh(uint32_t d, uint32_t a, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc,
                                              uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 bd;\nsetp.ne.b32 p, %5, 0;\nmov.b64 bd, {%2, %3};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, p;\n}\n" ::"r"(d),
        "r"(a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(acc)
        : "memory");
}

// Segments (parts of a tile) of one CTA, in order: first its whole tiles, then what its range of the
// split units covers.
struct WideSeg {
    int ss, nt;    // super-tile and column tile
    int u0, u1;    // units
    int split;     // index of the split tile, -1 for a whole tile
};
struct WideWork {
    int whole, grid, cta, sst, units, i0, i1;
    __device__ __forceinline__ WideWork(const WideParams &p) {
        whole = p.whole;
        grid = static_cast<int>(gridDim.x);
        cta = static_cast<int>(blockIdx.x);
        sst = p.sst;
        units = p.units;
        i0 = i1 = 0;
        if (cta < p.split_grid) {
            i0 = part32_begin(p.part, cta);
            i1 = part32_begin(p.part, cta + 1);
        }
    }
    __device__ __forceinline__ int count() const { return whole + (i1 > i0 ? (i1 - 1) / units - i0 / units + 1 : 0); }
    __device__ __forceinline__ WideSeg get(int seg) const {
        WideSeg s;
        int tile;
        if (seg < whole) {
            tile = seg * grid + cta;
            s.u0 = 0;
            s.u1 = units;
            s.split = -1;
        } else {
            s.split = i0 / units + (seg - whole);
            tile = whole * grid + s.split;
            const int a = s.split * units;
            s.u0 = i0 > a ? i0 - a : 0;
            s.u1 = i1 < a + units ? i1 - a : units;
        }
        s.nt = tile / sst;
        s.ss = tile - s.nt * sst;
        return s;
    }
};

// Fix-up of a split tile by all the CTAs that have a part of it (share_fixup).  Its ticket word counts, in three fields, the CTAs that
// have written their part, the CTAs that have left, and the pieces (32 rows x 16 columns) that have been handed out: at
// most 32, and one more per warp that asks, less than 2^12.  A CTA with nothing else to do stays until all parts are there, but
// never longer than kWHelpCycles; then the warps of all CTAs that stayed take pieces until none is left and add up each in
// the order of the contributors, so that the sums do not depend on who does it.  The last CTA to arrive never waits:
// nothing depends on another CTA being resident.  The last one to leave clears the word.
constexpr unsigned kWCountMask = 1023, kWLeftShift = 10, kWItemShift = 20;
constexpr long long kWHelpCycles = 10000;

// After the part has been written: flags[1] = all parts are there.
__device__ __forceinline__ void fixup_arrive(unsigned *word, unsigned parts, bool stay, int tid, volatile int *flags) {
    __threadfence();
    named_barrier(1, kWDecWarps * 32);
    if (tid == 0) {
        bool all = ((atomicAdd(word, 1u) + 1u) & kWCountMask) == parts;
        if (stay) {
            const long long t0 = clock64();
            while (!all && clock64() - t0 < kWHelpCycles) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
                all = (v & kWCountMask) == parts;
            }
        }
        flags[1] = all;
    }
    named_barrier(1, kWDecWarps * 32);
}
__device__ __forceinline__ int fixup_item(unsigned *word, int lane) {
    unsigned got = 0;
    if (lane == 0) got = atomicAdd(word, 1u << kWItemShift);
    return static_cast<int>(__shfl_sync(0xffffffffu, got, 0) >> kWItemShift);
}
__device__ __forceinline__ void fixup_leave(unsigned *word, unsigned parts, int tid) {
    named_barrier(1, kWDecWarps * 32);  // (flags[1] is reused by the next segment)
    if (tid == 0) {
        const unsigned old = atomicAdd(word, 1u << kWLeftShift);
        if (((old >> kWLeftShift) & kWCountMask) == parts - 1u) *word = 0;
    }
}

// Chains of one segment: its units cut into equal parts of at most kWChain.
__device__ __forceinline__ int wide_chains(int units) { return (units + kWChain - 1) / kWChain; }

template <int kCols, bool kFast, bool kConv>
__global__ void __launch_bounds__(kConv ? kWConvThreads : kWThreads, 1) wide_kernel(const __grid_constant__ WideArgs args) {
    using Plan = WidePlan<kCols>;
    constexpr int kThreads = kConv ? kWConvThreads : kWThreads;
    constexpr int kSets = Plan::kSets, kRing = Plan::kRing;
    const WideParams &p = args.p;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t lut_addr = (base + kWPreBytes + 0xFFFFu) & ~0xFFFFu;
    const uint32_t x_addr = lut_addr + kLutBytes;  // 1024-byte aligned, as the swizzle needs
    volatile int *flags = reinterpret_cast<volatile int *>(smem_raw + Plan::kBarCount * 8);  // [0]=failed [1]=last
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem_raw + Plan::kBarCount * 8 + 16);
    auto bar = [&](int i) -> uint32_t { return base + 8u * static_cast<uint32_t>(i); };

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint4 cb_pre = lut_prefetch(p.cb, tid);
    // ring slots: kWRingPre below the table, the others behind the activation stages
    auto ring_slot = [&](int rs) -> uint32_t {
        return rs < kWRingPre ? base + kWBarBytes + static_cast<uint32_t>(rs) * kWUnitBytes
                              : x_addr + Plan::kXBytes + static_cast<uint32_t>(rs - kWRingPre) * kWUnitBytes;
    };
    if (x_addr + kWPostBytes > base + p.dyn_smem_bytes) {  // uniform over the grid
        if (tid == 0) raise_status(DMM_STATUS_BAD_SMEM);
        return;
    }
    const WideWork work(p);
    const int nseg = work.count();
    const uint32_t stage_b = static_cast<uint32_t>(p.nb) * 128u;

    // ---- set-up: the decoders build the table; the other warps initialise the barriers, allocate TMEM and go on
    // (the code stream starts flowing meanwhile), arriving on the decoders' barrier only ----
    bool bad_cb = false;
    if (warp < kWDecWarps) {
        bad_cb = lut_fill(lut_addr, p.cb, 1, p.sign_convention, kFmtHalf, tid, kWDecWarps * 32, true, &cb_pre);
        named_barrier(4, kThreads);
    } else {
        const int bt = tid - kWDecWarps * 32;
        if (bt < Plan::kBarCount) {
            uint32_t count = 1;                                                     // TMA completion, commit
            if (bt >= Plan::kBarEmpty && bt < Plan::kBarFull) count = 8;
            if (bt >= Plan::kBarFull && bt < Plan::kBarXFull) count = 4;
            if (bt >= Plan::kBarDone && bt < Plan::kBarDReady) count = 2;
            if (bt >= Plan::kBarDFree) count = kWDecWarps / 2;
            mbar_init(bar(bt), count);
            if (bt == 0) {
                flags[0] = 0;
                flags[1] = 0;
            }
            fence_mbar_init();
        }
        if (warp == kWMmaWarp) tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kUTmemCols);
        fence_async_smem();
        tc_fence_before();
        named_barrier(3, kThreads - kWDecWarps * 32);
        named_barrier_arrive(4, kThreads);
    }
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    grid_dep_launch();

    // 128 columns: the decoders need 64 registers for the sums.  Of the 96 x 640 registers of the launch they take
    // 112 x 512 and leave 32 x 128 to the other warpgroup, which is all of them.
    if (kCols > 64 && warp >= kWDecWarps) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp < kWDecWarps) {
        // =============================== decoders ===============================
        if (kCols > 64) asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        const int q = warp >> 2, wq = warp & 3;
        if (bad_cb) raise_status(DMM_STATUS_BAD_CODEBOOK);
        const LutLane ll = lut_lane(lut_addr, lane, true);
        const uint32_t tlane = tmem + (static_cast<uint32_t>(wq * 32) << 16);
        // this group decodes half `hf` of the units of parity `par`, into weight slot q
        const int par = q >> 1, hf = q & 1;
        const uint32_t acol = tlane + Plan::kACol + static_cast<uint32_t>(q) * Plan::kSlotCols;
        const uint32_t lane_off = (wq * 4 + (lane >> 3)) * 512 + hf * 256 + (lane & 7) * 16;
        const int mt = q >> 1;   // its part of the sums: MMA tile mt, column groups of parity q % 2
        int rs = par;            // ring slot of my next unit, and the parity of its barrier
        uint32_t cpar = 0;
        constexpr int kFix = 3;  // partial tiles read at a time in the fix-up
        constexpr int kGroups = kCols / 32;  // groups of 16 columns whose sums this thread keeps
        float sum[kGroups][16];  // of the chains of the current segment that have been read
        auto clear_sums = [&] {
#pragma unroll
            for (int g = 0; g < kGroups; ++g)
#pragma unroll
                for (int e = 0; e < 16; ++e) sum[g][e] = 0.f;
        };
        clear_sums();

        int un = 0;              // units of this CTA before the current chain
        int chains = 0;          // chains of this CTA so far (the accumulator set and the phase of its barriers)
        bool code_ok = false;    // the codes of my next unit were seen to have landed
        bool pending = false;    // there is a chain that has not been read yet
        int ended = -1;          // the segment that it ends, if it does (looked up again then: registers are short here)
        for (int seg = 0, c = 0, nc = 0, len = 0;;) {
            // next chain: c of nc of segment seg
            const bool more = seg < nseg;
            int u_end = un, first_part = un;
            if (more) {
                if (c == 0) {
                    const WideSeg s = work.get(seg);
                    len = s.u1 - s.u0;
                    nc = wide_chains(len);
                }
                u_end = un + (len * (c + 1) / nc - len * c / nc);
                // what is decoded before the previous chain is read: one half unit per group
                first_part = pending ? (un + 2 < u_end ? un + 2 : u_end) : u_end;
            }
            int u = un + ((un ^ par) & 1);
            for (int part = 0; part < 2; ++part) {
                const int stop = part == 0 ? first_part : u_end;
                for (; u < stop; u += 2) {
                    if (!code_ok) mbar_wait(bar(Plan::kBarCode + rs), cpar, flags);
                    const uint32_t slot_addr = ring_slot(rs);
                    const int v = 2 * u + hf - 4;  // the half unit that the weight slot held before
                    const bool done_ok = v < 0 || mbar_test(bar(Plan::kBarDone + (v & (kWDone - 1))), (v / kWDone) & 1);
                    uint4 cw[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if constexpr (kFast)
                            cw[i] = fetch_fast_ktile(slot_addr, 4, wq, lane, 2 * hf + i);
                        else
                            cw[i] = lds128(slot_addr + lane_off + i * 128);
                    }
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t w[4] = {cw[i].x, cw[i].y, cw[i].z, cw[i].w};
                        uint32_t r[16];
                        if constexpr (kCols <= 64) {
                            uint32_t r1[16];
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const uint4 d0 = decode8_half<0>(w[t], ll), d1 = decode8_half<1>(w[t], ll);
                                r[4 * t] = d0.x; r[4 * t + 1] = d0.y; r[4 * t + 2] = d0.z; r[4 * t + 3] = d0.w;
                                r1[4 * t] = d1.x; r1[4 * t + 1] = d1.y; r1[4 * t + 2] = d1.z; r1[4 * t + 3] = d1.w;
                            }
                            if (i == 0) {
                                if (!done_ok) mbar_wait(bar(Plan::kBarDone + (v & (kWDone - 1))), (v / kWDone) & 1, flags);
                                tc_fence_after();
                            }
                            tmem_st16(acol + i * 32, r);
                            tmem_st16(acol + i * 32 + 16, r1);
                        } else {  // one MMA tile after the other: the sums leave no registers for both
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const uint4 d = decode8_half<0>(w[t], ll);
                                r[4 * t] = d.x; r[4 * t + 1] = d.y; r[4 * t + 2] = d.z; r[4 * t + 3] = d.w;
                            }
                            if (i == 0) {
                                if (!done_ok) mbar_wait(bar(Plan::kBarDone + (v & (kWDone - 1))), (v / kWDone) & 1, flags);
                                tc_fence_after();
                            }
                            tmem_st16(acol + i * 32, r);
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const uint4 d = decode8_half<1>(w[t], ll);
                                r[4 * t] = d.x; r[4 * t + 1] = d.y; r[4 * t + 2] = d.z; r[4 * t + 3] = d.w;
                            }
                            tmem_st16(acol + i * 32 + 16, r);
                        }
                    }
                    const int rs_done = rs;
                    rs += 2;
                    if (rs >= kRing) {
                        rs -= kRing;
                        cpar ^= 1u;
                    }
                    code_ok = mbar_test(bar(Plan::kBarCode + rs), cpar);
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bar(Plan::kBarFull + q));
                        mbar_arrive(bar(Plan::kBarEmpty + rs_done));
                    }
                }
                if (part == 0 && pending) {
                    // ---------------- the previous chain: its accumulators into the sums ----------------
                    const int set = (chains - 1) & (kSets - 1);
                    mbar_wait(bar(Plan::kBarDReady + 2 * set + mt), ((chains - 1) / kSets) & 1, flags);
                    tc_fence_after();
                    const uint32_t dcol = tlane + static_cast<uint32_t>(set) * Plan::kSetCols + static_cast<uint32_t>(mt * kCols);
#pragma unroll
                    for (int g = 0; g < kGroups; ++g) {
                        const int b0 = 32 * g + 16 * (q & 1);
                        if (b0 < p.nb) {
                            uint32_t a[16];
                            __syncwarp();
                            tmem_ld16(dcol + static_cast<uint32_t>(b0), a);
                            tmem_wait_ld(a);
#pragma unroll
                            for (int e = 0; e < 16; ++e) sum[g][e] += __uint_as_float(a[e]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(Plan::kBarDFree + 2 * set + mt));

                    if (ended >= 0) {
                        // ---------------- epilogue of the previous segment ----------------
                        const WideSeg prev = work.get(ended);
                        const int trow = wq * 32 + lane;
                        const long long n = kFast ? static_cast<long long>(prev.ss) * 256 + 32 * (4 * mt + wq) + lane
                                                  : (static_cast<long long>(prev.ss) * 16 + wq * 4 + (lane >> 3)) * 16 + 8 * mt + (lane & 7);
                        const long long m0 = static_cast<long long>(prev.nt) * p.nb;
                        const int mcols = static_cast<int>(p.M - m0 < p.nb ? p.M - m0 : p.nb);  // columns that are batch rows
                        const bool row_ok = n < p.N;
                        float *const out = p.out + m0 * p.N + n;
                        const bool full = prev.u0 == 0 && prev.u1 == p.units;
                        // (2^15 first: exact, and the product with scale then rounds and overflows as scale * sum does)
                        auto put = [&](int b, float v) {
                            float *const o = out + b * p.N;
                            const float r = v * 32768.0f * p.scale;
                            *o = p.accumulate ? *o + r : r;
                        };
                        if (p.atomic_reduce || full) {
                            if (row_ok) {
#pragma unroll
                                for (int g = 0; g < kGroups; ++g) {
                                    const int b0 = 32 * g + 16 * (q & 1);
#pragma unroll
                                    for (int e = 0; e < 16; ++e) {
                                        if (b0 + e >= mcols) continue;
                                        if (p.atomic_reduce)
                                            atomicAdd(out + (b0 + e) * p.N, sum[g][e] * 32768.0f * p.scale);
                                        else
                                            put(b0 + e, sum[g][e]);
                                    }
                                }
                            }
                        } else {
                            const long long part_sz = static_cast<long long>(p.nb) * 256;
                            float *const mine = p.partials + (2ll * work.cta + (prev.u0 > 0 ? 0 : 1)) * part_sz +
                                                static_cast<long long>(mt) * p.nb * 128 + trow;
#pragma unroll
                            for (int g = 0; g < kGroups; ++g) {
                                const int b0 = 32 * g + 16 * (q & 1);
#pragma unroll
                                for (int e = 0; e < 16; ++e)
                                    if (b0 + e < mcols) __stcg(mine + (b0 + e) * 128, sum[g][e]);
                            }
                            if constexpr (kCols == 64) {
                                if (p.share_fixup) {
                                    const int a = prev.split * p.units;
                                    const int c_lo = part32_owner(p.part, a), c_hi = part32_owner(p.part, a + p.units - 1);
                                    const unsigned parts = static_cast<unsigned>(c_hi - c_lo + 1);
                                    unsigned *const word = p.tickets + c_lo;
                                    fixup_arrive(word, parts, ended == nseg - 1, tid, flags);
                                    if (flags[1] != 0) {
                                        __threadfence();
                                        const int items = (mcols + 15) / 16 * 8;  // (16 columns, MMA tile, lane quarter)
                                        for (;;) {
                                            const int item = fixup_item(word, lane);
                                            if (item >= items) break;
                                            const int iq = item & 3, im = (item >> 2) & 1, b0 = (item >> 3) * 16;
                                            float v[16];
#pragma unroll
                                            for (int e = 0; e < 16; ++e) v[e] = 0.f;
                                            // fixed summation order; kFix contributors at a time
                                            for (int c0 = c_lo; c0 <= c_hi; c0 += kFix) {
                                                float l[kFix][16];
#pragma unroll
                                                for (int k = 0; k < kFix; ++k) {
                                                    const int cc = c0 + k <= c_hi ? c0 + k : c_hi;
                                                    const float *src = p.partials + (2ll * cc + (part32_begin(p.part, cc) > a ? 0 : 1)) * part_sz +
                                                                       (static_cast<long long>(im) * p.nb + b0) * 128 + iq * 32 + lane;
#pragma unroll
                                                    for (int e = 0; e < 16; ++e)
                                                        l[k][e] = b0 + e < mcols && c0 + k <= c_hi ? __ldcg(src + e * 128) : 0.f;
                                                }
#pragma unroll
                                                for (int k = 0; k < kFix; ++k)
#pragma unroll
                                                    for (int e = 0; e < 16; ++e) v[e] += l[k][e];
                                            }
                                            const long long in = kFast ? static_cast<long long>(prev.ss) * 256 + 32 * (4 * im + iq) + lane
                                                                       : (static_cast<long long>(prev.ss) * 16 + iq * 4 + (lane >> 3)) * 16 + 8 * im + (lane & 7);
                                            if (in < p.N) {
                                                float *const o = p.out + (m0 + b0) * p.N + in;
#pragma unroll
                                                for (int e = 0; e < 16; ++e)
                                                    if (b0 + e < mcols) {
                                                        const float r = v[e] * 32768.0f * p.scale;
                                                        o[e * p.N] = p.accumulate ? o[e * p.N] + r : r;
                                                    }
                                            }
                                        }
                                    }
                                    fixup_leave(word, parts, tid);
                                    clear_sums();
                                    continue;
                                }
                            }
                            __threadfence();
                            named_barrier(1, kWDecWarps * 32);
                            const int a = prev.split * p.units;
                            const int c_lo = part32_owner(p.part, a), c_hi = part32_owner(p.part, a + p.units - 1);
                            if (tid == 0) {
                                const unsigned old = atomicAdd(p.tickets + c_lo, 1u);
                                const int last = old == static_cast<unsigned>(c_hi - c_lo);
                                if (last) p.tickets[c_lo] = 0;
                                flags[1] = last;
                            }
                            named_barrier(1, kWDecWarps * 32);
                            if (flags[1] != 0) {
                                __threadfence();
#pragma unroll
                                for (int g = 0; g < kGroups; ++g) {
                                    const int b0 = 32 * g + 16 * (q & 1);
                                    if (b0 < mcols) {
                                        float v[16];
#pragma unroll
                                        for (int e = 0; e < 16; ++e) v[e] = 0.f;
                                        // fixed summation order; kFix contributors at a time
                                        for (int c0 = c_lo; c0 <= c_hi; c0 += kFix) {
                                            float l[kFix][16];
#pragma unroll
                                            for (int k = 0; k < kFix; ++k) {
                                                const int cc = c0 + k <= c_hi ? c0 + k : c_hi;
                                                const float *src = p.partials + (2ll * cc + (part32_begin(p.part, cc) > a ? 0 : 1)) * part_sz +
                                                                   (static_cast<long long>(mt) * p.nb + b0) * 128 + trow;
#pragma unroll
                                                for (int e = 0; e < 16; ++e)
                                                    l[k][e] = b0 + e < mcols && c0 + k <= c_hi ? __ldcg(src + e * 128) : 0.f;
                                            }
#pragma unroll
                                            for (int k = 0; k < kFix; ++k)
#pragma unroll
                                                for (int e = 0; e < 16; ++e) v[e] += l[k][e];
                                        }
                                        if (row_ok) {
#pragma unroll
                                            for (int e = 0; e < 16; ++e)
                                                if (b0 + e < mcols) put(b0 + e, v[e]);
                                        }
                                    }
                                }
                            }
                            named_barrier(1, kWDecWarps * 32);  // flags[1] is reused by the next segment
                        }
                        clear_sums();
                    }
                }
            }
            if (!more) break;
            un = u_end;
            ++chains;
            pending = true;
            ended = -1;
            if (++c == nc) {
                c = 0;
                ended = seg++;
            }
        }
    } else if (warp < kWCodeWarp) {
        // =============================== MMA issuers ===============================
        const int mt = warp - kWMmaWarp;
        const bool leader = elect_one();
        // D fp32 (1 at bit 4), A and B fp16 (0), N >> 3 at bit 17, M >> 4 at bit 24
        const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(p.nb >> 3) << 17) | ((128u >> 4) << 24);
        // 128-byte swizzle (2 at bit 61), 8-row groups 1024 bytes apart, version 1 at bit 46
        const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
        const uint32_t a0 = tmem + Plan::kACol + static_cast<uint32_t>(mt * 16);
        const uint32_t d0 = tmem + static_cast<uint32_t>(mt * kCols);
        const uint32_t x16 = ((x_addr >> 4) & 0x3FFFu) | (1u << 16), stage16 = stage_b >> 4;
        int xs = 0, h = 0, chains = 0;  // h: half units of this CTA so far
        uint32_t xpar = 0;
        bool x_ok = false, a_ok = false;  // the operands of the next half unit were seen to be ready
        for (int seg = 0; seg < nseg; ++seg) {
            const WideSeg s = work.get(seg);
            const int len = s.u1 - s.u0, nc = wide_chains(len);
            for (int c = 0; c < nc; ++c, ++chains) {
                const int set = chains & (kSets - 1);
                if (chains >= kSets) {
                    mbar_wait(bar(Plan::kBarDFree + 2 * set + mt), ((chains / kSets) - 1) & 1, flags);
                    tc_fence_after();
                }
                const uint32_t d = d0 + static_cast<uint32_t>(set) * Plan::kSetCols;
                uint32_t acc = 0u;
                const int n = len * (c + 1) / nc - len * c / nc;
                for (int e = 0; e < 2 * n; ++e) {
                    const int sl = h & 3;
                    if (!x_ok) mbar_wait(bar(Plan::kBarXFull + xs), xpar, flags);
                    if (!a_ok) mbar_wait(bar(Plan::kBarFull + sl), (h >> 2) & 1, flags);
                    tc_fence_after();
                    const uint32_t xlo = x16 + static_cast<uint32_t>(xs) * stage16;
                    const uint32_t a = a0 + static_cast<uint32_t>(sl) * Plan::kSlotCols;
                    const int done = h & (kWDone - 1);
                    ++h;
                    if (++xs == p.stages) {
                        xs = 0;
                        xpar ^= 1u;
                    }
                    x_ok = mbar_test(bar(Plan::kBarXFull + xs), xpar);
                    a_ok = mbar_test(bar(Plan::kBarFull + (h & 3)), (h >> 2) & 1);
                    if (leader) {
                        mma_ts_f16_lh(d, a, xlo, desc_hi, idesc, acc);
                        mma_ts_f16_lh(d, a + 8, xlo + 2, desc_hi, idesc, 1u);
                        mma_ts_f16_lh(d, a + 32, xlo + 4, desc_hi, idesc, 1u);
                        mma_ts_f16_lh(d, a + 40, xlo + 6, desc_hi, idesc, 1u);
                        tc_commit(bar(Plan::kBarDone + done));
                    }
                    acc = 1u;
                }
                if (leader) tc_commit(bar(Plan::kBarDReady + 2 * set + mt));
            }
        }
    } else if (warp == kWCodeWarp) {
        // =============================== TMA producer: codes ===============================
        if (lane == 0) {
            // codes that no other column tile reads again need not stay in L2
            const uint64_t policy = p.M <= p.nb ? policy_evict_first() : policy_evict_normal();
            int rs = 0;
            uint32_t par = 1;
            uint32_t n = 0;
            for (int seg = 0; seg < nseg; ++seg) {
                const WideSeg s = work.get(seg);
                for (int u = s.u0; u < s.u1; ++u, ++n) {
                    if (n >= kRing) mbar_wait(bar(Plan::kBarEmpty + rs), par, flags);
                    const uint32_t b = bar(Plan::kBarCode + rs);
                    mbar_arrive_expect_tx(b, kWUnitBytes);
                    // always the full box: words past the row or strips past N read as zero
                    tma_load_2d(ring_slot(rs), &args.codes_map, kFast ? u * 256 : u * 128,
                                kFast ? s.ss * 8 : s.ss * 16, b, policy);
                    if (++rs == kRing) {
                        rs = 0;
                        par ^= 1u;
                    }
                }
            }
            if (flags[0]) {  // a wait gave up: let the loads in flight land before the CTA exits
                for (uint32_t e = 0; e < kRing && e < n; ++e) {
                    const uint32_t i = n - 1 - e;
                    mbar_wait_limit(bar(Plan::kBarCode + static_cast<int>(i % kRing)), (i / kRing) & 1, 20ll * 1000 * 1000);
                }
            }
        }
    } else if (kConv) {
        // ======================= activation loaders: fp32 to fp16 =======================
        grid_dep_wait();
        if (warp == kWClearWarp) {
            if (p.zero_ptr != nullptr)  // a later kernel will accumulate into it
                for (long long i = static_cast<long long>(blockIdx.x) * 32 + lane; i < p.zero_count;
                     i += static_cast<long long>(gridDim.x) * 32)
                    p.zero_ptr[i] = 0.f;
        } else {
            const int total = static_cast<int>(p.M) * 8;  // pieces of a unit: 8 k of one row, 16 bytes of shared memory
            const int ns = p.stages;
            int n = warp - kWXWarp, nbase = 0;
            for (int seg = 0; seg < nseg; ++seg) {
                const WideSeg s = work.get(seg);
                const int nend = nbase + 2 * (s.u1 - s.u0);  // half units
                for (; n < nend; n += kWLoaders) {
                    const int k0 = (2 * s.u0 + n - nbase) * 64, xs = n % ns;
                    const uint32_t stage = x_addr + static_cast<uint32_t>(xs) * stage_b;
                    // All loads of the four pieces first, at addresses that are always valid: with a branch around
                    // each piece they went out one after the other.  (Rows past M are not written: they only
                    // reach accumulator columns that nobody reads.  k past the row is zero.)
                    float4 f[4][2], g[4][2];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int pc = min(e * 32 + lane, total - 1), k = k0 + (pc & 7) * 8;
                        const float *src = reinterpret_cast<const float *>(p.x) + (pc >> 3) * p.x_ld + (k < p.K ? k : 0);
                        f[e][0] = __ldcg(reinterpret_cast<const float4 *>(src));
                        f[e][1] = __ldcg(reinterpret_cast<const float4 *>(src + 4));
                        if (p.x_mode == kXSiluMul) {
                            g[e][0] = __ldcg(reinterpret_cast<const float4 *>(src + p.x_gap));
                            g[e][1] = __ldcg(reinterpret_cast<const float4 *>(src + p.x_gap + 4));
                        }
                    }
                    if (n >= ns) {  // the stage held half unit n - ns
                        const int v = n - ns;
                        mbar_wait(bar(Plan::kBarDone + (v & (kWDone - 1))), (v / kWDone) & 1, flags);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int pc = e * 32 + lane, row = pc >> 3, ch = pc & 7;
                        uint32_t h[4];
                        pack_piece(p.x_mode, f[e], g[e], h);
                        const bool in = k0 + ch * 8 < p.K;
                        if (pc < total)
                            sts128(stage + row * 128 + ((ch ^ (row & 7)) << 4),
                                   make_uint4(in ? h[0] : 0u, in ? h[1] : 0u, in ? h[2] : 0u, in ? h[3] : 0u));
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(Plan::kBarXFull + xs));
                }
                nbase = nend;
            }
        }
    } else if (warp == kWXWarp) {
        // ============================ TMA producer: activations ============================
        grid_dep_wait();
        asm volatile("fence.proxy.async;" ::: "memory");  // x may be the previous kernel's plain stores
        if (lane == 0) {
            int xs = 0;
            uint32_t n = 0;
            const uint32_t ns = static_cast<uint32_t>(p.stages);
            for (int seg = 0; seg < nseg; ++seg) {
                const WideSeg s = work.get(seg);
                for (int u = 2 * s.u0; u < 2 * s.u1; ++u, ++n) {
                    if (n >= ns) {  // the stage held half unit n - ns
                        const uint32_t v = n - ns;
                        mbar_wait(bar(Plan::kBarDone + static_cast<int>(v & (kWDone - 1))), (v / kWDone) & 1, flags);
                    }
                    const uint32_t b = bar(Plan::kBarXFull + xs);
                    mbar_arrive_expect_tx(b, stage_b);
                    // k past the row reads as zero (the weights decoded there are finite), and so do rows past M
                    tma_load_2d_plain(x_addr + static_cast<uint32_t>(xs) * stage_b, &args.x_map, u * 64, s.nt * p.nb, b);
                    if (++xs == p.stages) xs = 0;
                }
            }
            if (flags[0]) {
                for (uint32_t e = 0; e < ns && e < n; ++e) {
                    const uint32_t i = n - 1 - e;
                    mbar_wait_limit(bar(Plan::kBarXFull + static_cast<int>(i % ns)), (i / ns) & 1, 20ll * 1000 * 1000);
                }
            }
        } else if (p.zero_ptr != nullptr) {  // a later kernel will accumulate into it
            for (long long i = static_cast<long long>(blockIdx.x) * 31 + lane - 1; i < p.zero_count;
                 i += static_cast<long long>(gridDim.x) * 31)
                p.zero_ptr[i] = 0.f;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kWMmaWarp) tmem_dealloc(tmem, kUTmemCols);
}

// Batch columns per tile: as few equal column tiles as fit, in steps of 16.
inline int wide_cols(long long M) {
    const long long nt = (M + kWMaxCols - 1) / kWMaxCols;
    return static_cast<int>(((M + nt - 1) / nt + 15) / 16 * 16);
}
// Workspace bytes of the partial tiles.
inline size_t wide_partial_bytes(long long M, int num_sms) {
    return static_cast<size_t>(num_sms) * 2 * static_cast<size_t>(wide_cols(M)) * 256 * sizeof(float);
}

// fp32 activations (plain, or silu(gate) * up) rounded to fp16 once per call: [M, K] fp16 for the TMA of
// wide_kernel.  One thread per eight values.
__global__ void __launch_bounds__(128) half_kernel(const void *x, int x_mode, long long x_ld, long long x_gap, int M,
                                                   long long K, __half *out) {
    grid_dep_wait();
    grid_dep_launch();
    const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long per_row = K / 8;
    if (idx >= M * per_row) return;
    const int row = static_cast<int>(idx / per_row);
    const long long k0 = (idx - row * per_row) * 8;
    uint32_t h[4];
    load_piece(x, x_mode, x_ld, x_gap, row, k0, h);
    *reinterpret_cast<uint4 *>(out + row * K + k0) = make_uint4(h[0], h[1], h[2], h[3]);
}
inline int launch_half(const void *x, int x_mode, long long x_ld, long long x_gap, int M, long long K, void *out, bool pdl,
                       cudaStream_t stream) {
    const long long pieces = M * (K / 8);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>((pieces + 127) / 128));
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, half_kernel, x, x_mode, x_ld, x_gap, M, K, reinterpret_cast<__half *>(out));
}

// Tensor map of the activations: fp16 [M, K], rows x_ld elements apart, box 64 k x nb rows, 128-byte swizzle.
inline int make_x_map(CUtensorMap *map, const void *x, long long M, long long K, long long x_ld, int nb) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return cudaErrorNotSupported;
    const cuuint64_t gdim[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(M)};
    const cuuint64_t gstride[1] = {static_cast<cuuint64_t>(x_ld) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(nb)};
    const cuuint32_t estride[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x), gdim, gstride, box, estride,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : static_cast<int>(cudaErrorInvalidValue);
}

template <int kCols, bool kFast, bool kConv>
inline int launch_wide_as(WideArgs &args, unsigned grid, bool pdl, cudaStream_t stream) {
    auto kernel = wide_kernel<kCols, kFast, kConv>;
    // the shared-memory attribute is set once per kernel variant and device, not on every launch
    static std::atomic<unsigned long long> attr_done;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev >= 64 || !((attr_done.load(std::memory_order_acquire) >> dev) & 1ull)) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kWDynBytes));
        if (err != cudaSuccess) return err;
        if (dev < 64) attr_done.fetch_or(1ull << dev, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kConv ? kWConvThreads : kWThreads);
    cfg.dynamicSmemBytes = kWDynBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

// p carries cb, out, partials, tickets, M, N, scale, flags, sign convention and the buffer to clear; x is fp16
// [M, K] with rows x_ld elements apart, or fp32 as x_mode says (at most kWConvRows rows).  partial_capacity: bytes of workspace behind p.partials.
inline int launch_wide(WideParams p, const void *x, int x_mode, long long x_ld, long long x_gap, const void *codes, long long K, bool fast_layout,
                       size_t partial_capacity, int num_sms, bool pdl, cudaStream_t stream) {
    WideArgs args = {};
    p.nb = wide_cols(p.M);
    p.units = static_cast<int>((K + 127) / 128);
    p.sst = static_cast<int>((p.N + 255) / 256);
    const long long tiles = static_cast<long long>(p.sst) * ((p.M + p.nb - 1) / p.nb);
    if (tiles * p.units >= (1ll << 31)) return DMM_ERR_SHAPE;
    long long whole = tiles / num_sms, rest = tiles - whole * num_sms;
    long long grid = whole > 0 ? num_sms : 0;
    const bool can_split = p.atomic_reduce || partial_capacity >= wide_partial_bytes(p.M, num_sms);
    if (rest > 0) {
        const WideSplit split = wide_split(p.nb, p.units, rest, num_sms, can_split, p.atomic_reduce != 0);
        const long long parts = split.parts;
        p.share_fixup = split.share ? 1 : 0;
        p.split_grid = static_cast<int>(parts);
        if (!can_split) {  // one whole tile each
            p.part.a = p.units;
            p.part.b = 0;
        } else {
            p.part.a = static_cast<int>(rest * p.units / parts);
            p.part.b = static_cast<int>(rest * p.units % parts);
        }
        if (parts > grid) grid = parts;
    }
    p.whole = static_cast<int>(whole);
    const uint32_t x_bytes = p.nb <= 32 ? WidePlan<32>::kXBytes : (p.nb <= 64 ? WidePlan<64>::kXBytes : WidePlan<128>::kXBytes);
    const int fit = static_cast<int>(x_bytes / (static_cast<uint32_t>(p.nb) * 128u));
    p.stages = fit < kWMaxStages ? fit : kWMaxStages;
    p.dyn_smem_bytes = kWDynBytes;
    p.x = x;
    p.x_mode = x_mode;
    p.x_ld = x_ld;
    p.x_gap = x_gap;
    p.K = K;
    args.p = p;
    int rc = make_codes_map(&args.codes_map, codes, p.N, K, 4, fast_layout);
    if (rc) return rc;
    const unsigned g = static_cast<unsigned>(grid);
    if (x_mode != kXHalf) {
        if (p.M > kWConvRows) return DMM_ERR_SHAPE;
        return fast_layout ? launch_wide_as<32, true, true>(args, g, pdl, stream)
                           : launch_wide_as<32, false, true>(args, g, pdl, stream);
    }
    rc = make_x_map(&args.x_map, x, p.M, K, x_ld, p.nb);
    if (rc) return rc;
    if (p.nb <= 32)
        return fast_layout ? launch_wide_as<32, true, false>(args, g, pdl, stream)
                           : launch_wide_as<32, false, false>(args, g, pdl, stream);
    if (p.nb <= 64)
        return fast_layout ? launch_wide_as<64, true, false>(args, g, pdl, stream)
                           : launch_wide_as<64, false, false>(args, g, pdl, stream);
    return fast_layout ? launch_wide_as<128, true, false>(args, g, pdl, stream)
                       : launch_wide_as<128, false, false>(args, g, pdl, stream);
}

}  // namespace dmm
