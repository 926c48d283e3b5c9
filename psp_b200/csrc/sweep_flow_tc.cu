// The tree walk of sweep_flow.cu with the products on the tensor cores
// (tcgen05, split TF32), for complex-single factors and kFlowTcMinCols or more
// right-hand sides: same ordered tile list, tickets and
// per-front counters, one CTA per SM.
//
// A complex product C = A B (A: 128 rows x K, B: K x NC right-hand sides) runs
// as one real product: A's rows read as interleaved (re, im) pairs form a
// rows x 2K real matrix, and every entry b of B becomes the 2x2 real block
// [[re b, im b], [-im b, re b]], so the 2 NC real accumulator columns are C's
// (re, im) pairs.  Both operands are split into a tf32 head and tail
// (x = hi + lo) and hi hi + hi lo + lo hi is accumulated in FP32 in tensor
// memory with two MMAs per 8-value K step: A_hi [B_hi | B_lo] (N = 4 NC) and
// A_lo B_hi (N = 2 NC, onto the first 2 NC columns).
//
// One ring of stages (16 complex K columns) holds the TMA copy of G and B's
// planes; a slot is free again when its MMAs have completed.
//   producer (1 warp)     tickets, one tiled TMA copy of G per stage
//   loaders (8 warps)     right-hand sides, copied up to kAhead stages ahead (into
//                         the next tile when what it reads is there) into a small
//                         ring, -> B's planes (128-byte swizzled, K-major); two
//                         groups on alternating stages, each warp a quarter of
//                         a stage's K rows on its own
//   converters (8 warps)  A's split into tensor memory (the MMA reads A there),
//                         lane = row; two groups on alternating stages
//   MMA (1 warp)          a tile's stages in chains of kChainStages, one of
//                         kAccs accumulators per chain
//   epilogue (8 warps)    two groups on alternating tiles (a small tile's write-
//                         out takes longer than its stages); thread = row: sums
//                         a tile's chains in FP32 in tensor memory, adds the
//                         split-K partials and writes its row (8 columns, 64
//                         contiguous bytes, at a time)
//
// What bounds it: at the wide levels a stage takes 0.4 us (converters and MMAs
// about 750 cycles each; 16 KB per SM and 0.4 us is 5.9 TB/s over 148 SMs), at
// the narrow ones the chain of levels (a tile needs about 8 us beside its
// stages).  Everything that is not the product runs beside it: with the right-
// hand sides loaded through registers a stage took 0.85 us, with the children's
// updates and the grid written on the way out a tile's write-out took 5 us
// instead of 3, and with tickets taken two tiles ahead the narrow levels were
// badly balanced (39 instead of 29 ms then per sweep at 116^3).  Measured against one
// launch per level and direction, whole sweeps: 116^3, k = 16: 44.1 -> 26.9 ms
// (1.9 TB/s of factors); 96 x 96 x 76, k = 32: 34.7 -> 16.7 ms.
#include <algorithm>

#include "sweep_flow.cuh"

namespace psp_b200 {

namespace {

using namespace flow;

constexpr int kEpiWarps = 4, kConvWarps = 8, kLoadWarps = 8;
constexpr int kEpiGroups = 2;
constexpr int kEpiThreads = 32 * kEpiWarps, kConvThreads = 32 * kConvWarps, kLoadThreads = 32 * kLoadWarps;
constexpr int kConv0 = kEpiGroups * kEpiThreads, kLoad0 = kConv0 + kConvThreads, kMma0 = kLoad0 + kLoadThreads, kProd0 = kMma0 + 32;
constexpr int kTcThreads = kProd0 + 32;  // 832
constexpr int kGroups = 2, kGroupThreads = kConvThreads / kGroups, kGroupWarps = kConvWarps / kGroups;
constexpr int kLoadGroups = 2, kLoadGroupThreads = kLoadThreads / kLoadGroups, kLoadGroupWarps = kLoadWarps / kLoadGroups;
constexpr int kStageK = kFlowStageK;
constexpr int kRows = kTcRows;
constexpr uint32_t kGBytes = 16384;
constexpr uint32_t kAStageCols = 2 * kStageK;
constexpr uint32_t kTmemCols = 512;
constexpr int kQueue = 3;
constexpr int kSlotMax = 7, kAccMax = 4;
// The tensor core adds each MMA's products into its FP32 accumulator with
// truncation, so an accumulator holds at most kChainStages stages (48 complex
// K); the epilogue sums the chains of a tile in FP32 (round to nearest).
constexpr int kChainStages = 3;
constexpr int kSub = 8;                       // columns of the write-out at a time
static_assert(FlowRows<float>() == kRows, "the tile list's rows");

template <int NC>
struct Cfg {
    static constexpr uint32_t kBPlane = 2 * NC * 128;         // 2 NC rows of B', 32 tf32 each
    static constexpr uint32_t kSlot = kGBytes + 2 * kBPlane;  // G, B hi, B lo
    static constexpr int kSlots = NC == 16 ? 7 : 5;
    static constexpr int kSets = NC == 16 ? 3 : 2;            // split A stages in flight
    static constexpr int kAhead = NC == 16 ? 3 : 2;           // right-hand-side stages in flight per loader group
    static constexpr uint32_t kAccCols = 4 * NC;
    static constexpr int kAccs = NC == 16 ? 4 : 2;
    static constexpr uint32_t kIdescHi = umma::InstrDescTf32(kRows, 4 * NC);
    static constexpr uint32_t kIdescLo = umma::InstrDescTf32(kRows, 2 * NC);
    static constexpr int kWarpK = kStageK / kLoadGroupWarps;  // K rows of a loader warp
    static constexpr uint32_t kPlane = kWarpK * NC * 8;       // one source of its right-hand sides
    static constexpr uint32_t kRawOff = kSlots * kSlot;  // copied right-hand sides: [warp][kAhead][3 planes]
    static constexpr size_t kSmem = kRawOff + kLoadWarps * kAhead * 3 * kPlane + 1024;
    static constexpr int kPer = kWarpK * NC / 2 / 32;         // units per lane: (column, K row pair), or 16-byte copies
    __host__ __device__ static constexpr uint32_t ACol(int ps) { return kAccs * kAccCols + (uint32_t)ps * 2 * kAStageCols; }
    static constexpr uint32_t kSumCol = kAccs * kAccCols + kSets * 2 * kAStageCols;  // sum of a tile's finished chains, per epilogue group
    static_assert(kSumCol + kEpiGroups * 2 * NC <= kTmemCols, "accumulators, A stages and the chain sum fit in TMEM");
    static_assert(kSlots <= kSlotMax && kAccs <= kAccMax && kPer >= 1, "sync arrays");
    static_assert(kSmem <= 225 * 1024, "shared memory per CTA");
};

struct Sync {
    TileCtx<float> queue[kQueue];
    uint64_t tma[kSlotMax], full[kSlotMax], empty[kSlotMax];  // G copied; split and B planes written; MMAs done
    // finished chains, per epilogue group (which only ever sees its own tiles'
    // phases); drained accumulators
    uint64_t accFull[kEpiGroups][kAccMax], accEmpty[kAccMax];
    uint64_t tileFull[kQueue], tileEmpty[kQueue];
    uint64_t mmaDrain;         // the MMA thread's last commit when a role gave up
    uint32_t tmem;
    int abort, isLast[kEpiGroups], lastCta, issued;
};
// loader, converter, epilogue and MMA warps read a tile's words
constexpr int kReaders = kLoadWarps + kConvWarps + kEpiGroups * kEpiWarps + 1;

// ------------------------------------------------------------------ producer

template <int NC>
__device__ void ProducerRole(const FlowFront<float>* __restrict__ fr, const FlowTile* __restrict__ tiles, int n,
                             unsigned char* smem, Sync& S, const FlowWork& w) {
    using C = Cfg<NC>;
    const int lane = threadIdx.x & 31;
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    TileSource<float> src(fr, tiles, n, w.ctrl);
    int g = 0;
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        if (q >= kQueue && !WaitWarp(&S.tileEmpty[qs], ((q / kQueue) - 1) & 1, S, w.status)) break;
        if (lane < kCtxWords) reinterpret_cast<int4*>(&S.queue[qs])[lane] = src.ctx;
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.tileFull[qs]);
        if (src.Done()) break;
        const FlowTile& t = S.queue[qs].t;
        const unsigned char* map = static_cast<const unsigned char*>(S.queue[qs].f.map) + (t.bwd ? 128 : 0);
        const int nst = t.nst;
        bool ok = true;
        for (int st = 0; st < nst; ++st, ++g) {
            const int slot = g % C::kSlots;
            ok = g < C::kSlots || WaitWarp(&S.empty[slot], ((g / C::kSlots) - 1) & 1, S, w.status);
            if (!ok) break;
            if (lane == 0) {
                const int kBase = t.k0 + st * kStageK;
                umma::MbarArriveExpectTx(&S.tma[slot], kGBytes);
                TmaLoadStream(smem + slot * C::kSlot, map, t.bwd ? kBase : t.row0, t.bwd ? t.row0 : kBase, &S.tma[slot],
                              policy);
                S.issued = g + 1;
            }
            __syncwarp();
        }
        if (!ok) break;
        src.Take();
    }
}

// ------------------------------------------------------------------ loaders

__device__ __forceinline__ void Split2(c32 x, float2& hi, float2& lo) {
    umma::SplitTf32Fast(x.re, hi.x, lo.x);
    umma::SplitTf32Fast(x.im, hi.y, lo.y);
}

// Stores column n of K rows 2 kp, 2 kp + 1 into B's planes: one 16-byte chunk
// of each of the rows 2n, 2n + 1 of B'.  Lanes with bit 2 of n store their odd
// row first, so that the lanes of a store instruction cover all eight swizzle
// phases.
__device__ __forceinline__ void StoreB(unsigned char* bHi, uint32_t planeBytes, int kp, int n, c32 b0, c32 b1) {
    float2 h0, l0, h1, l1;
    Split2(b0, h0, l0);
    Split2(b1, h1, l1);
    const uint32_t o0 = umma::Sw128Offset(2 * n, kp), o1 = umma::Sw128Offset(2 * n + 1, kp);
    const bool odd = (n >> 2) & 1;
    const float4 hr = make_float4(h0.x, -h0.y, h1.x, -h1.y), hi = make_float4(h0.y, h0.x, h1.y, h1.x);
    const float4 lr = make_float4(l0.x, -l0.y, l1.x, -l1.y), li = make_float4(l0.y, l0.x, l1.y, l1.x);
    const uint32_t a = odd ? o1 : o0, b = odd ? o0 : o1;
    *reinterpret_cast<float4*>(bHi + a) = odd ? hi : hr;
    *reinterpret_cast<float4*>(bHi + b) = odd ? hr : hi;
    *reinterpret_cast<float4*>(bHi + planeBytes + a) = odd ? li : lr;
    *reinterpret_cast<float4*>(bHi + planeBytes + b) = odd ? lr : li;
}

// One test of a phase, without waiting.
__device__ __forceinline__ bool MbarTest(uint64_t* mbar, uint32_t phase) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(ok)
        : "r"(umma::SmemAddr(mbar)), "r"(phase)
        : "memory");
    return ok != 0;
}

template <int NC>
__device__ void LoaderRole(int k, unsigned char* smem, Sync& S, const FlowWork& w) {
    using C = Cfg<NC>;
    constexpr int kPer = C::kPer, kCopyRows = 64 / NC;  // K rows of one copy of the whole warp
    const int lane = threadIdx.x & 31, lw = (threadIdx.x - kLoad0) / 32;
    const int group = lw / kLoadGroupWarps, k4 = lw % kLoadGroupWarps * C::kWarpK;
    const int n = lane % NC, kp = lane / NC;                     // split: column, pair of the warp's K rows
    const int cn = 2 * (lane % (NC / 2)), cr = lane / (NC / 2);  // copies: column pair, K row of the warp
    const bool pair = (k & 1) == 0;                              // rows start on 16-byte boundaries
    unsigned char* const raw = smem + C::kRawOff + lw * C::kAhead * 3 * C::kPlane;
    const c32* const any = static_cast<const c32*>(w.rnd);       // what a copy of no bytes names
    PdlWait();     // right-hand sides come from the preceding kernels
    PdlTrigger();
    // This warp's stages are the CTA's stages group, group + 2, ...; `gi` is the
    // first stage of tile q, whose words are in registers when `have`, and
    // whose right-hand sides are there when `ready`.
    int q = 0, gi = 0, next = group, now = group;  // stages to copy, to split
    int pending = 0, head = 0, tail = 0;
    uint32_t sources = 0;                          // per ring slot: children's planes copied (2 bits)
    bool have = false, ready = false, done = false;
    int nst = 0, k0 = 0, ke = 0, bwd = 0, s = 0;
    uint32_t bytes = 0;
    const int* lower = nullptr;
    const c32 *src = nullptr, *X = nullptr, *p0 = nullptr, *p1 = nullptr;
    int at[kPer];  // solution rows of the next stage to copy (backward, below the pivots; else -1)
    auto rows = [&](int st) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int kk = k0 + st * kStageK + k4 + cr + i * kCopyRows;
            at[i] = bwd && kk >= s && kk < ke ? __ldg(lower + kk) : -1;
        }
    };
    auto copy = [&](unsigned char* dst, const c32* p, uint32_t b) {
        if (pair) {
            umma::CpAsync16(dst, b ? p : any, b);
        } else {
            umma::CpAsync8(dst, b ? p : any, b ? 8u : 0u);
            umma::CpAsync8(dst + 8, b > 8 ? p + 1 : any, b > 8 ? 8u : 0u);
        }
    };
    auto leave = [&] {  // tile q needs nothing more from this warp
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.tileEmpty[q % kQueue]);
        gi += nst;
        ++q;
        have = false;
    };
    for (;;) {
        while (pending < C::kAhead && !done) {
            if (!have) {
                const int qs = q % kQueue;
                const uint32_t phase = (q / kQueue) & 1;
                if (!__all_sync(~0u, MbarTest(&S.tileFull[qs], phase))) {
                    if (pending > 0) break;
                    if (!WaitWarp(&S.tileFull[qs], phase, S, w.status)) { done = true; break; }
                }
                const FlowTile& t = S.queue[qs].t;
                const FlowFront<float>& f = S.queue[qs].f;
                if (t.front < 0) { done = true; break; }
                nst = t.nst;
                if (next >= gi + nst) { leave(); continue; }  // no stage of this warp
                k0 = t.k0; ke = t.ke; bwd = t.bwd; s = f.s;
                lower = f.lower - s;
                const int c = t.col0 + cn;
                bytes = c + 1 < k ? 16u : c < k ? 8u : 0u;
                src = static_cast<const c32*>(bwd ? w.w : w.rnd) + (int64_t)f.ndOff * k + c;
                X = static_cast<const c32*>(w.x) + c;
                p0 = f.P0 && !bwd ? f.P0 + c : nullptr;
                p1 = f.P1 && !bwd ? f.P1 + c : nullptr;
                have = true;
                ready = false;
                rows(next - gi);
            }
            if (!ready) {
                const FlowTile& t = S.queue[q % kQueue].t;
                ready = TileReady(t, false, S, w);
                if (!ready) {
                    if (pending > 0) break;  // split what is here first
                    ready = TileReady(t, true, S, w);
                    if (!ready) { done = true; break; }
                }
            }
            unsigned char* dst = raw + tail * 3 * C::kPlane + (cr * NC + cn) * 8;
            const int st = next - gi;
#pragma unroll
            for (int i = 0; i < kPer; ++i, dst += kCopyRows * NC * 8) {
                const int kk = k0 + st * kStageK + k4 + cr + i * kCopyRows;
                const uint32_t b = kk < ke ? bytes : 0u;
                copy(dst, at[i] >= 0 ? X + (int64_t)at[i] * k : src + (int64_t)kk * k, b);
                if (p0) copy(dst + C::kPlane, p0 + (int64_t)kk * k, b);
                if (p1) copy(dst + 2 * C::kPlane, p1 + (int64_t)kk * k, b);
            }
            umma::CpAsyncCommit();
            sources = (sources & ~(3u << 2 * tail)) | ((p0 ? 1u : 0u) | (p1 ? 2u : 0u)) << 2 * tail;
            if (++tail == C::kAhead) tail = 0;
            ++pending;
            next += kLoadGroups;
            if (next >= gi + nst) leave();
            else rows(next - gi);
        }
        if (pending == 0) {
            if (done) break;
            continue;
        }
        if (pending >= 3) umma::CpAsyncWait<2>();
        else if (pending == 2) umma::CpAsyncWait<1>();
        else umma::CpAsyncWait<0>();
        __syncwarp();  // every lane's copies of this stage are there
        c32 v[2 * kPer];
        const c32* r = reinterpret_cast<const c32*>(raw + head * 3 * C::kPlane) + 2 * kp * NC + n;
        const uint32_t planes = sources >> 2 * head;
#pragma unroll
        for (int i = 0; i < 2 * kPer; ++i) {
            const int o = i * NC;
            c32 a = mk(0.f, 0.f), b = a;
            if (planes & 1) a = r[o + C::kWarpK * NC];
            if (planes & 2) b = r[o + 2 * C::kWarpK * NC];
            v[i] = r[o] + a + b;
        }
        __syncwarp();  // the ring slot is free again
        if (++head == C::kAhead) head = 0;
        --pending;
        const int slot = now % C::kSlots;
        if (now >= C::kSlots && !WaitWarp(&S.empty[slot], ((now / C::kSlots) - 1) & 1, S, w.status)) break;
        unsigned char* bHi = smem + slot * C::kSlot + kGBytes;
#pragma unroll
        for (int i = 0; i < kPer; ++i) StoreB(bHi, C::kBPlane, k4 / 2 + kp + i, n, v[2 * i], v[2 * i + 1]);
        umma::FenceProxyAsync();
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.full[slot]);
        now += kLoadGroups;
    }
    umma::CpAsyncWaitAll();
}

// ------------------------------------------------------------------ converters

template <int NC>
__device__ void ConverterRole(unsigned char* smem, Sync& S, const FlowWork& w) {
    using C = Cfg<NC>;
    const int lt = threadIdx.x - kConv0, gr = lt / kGroupThreads, ct = lt % kGroupThreads, lane = threadIdx.x & 31;
    int g = 0;
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        if (!WaitWarp(&S.tileFull[qs], (q / kQueue) & 1, S, w.status)) return;
        const int front = S.queue[qs].t.front, nst = S.queue[qs].t.nst, bwd = S.queue[qs].t.bwd;
        if (front < 0) return;
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.tileEmpty[qs]);
        for (int gs = g + ((gr - g) & (kGroups - 1)); gs < g + nst; gs += kGroups) {
            const int slot = gs % C::kSlots;
            if (!WaitWarp(&S.tma[slot], (gs / C::kSlots) & 1, S, w.status)) return;
            // the set is free once the MMAs of its previous stage are done
            const int pg = gs - C::kSets, set = gs % C::kSets;
            const uint32_t tmemA = S.tmem + C::ACol(set) + ((uint32_t)(ct & ~31) << 16);
            if (pg >= 0 && !WaitWarp(&S.empty[pg % C::kSlots], (pg / C::kSlots) & 1, S, w.status)) return;
            const unsigned char* raw = smem + slot * C::kSlot;
            if (!bwd) {
                const c32* ra = reinterpret_cast<const c32*>(raw) + ct;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float hi[kStageK], lw[kStageK];
#pragma unroll
                    for (int kc = 0; kc < kStageK / 2; ++kc) {
                        float2 hv, lv;
                        Split2(ra[(h * kStageK / 2 + kc) * kRows], hv, lv);
                        hi[2 * kc] = hv.x;
                        hi[2 * kc + 1] = hv.y;
                        lw[2 * kc] = lv.x;
                        lw[2 * kc + 1] = lv.y;
                    }
                    umma::TmemStore16(tmemA + h * kStageK, hi);
                    umma::TmemStore16(tmemA + kAStageCols + h * kStageK, lw);
                }
                umma::TmemStoreWait();
                umma::FenceBeforeSync();
            } else {
                // lane = row of G^T: its 128-byte row, chunks swizzled
                const unsigned char* rowp = raw + ct * 128;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float hi[kStageK], lw[kStageK];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 x = *reinterpret_cast<const float4*>(rowp + (((4 * h + i) ^ (ct & 7)) * 16));
                        umma::SplitTf32Fast(x.x, hi[4 * i], lw[4 * i]);
                        umma::SplitTf32Fast(x.y, hi[4 * i + 1], lw[4 * i + 1]);
                        umma::SplitTf32Fast(x.z, hi[4 * i + 2], lw[4 * i + 2]);
                        umma::SplitTf32Fast(x.w, hi[4 * i + 3], lw[4 * i + 3]);
                    }
                    umma::TmemStore16(tmemA + h * kStageK, hi);
                    umma::TmemStore16(tmemA + kAStageCols + h * kStageK, lw);
                }
                umma::TmemStoreWait();
                umma::FenceBeforeSync();
            }
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.full[slot]);
        }
        g += nst;
    }
}

// ------------------------------------------------------------------ MMA

__device__ __forceinline__ int NumChains(int nst) { return (nst + kChainStages - 1) / kChainStages; }

// One lane of a converged warp, always the same.
__device__ __forceinline__ bool ElectOne() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(p));
    return p != 0;
}

// The whole warp walks the stages, so that what the MMAs take (descriptors,
// addresses) stays in warp-uniform registers, and one lane issues.
template <int NC>
__device__ void MmaRole(unsigned char* smem, Sync& S, const FlowWork& w) {
    using C = Cfg<NC>;
    const uint32_t base = __shfl_sync(~0u, umma::SmemAddr(smem), 0), tmem = __shfl_sync(~0u, S.tmem, 0);
    // descriptors of slot 0; an address is their low 14 bits, in 16-byte units
    const uint64_t bDesc = umma::SmemDescSw128(base + kGBytes);
    int slot = 0, set = 0, acc = 0, chain0 = 0, chain1 = 0;  // chains: next barrier of each epilogue group
    uint32_t slotPhase = 0, accPhase = 0;
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        if (!WaitWarp(&S.tileFull[qs], (q / kQueue) & 1, S, w.status)) return;
        const int front = __shfl_sync(~0u, S.queue[qs].t.front, 0), nst = __shfl_sync(~0u, S.queue[qs].t.nst, 0);
        if (front < 0) return;
        const bool one = ElectOne();
        if (one) umma::MbarArrive(&S.tileEmpty[qs]);
        for (int st = 0; st < nst; ++st) {
            const bool first = st % kChainStages == 0, last = st % kChainStages == kChainStages - 1 || st == nst - 1;
            if (first && !WaitWarp(&S.accEmpty[acc], accPhase, S, w.status)) return;
            if (!WaitWarp(&S.full[slot], slotPhase, S, w.status)) return;
            umma::FenceAfterSync();
            const uint32_t d = tmem + acc * C::kAccCols, aHi = tmem + C::ACol(0) + set * 2 * kAStageCols;
            const uint64_t bd = bDesc + (uint32_t)(slot * (C::kSlot >> 4));
            if (one) {
#pragma unroll
                for (int s = 0; s < 2 * kStageK / 8; ++s) {
                    umma::MmaTf32TmemA(d, aHi + 8 * s, bd + 2 * s, C::kIdescHi, s > 0 || !first ? 1u : 0u);
                    umma::MmaTf32TmemA(d, aHi + kAStageCols + 8 * s, bd + 2 * s, C::kIdescLo, 1u);
                }
                umma::CommitTo(&S.empty[slot]);
                if (last) umma::CommitTo(q & 1 ? &S.accFull[1][chain1] : &S.accFull[0][chain0]);
            }
            __syncwarp();
            if (last) {
                if (++acc == C::kAccs) { acc = 0; accPhase ^= 1; }
                int& chain = q & 1 ? chain1 : chain0;
                if (++chain == C::kAccs) chain = 0;
            }
            if (++slot == C::kSlots) { slot = 0; slotPhase ^= 1; }
            if (++set == C::kSets) set = 0;
        }
    }
}

// ------------------------------------------------------------------ epilogue

// Columns 8 h .. 8 h + 7 of the accumulator at taddr (its first half plus the
// same columns of the second half), plus those of the chain sum at tsum.
template <int NC>
__device__ __forceinline__ void LoadSums(uint32_t taddr, uint32_t tsum, bool addSum, int h, c32 (&acc)[kSub]) {
    float a[2 * kSub], b[2 * kSub];
    umma::TmemLoad16(taddr + 2 * kSub * h, a);
    umma::TmemLoad16(taddr + 2 * NC + 2 * kSub * h, b);
#pragma unroll
    for (int c = 0; c < 2 * kSub; ++c) a[c] += b[c];
    if (addSum) {
        umma::TmemLoad16(tsum + 2 * kSub * h, b);
#pragma unroll
        for (int c = 0; c < 2 * kSub; ++c) a[c] += b[c];
    }
#pragma unroll
    for (int c = 0; c < kSub; ++c) acc[c] = mk(a[2 * c], a[2 * c + 1]);
}

// 32-byte accesses of four columns (k a multiple of 4: rows of whole 32-byte
// sectors).  A lane's row is a line of its own, so every access costs a request
// of its own: with 16-byte ones the children's rows and the write-out held up
// the loads of all other roles at the wide levels (116^3, k = 16: 28.8 -> 27.2 ms
// per sweep; 96 x 96 x 76, k = 32: 18.5 -> 17.0 ms; 140^2, k = 32 solve 401 -> 376 ms).
__device__ __forceinline__ void Store4(c32* dst, const c32* v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "f"(v[0].re), "f"(v[0].im), "f"(v[1].re),
                 "f"(v[1].im), "f"(v[2].re), "f"(v[2].im), "f"(v[3].re), "f"(v[3].im)
                 : "memory");
}
__device__ __forceinline__ void Load4(c32* v, const c32* src) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0].re), "=f"(v[0].im), "=f"(v[1].re), "=f"(v[1].im), "=f"(v[2].re), "=f"(v[2].im), "=f"(v[3].re),
                   "=f"(v[3].im)
                 : "l"(src)
                 : "memory");
}

__device__ __forceinline__ void StoreRow(c32* dst, const c32 (&v)[kSub], int n, int align) {
    if (align == 4) {
#pragma unroll
        for (int j = 0; j < kSub; j += 4)
            if (j < n) Store4(dst + j, v + j);
        return;
    }
    const bool pair = align == 2;
#pragma unroll
    for (int j = 0; j < kSub; j += 2) {
        if (pair) {
            if (j < n) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j].re, v[j].im, v[j + 1].re, v[j + 1].im);
        } else {
            if (j < n) dst[j] = v[j];
            if (j + 1 < n) dst[j + 1] = v[j + 1];
        }
    }
}

// What the write-out of this thread's row needs: where it goes, the inverse
// pivot (forward pivot rows), the row's grid entries (backward; null: padding).
struct RowOut {
    c32* dst;  // column 0 of the row (null: no such row)
    z64* grid;
    c32 dinv;
    bool pivot;
};

// Writes columns col .. col + n - 1 of the row.
__device__ __forceinline__ void WriteRow(const RowOut& o, int col, int n, int align, c32 (&acc)[kSub]) {
    if (!o.dst) return;
    if (o.pivot) {
#pragma unroll
        for (int j = 0; j < kSub; ++j) acc[j] = acc[j] * o.dinv;
    }
    StoreRow(o.dst + col, acc, n, align);
}

// The same columns of the grid (+)= acc.  A grid entry is written once per
// launch, so an addition that does not return is the same as one that does.
// Two columns (32 bytes) at a time where the rows are aligned for it (`wide`): a
// lane's row is far from its neighbours', and eight-byte additions ask L2 four
// times as often.  With 16 columns per tile the loads' latency costs more than
// that (116^3: 27.6 instead of 27.2 ms); with 32 it is 16.9 instead of 17.0 ms.
__device__ __forceinline__ void WriteGrid(z64* dst, int n, bool accumulate, bool wide, const c32 (&acc)[kSub]) {
    if (wide) {
        double v[kSub][2];
#pragma unroll
        for (int j = 0; j < kSub; j += 2) {
            v[j][0] = v[j][1] = v[j + 1][0] = v[j + 1][1] = 0;
            if (accumulate && j < n)
                asm volatile("ld.global.L1::no_allocate.v4.f64 {%0,%1,%2,%3}, [%4];"
                             : "=d"(v[j][0]), "=d"(v[j][1]), "=d"(v[j + 1][0]), "=d"(v[j + 1][1]) : "l"(dst + j) : "memory");
        }
#pragma unroll
        for (int j = 0; j < kSub; j += 2)
            if (j < n)
                asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(dst + j), "d"(v[j][0] + acc[j].re),
                             "d"(v[j][1] + acc[j].im), "d"(v[j + 1][0] + acc[j + 1].re), "d"(v[j + 1][1] + acc[j + 1].im)
                             : "memory");
        return;
    }
#pragma unroll
    for (int j = 0; j < kSub; ++j) {
        if (j >= n) break;
        const z64 v = ccast<double>(acc[j]);
        if (accumulate) {
            asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(&dst[j].re), "d"(v.re) : "memory");
            asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(&dst[j].im), "d"(v.im) : "memory");
        } else {
            dst[j] = v;
        }
    }
}

__device__ __forceinline__ void StoreSums(uint32_t tsum, int h, const c32 (&acc)[kSub]) {
    float v[2 * kSub];
#pragma unroll
    for (int j = 0; j < kSub; ++j) {
        v[2 * j] = acc[j].re;
        v[2 * j + 1] = acc[j].im;
    }
    umma::TmemStore16(tsum + 2 * kSub * h, v);
}

// Waits (bounded) for the fronts that a tile reads.  Two lanes acquire a counter
// each, and the warp barrier orders the other lanes' loads after that: the registers
// of this role are all taken, and with both counters acquired by every lane, as
// the loaders do it, a 220 x 220 x 48 sweep took 43.0 instead of 42.6 ms at k = 32.
__device__ __forceinline__ bool WaitCarry(const FlowTile& t, Sync& S, const FlowWork& w) {
    const int lane = threadIdx.x & 31, need = lane == 0 ? t.need0 : lane == 1 ? t.need1 : 0;
    bool ok = true;
    if (need > 0) {
        const int* const count = w.done + t.dep + lane;
        ok = WaitUntil([&] { return LoadAcquire(count) >= need; }, S, w.status);
    }
    ok = __all_sync(~0u, ok);
    __syncwarp();
    return ok;
}

template <int NC>
__device__ void EpilogueRole(int k, Sync& S, z64* B, const PanelIO& io, const FlowWork& w) {
    using C = Cfg<NC>;
    const int group = threadIdx.x / kEpiThreads, row = threadIdx.x % kEpiThreads, lane = threadIdx.x & 31;
    const int bar = group ? 4 : 1;  // this group's named barrier
    PdlWait();  // carries, split-K scratch and outputs are shared with the preceding kernels
    if (group == 0)
        for (int q = 0; q < C::kAccs; ++q) umma::MbarArrive(&S.accEmpty[q]);  // every accumulator starts free
    const uint32_t lanes = (uint32_t)(row & ~31) << 16;
    const uint32_t tsum = S.tmem + C::kSumCol + group * 2 * NC + lanes;
    const bool pair = (k & 1) == 0, accumulate = io.outAccumulate;
    const int align = k % 4 == 0 ? 4 : pair ? 2 : 1;  // columns of an aligned access
    const bool wide = NC == 32 && pair && io.ldk % 2 == 0 && (reinterpret_cast<uintptr_t>(B) & 31) == 0;
    int c = 0, own = 0;  // chains of all tiles, and of this group's
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        bool ok = WaitWarp(&S.tileFull[qs], (q / kQueue) & 1, S, w.status);
        // every thread of a group takes the same branches (they share named barriers)
        if (umma::NamedBarrierOr(bar, kEpiThreads, !ok)) return;
        const FlowTile& t = S.queue[qs].t;
        if (t.front < 0) return;
        const int nch = NumChains(t.nst), nsplit = t.nsplit, col0 = t.col0, ncol = min(NC, k - t.col0);
        if ((q & 1) != group) {
            c += nch;
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.tileEmpty[qs]);
            continue;
        }
        RowOut o;
        bool carried = false;  // the chain sum starts from the children's updates
        {
            const FlowFront<float>& f = S.queue[qs].f;
            const int r = t.row0 + row, s = f.s;
            o.dst = nullptr;
            o.grid = nullptr;
            o.pivot = false;
            o.dinv = mk(1.f, 0.f);
            if (t.bwd) {
                if (r < s) {
                    o.dst = static_cast<c32*>(w.x) + (int64_t)(f.ndOff + r) * k;
                    const int at = NaturalRow(io, f.ndOff + r);
                    if (at >= 0) o.grid = B + (int64_t)at * io.ldk;
                }
            } else if (r < s) {
                o.dst = static_cast<c32*>(w.w) + (int64_t)(f.ndOff + r) * k;
                o.pivot = true;
                o.dinv = cinv(f.D[r]);
            } else if (r < s + f.u) {
                o.dst = f.Pp + (int64_t)__ldg(f.rel + r - s) * k;
            }
            if (t.carry) {  // into the sum while the tile's stages run
                ok = WaitCarry(t, S, w);
                if (ok) {
                    const bool in = r >= s && r < s + f.u;
                    const c32* c0 = in && f.P0 ? f.P0 + (int64_t)r * k + col0 : nullptr;
                    const c32* c1 = in && f.P1 ? f.P1 + (int64_t)r * k + col0 : nullptr;
#pragma unroll 1
                    for (int h = 0; h < NC / kSub; ++h) {
                        c32 v[kSub];
                        if (align == 4) {
                            c32 a[kSub], b[kSub];
#pragma unroll
                            for (int j = 0; j < kSub; ++j) a[j] = b[j] = mk(0.f, 0.f);
#pragma unroll
                            for (int j = 0; j < kSub; j += 4) {
                                const int n = h * kSub + j;
                                if (c0 && n < ncol) Load4(a + j, c0 + n);
                                if (c1 && n < ncol) Load4(b + j, c1 + n);
                            }
#pragma unroll
                            for (int j = 0; j < kSub; ++j) v[j] = a[j] + b[j];
                        } else {
                            Unit<float, 2> a[kSub / 2], b[kSub / 2];
#pragma unroll
                            for (int j = 0; j < kSub / 2; ++j) {
                                const int n = h * kSub + 2 * j;
                                a[j] = b[j] = ZeroUnit<float, 2>();
                                if (c0 && n < ncol) LoadUnit<float, 2>(a[j], c0 + n, pair, n + 1 < ncol);
                                if (c1 && n < ncol) LoadUnit<float, 2>(b[j], c1 + n, pair, n + 1 < ncol);
                            }
#pragma unroll
                            for (int j = 0; j < kSub; ++j) v[j] = a[j / 2].z[j % 2] + b[j / 2].z[j % 2];
                        }
                        StoreSums(tsum, h, v);
                    }
                    umma::TmemStoreWait();
                    carried = true;
                }
            }
        }
        for (int ch = 0; ch + 1 < nch; ++ch, ++c, ++own) {
            const int b = c % C::kAccs;
            ok = ok && WaitWarp(&S.accFull[group][own % C::kAccs], (own / C::kAccs) & 1, S, w.status);
            if (umma::NamedBarrierOr(bar, kEpiThreads, !ok)) return;
            umma::FenceAfterSync();
            const uint32_t taddr = S.tmem + b * C::kAccCols + lanes;
#pragma unroll 2
            for (int h = 0; h < NC / kSub; ++h) {
                c32 acc[kSub];
                LoadSums<NC>(taddr, tsum, ch > 0 || carried, h, acc);
                StoreSums(tsum, h, acc);
            }
            umma::TmemStoreWait();
            umma::FenceBeforeSync();
            umma::MbarArrive(&S.accEmpty[b]);
        }
        const int b = c % C::kAccs;
        ok = ok && WaitWarp(&S.accFull[group][own % C::kAccs], (own / C::kAccs) & 1, S, w.status);
        ++c;
        ++own;
        if (umma::NamedBarrierOr(bar, kEpiThreads, !ok)) return;
        umma::FenceAfterSync();
        const uint32_t taddr = S.tmem + b * C::kAccCols + lanes;
        // A split tile: partials [slot][column pair][row], summed in split order
        // by the last CTA to arrive.
        float4* const part = static_cast<float4*>(w.partials) + row;
        const bool bwd = t.bwd;
        bool finish = true;
#pragma unroll 1
        for (int h = 0; h < NC / kSub; ++h) {
            c32 acc[kSub];
            LoadSums<NC>(taddr, tsum, nch > 1 || carried, h, acc);
            if (bwd && nsplit == 1) StoreSums(tsum, h, acc);  // for the grid, below
            if (h == NC / kSub - 1) {
                umma::FenceBeforeSync();
                umma::MbarArrive(&S.accEmpty[b]);
            }
            if (h * kSub >= ncol) continue;
            if (nsplit > 1) {
                float4* mine = part + ((int64_t)(t.slot + t.split) * NC + h * kSub) / 2 * kRows;
#pragma unroll
                for (int n = 0; n < kSub; n += 2)
                    mine[n / 2 * kRows] = make_float4(acc[n].re, acc[n].im, acc[n + 1].re, acc[n + 1].im);
            } else {
                WriteRow(o, col0 + h * kSub, ncol - h * kSub, align, acc);
            }
        }
        if (nsplit > 1) {
            umma::NamedBarrier(bar, kEpiThreads);
            if (row == 0) {
                int before;
                asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;"
                             : "=r"(before) : "l"(w.counters + t.counter) : "memory");
                S.isLast[group] = before == nsplit - 1;
                if (before == nsplit - 1) w.counters[t.counter] = 0;  // ready for the next launch
            }
            umma::NamedBarrier(bar, kEpiThreads);
            finish = S.isLast[group];
            if (finish) {
#pragma unroll 1
                for (int h = 0; h * kSub < ncol; ++h) {
                    c32 acc[kSub];
#pragma unroll
                    for (int n = 0; n < kSub; ++n) acc[n] = mk(0.f, 0.f);
                    const float4* p = part + ((int64_t)t.slot * NC + h * kSub) / 2 * kRows;
                    constexpr int kFly = 2;  // splits in flight
                    for (int s = 0; s < nsplit; s += kFly, p += kFly * NC / 2 * kRows) {
                        float4 v[kFly][kSub / 2];
#pragma unroll
                        for (int f = 0; f < kFly; ++f)
#pragma unroll
                            for (int n = 0; n < kSub / 2; ++n)
                                v[f][n] = s + f < nsplit ? __ldcg(p + (f * NC / 2 + n) * kRows) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int f = 0; f < kFly; ++f)
#pragma unroll
                            for (int n = 0; n < kSub / 2; ++n) {
                                acc[2 * n] += mk(v[f][n].x, v[f][n].y);
                                acc[2 * n + 1] += mk(v[f][n].z, v[f][n].w);
                            }
                    }
                    if (bwd) StoreSums(tsum, h, acc);
                    WriteRow(o, col0 + h * kSub, ncol - h * kSub, align, acc);
                }
            }
        }
        umma::NamedBarrier(bar, kEpiThreads);
        if (finish && row == 0) AddRelease(w.done + t.signal);
        if (bwd && finish) {  // nothing in this launch reads the grid: after the release
            __syncwarp();
            umma::TmemStoreWait();
#pragma unroll 1
            for (int h = 0; h * kSub < ncol; ++h) {
                float a[2 * kSub];
                umma::TmemLoad16(tsum + 2 * kSub * h, a);
                c32 acc[kSub];
#pragma unroll
                for (int j = 0; j < kSub; ++j) acc[j] = mk(a[2 * j], a[2 * j + 1]);
                if (o.grid) WriteGrid(o.grid + col0 + h * kSub, ncol - h * kSub, accumulate, wide, acc);
            }
        }
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.tileEmpty[qs]);
    }
}

// ------------------------------------------------------------------ kernel

template <int NC>
__global__ void __launch_bounds__(kTcThreads, 1) sweep_flow_tc_kernel(const FlowFront<float>* __restrict__ fr,
                                                                      const FlowTile* __restrict__ tiles, int n, int k,
                                                                      z64* __restrict__ B,
                                                                      const __grid_constant__ PanelIO io,
                                                                      const __grid_constant__ FlowWork w) {
    using C = Cfg<NC>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ Sync S;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < C::kSlots; ++i) {
            umma::MbarInit(&S.tma[i], 1);
            umma::MbarInit(&S.full[i], kLoadGroupWarps + kGroupWarps);
            umma::MbarInit(&S.empty[i], 1);
        }
        for (int i = 0; i < C::kAccs; ++i) {
            for (int e = 0; e < kEpiGroups; ++e) umma::MbarInit(&S.accFull[e][i], 1);
            umma::MbarInit(&S.accEmpty[i], kEpiThreads);
        }
        for (int i = 0; i < kQueue; ++i) {
            umma::MbarInit(&S.tileFull[i], 1);
            umma::MbarInit(&S.tileEmpty[i], kReaders);
        }
        umma::MbarInit(&S.mmaDrain, 1);
        S.abort = 0;
        S.issued = 0;
        umma::FenceMbarInit();
    }
    if (tid / 32 == 0) umma::TmemAlloc(&S.tmem, kTmemCols);
    umma::FenceBeforeSync();
    __syncthreads();
    umma::FenceAfterSync();
    if (tid < kConv0) EpilogueRole<NC>(k, S, B, io, w);
    else if (tid < kLoad0) ConverterRole<NC>(smem, S, w);
    else if (tid < kMma0) LoaderRole<NC>(k, smem, S, w);
    else if (tid < kProd0) MmaRole<NC>(smem, S, w);
    else ProducerRole<NC>(fr, tiles, n, smem, S, w);
    umma::FenceBeforeSync();
    __syncthreads();
    // Every role has returned.  When one gave up, the others may have left
    // asynchronous work behind: it is waited for (bounded) before tensor memory
    // is freed.  S.abort is no longer written, so every thread takes the same
    // branch.
    if (*reinterpret_cast<volatile int*>(&S.abort)) {
        if (tid / 32 == kMma0 / 32) {  // the lane that issued
            if (ElectOne()) umma::CommitTo(&S.mmaDrain);
            umma::MbarWaitBounded(&S.mmaDrain, 0, nullptr);
        }
        if (tid == kProd0) DrainCopies<C::kSlots>(S);
        umma::FenceBeforeSync();
        __syncthreads();
    }
    if (tid / 32 == 0) {
        umma::FenceAfterSync();
        umma::TmemDealloc(S.tmem, kTmemCols);
    }
    LeaveFlow(w, &S.lastCta);
}

int g_tcSMs = 0;

}  // namespace

int FlowTcSlots() { return g_tcSMs; }

void PrepareFlowTcKernels() {
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    CUDA_CHECK(cudaDeviceGetAttribute(&g_tcSMs, cudaDevAttrMultiProcessorCount, dev));
    CUDA_CHECK(cudaFuncSetAttribute(sweep_flow_tc_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)Cfg<16>::kSmem));
    CUDA_CHECK(cudaFuncSetAttribute(sweep_flow_tc_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)Cfg<32>::kSmem));
}

void LaunchFlowTc(const FlowFront<float>* fr, const FlowTile* tiles, int n, int k, int cols, z64* B, const PanelIO& io,
                  const FlowWork& w, cudaStream_t st) {
    if (n <= 0) return;
    const dim3 grid(std::min(n, g_tcSMs));
    if (cols == 32)
        LaunchPdl(sweep_flow_tc_kernel<32>, grid, dim3(kTcThreads), Cfg<32>::kSmem, st, fr, tiles, n, k, B, io, w);
    else
        LaunchPdl(sweep_flow_tc_kernel<16>, grid, dim3(kTcThreads), Cfg<16>::kSmem, st, fr, tiles, n, k, B, io, w);
}

}  // namespace psp_b200
