// One panel solve of the sweep (cliq::Solve replacement) on the selectively
// inverted factors G = [inv(L11); -L21 inv(L11)], as one launch that walks
// the whole elimination tree:
//
//   forward, per front   [Y; U] = G R_s + [0; R_u],   W = inv(D) Y
//   backward, per front  X_s = G^T [W; X_u]
//
// The tree has about twice log2(nx ny / cutoff) dependent levels, and one
// panel's factors are read in ~70 us per direction at HBM speed, so a launch
// per level spends most of its time filling and draining.  Here every level
// of both directions is in one list of tiles (rows x K-chunk of one front),
// ordered so that a tile only depends on tiles before it.  CTAs take tiles
// from that list by an atomic ticket and stream them through one ring of
// stages: the factors do not depend on the solve, so the copies of the next
// tiles run ahead across level boundaries while their right-hand sides are
// still being computed elsewhere.  A tile's right-hand sides wait for the
// fronts it reads (children forward, the parent backward) on per-front
// counters of finished tiles.
//
// Progress: a ticket is only taken by a running CTA, and CTAs work on theirs
// in order, so the lowest unfinished tile never waits for one that has not
// been started: no assumption that all CTAs are resident at the same time.
// Every wait is bounded (umma::kWaitLimitNs); one that runs out sets bit 2 of
// the status word and ends the CTA's roles.
//
// Roles of a CTA (256 threads, two CTAs per SM):
//   producer (1 warp)   takes tickets and issues one tiled TMA copy of G per
//                       stage: forward kStageK columns of kRows rows, backward
//                       kRows columns of kStageK rows (128-byte swizzled, so
//                       that lanes of different columns read different banks)
//   loaders (3 warps)   right-hand sides, a chunk of several stages at a time:
//                       forward the panel's own entries plus the planes that
//                       the front's two children write their updates to
//                       (rows no child writes stay zero), backward W or the
//                       ancestors' solution; at the end of a forward tile the
//                       same planes for its update rows (a carry chunk); and
//                       what the tile's write-out needs per row
//   compute (4 warps)   register tiles of RPT x CPT complex sums on the FP32
//                       (packed fma.f32x2) or FP64 pipes; a split-K tile's last
//                       CTA sums the partials in split order, so results do
//                       not depend on which CTA ran what.
// Column counts are 1, 2, 4, 8, 16 or 32 per tile.
//
// What bounds it: the chain of levels.  A tile of six stages takes about 6 us
// from the release of what it waits for to its own (first right-hand sides
// 0.8 us, stages 2.3, sum over the K groups and splits 2, write and release 1),
// twice per level and direction.  Stages and tiles hold 16 KB so that two CTAs
// of five slots fit on an SM.  Measured against one launch per level and
// direction with gathers between (sweeps of the whole preconditioner): FP64
// 57 x 53 x 61, k = 5: 12.8 -> 6.8 ms (0.74 TB/s of factors); complex single
// 75 x 67 x 58, k = 1: 8.4 -> 3.5 ms; 96 x 96 x 76, k = 1: 18.9 -> 7.5 ms
// (2.8 TB/s).
#include <algorithm>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "sweep_flow.cuh"

namespace psp_b200 {

namespace {

using namespace flow;

constexpr int kComputeWarps = 4, kLoadWarps = 3;
constexpr int kComputeThreads = 32 * kComputeWarps;
constexpr int kLoadThreads = 32 * kLoadWarps;
constexpr int kLoad0 = kComputeThreads;
constexpr int kProd0 = kLoad0 + kLoadThreads;
constexpr int kThreads = kProd0 + 32;
constexpr int kStageK = kFlowStageK;
constexpr uint32_t kGBytes = 16384;   // one stage of G
constexpr int kQueue = 3;             // tiles in flight between the roles
constexpr int kMaxSlots = 6, kMaxChunks = 3;

template <typename R, int NC>
struct Cfg {
    static constexpr int kRows = FlowRows<R>();              // rows of a tile
    static constexpr int RPT = kRows / 32;                   // rows per thread
    static constexpr int CPT = NC >= 32 ? 8 : NC >= 4 ? 4 : NC;
    static constexpr int CG = NC / CPT, RG = 32 / CG;        // lanes along columns and rows
    static constexpr int kWarpRows = RG * RPT;
    static constexpr int RW = kRows / kWarpRows;             // warps along rows
    static constexpr int KG = kComputeWarps / RW;            // warp groups along K
    static constexpr int KPG = kStageK / KG;
    // right-hand sides: chunks of CH stages, 16 bytes per entry
    static constexpr int CH = NC >= 32 ? 2 : NC >= 16 ? 4 : 8;
    static constexpr int kChunks = NC >= 8 ? 2 : 3;
    static constexpr uint32_t kChunkBytes = CH * kStageK * NC * 16;
    static constexpr int kCarryRows = kChunkBytes / (NC * sizeof(cpx<R>)) < kRows ? kChunkBytes / (NC * sizeof(cpx<R>)) : kRows;
    static constexpr int kCarry = kRows / kCarryRows;        // carry chunks of a tile
    static constexpr int V = sizeof(R) == 4 && NC > 1 ? 2 : 1;   // columns per 16-byte load
    static constexpr uint32_t kRed = KG > 1 ? (KG - 1) * RW * 32 * RPT * CPT * sizeof(cpx<R>) : 0;
    static constexpr int kSlotsFit = (int)((106 * 1024 - kChunks * kChunkBytes - kRed) / kGBytes);
    static constexpr int kSlots = kSlotsFit > kMaxSlots ? kMaxSlots : kSlotsFit;
    static constexpr uint32_t kRhsOff = kSlots * kGBytes, kRedOff = kRhsOff + kChunks * kChunkBytes;
    static constexpr size_t kSmem = kRedOff + kRed + 1024;
    static_assert(RW * KG == kComputeWarps && RW >= 1 && KG >= 1, "warp grid");
    static_assert(kSlots >= 3 && kChunks <= kMaxChunks, "rings");
};

template <typename R>
struct Sync {
    TileCtx<R> queue[kQueue];
    // per tile row: inverse pivot (pivot rows, forward); and the row of the
    // parent's plane (update rows, forward) or the grid point (backward; -1: padding)
    cpx<R> dinv[kQueue][FlowRows<R>()];
    int idx[kQueue][FlowRows<R>()];
    uint64_t tma[kMaxSlots], empty[kMaxSlots];
    uint64_t rhs[kMaxChunks], rhsEmpty[kMaxChunks];
    uint64_t tileFull[kQueue], tileEmpty[kQueue];
    int abort, isLast, lastCta, issued;
};

// A right-hand-side entry in a chunk: complex single as (re, re, im, im), the
// two packed multiplicands of a complex product; complex double as stored.
__device__ __forceinline__ void StoreRhs(unsigned char* rhs, int e, c32 v) {
    *reinterpret_cast<float4*>(rhs + e * 16) = make_float4(v.re, v.re, v.im, v.im);
}
__device__ __forceinline__ void StoreRhs(unsigned char* rhs, int e, z64 v) {
    *reinterpret_cast<double2*>(rhs + e * 16) = make_double2(v.re, v.im);
}

// ------------------------------------------------------------------ producer

template <typename R, int NC>
__device__ void ProducerRole(const FlowFront<R>* __restrict__ fr, const FlowTile* __restrict__ tiles, int n,
                             unsigned char* smem, Sync<R>& S, const FlowWork& w) {
    using C = Cfg<R, NC>;
    const int lane = threadIdx.x & 31;
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    TileSource<R> src(fr, tiles, n, w.ctrl);
    int g = 0;
    bool ok = true;
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
        for (int st = 0; st < nst; ++st, ++g) {
            const int slot = g % C::kSlots;
            ok = g < C::kSlots || WaitWarp(&S.empty[slot], ((g / C::kSlots) - 1) & 1, S, w.status);
            if (!ok) break;
            if (lane == 0) {
                unsigned char* dst = smem + slot * kGBytes;
                const int kBase = t.k0 + st * kStageK;
                umma::MbarArriveExpectTx(&S.tma[slot], kGBytes);
                if (!t.bwd) {
                    TmaLoadStream(dst, map, (int)(sizeof(R) / 4) * t.row0, kBase, &S.tma[slot], policy);
                } else if (sizeof(R) == 4) {
                    TmaLoadStream(dst, map, kBase, t.row0, &S.tma[slot], policy);
                } else {  // two swizzled halves of 8 complex doubles
                    TmaLoadStream(dst, map, 2 * kBase, t.row0, &S.tma[slot], policy);
                    TmaLoadStream(dst + kGBytes / 2, map, 2 * kBase + kStageK, t.row0, &S.tma[slot], policy);
                }
            }
            __syncwarp();
        }
        if (!ok) break;
        src.Take();
    }
    if (lane == 0) S.issued = g;  // read after all roles have returned
}

// ------------------------------------------------------------------ loaders

template <typename R, int NC>
__device__ void LoaderRole(int k, unsigned char* smem, Sync<R>& S, const PanelIO& io, const FlowWork& w) {
    using C = Cfg<R, NC>;
    constexpr int V = C::V, kUnitsRow = NC / V;
    constexpr int kUnits = C::CH * kStageK * kUnitsRow, kPer = (kUnits + kLoadThreads - 1) / kLoadThreads;
    constexpr int kBatch = kPer < 6 ? kPer : 6;
    constexpr int kCarryUnits = C::kCarryRows * kUnitsRow;
    const int lt = threadIdx.x - kLoad0, lane = threadIdx.x & 31;
    const cpx<R>* rnd = static_cast<const cpx<R>*>(w.rnd);
    const cpx<R>* W = static_cast<const cpx<R>*>(w.w);
    const cpx<R>* X = static_cast<const cpx<R>*>(w.x);
    const bool pair = (k & 1) == 0;
    PdlWait();     // right-hand sides come from the preceding kernels
    PdlTrigger();
    int gc = 0;    // chunks filled
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        if (!WaitWarp(&S.tileFull[qs], (q / kQueue) & 1, S, w.status)) return;
        const FlowTile t = S.queue[qs].t;
        if (t.front < 0) return;
        const FlowFront<R> f = S.queue[qs].f;
        // what does not depend on the solve comes before the wait
        for (int i = lt; i < C::kRows; i += kLoadThreads) {
            const int r = t.row0 + i;
            int id = 0;
            if (t.bwd) {
                if (r < f.s) id = NaturalRow(io, f.ndOff + r);
            } else if (r < f.s) {
                S.dinv[qs][i] = cinv(f.D[r]);
            } else if (r < f.s + f.u) {
                id = __ldg(f.rel + r - f.s);
            }
            S.idx[qs][i] = id;
        }
        const int ncol = min(NC, k - t.col0);
        bool waited = false;
        const int rows = t.nst * kStageK;
        for (int c0 = 0; c0 < rows; c0 += C::CH * kStageK, ++gc) {
            const int cb = gc % C::kChunks;
            unsigned char* rhs = smem + C::kRhsOff + cb * C::kChunkBytes;
#pragma unroll 1
            for (int b0 = 0; b0 < kPer; b0 += kBatch) {
                int at[kBatch];  // backward: solution row of entries below the pivots
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int row = c0 + (lt + (b0 + i) * kLoadThreads) / kUnitsRow, kk = t.k0 + row;
                    at[i] = t.bwd && row < rows && kk >= f.s && kk < t.ke ? __ldg(f.lower + kk - f.s) : f.ndOff + kk;
                }
                if (!waited) {
                    if (!TileReady(t, true, S, w)) return;
                    waited = true;
                }
                Unit<R, V> v[kBatch], p0[kBatch], p1[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int e = lt + (b0 + i) * kLoadThreads;
                    const int row = c0 + e / kUnitsRow, col = (e % kUnitsRow) * V, kk = t.k0 + row;
                    v[i] = p0[i] = p1[i] = ZeroUnit<R, V>();
                    if (e < kUnits && kk < t.ke && row < rows && col < ncol) {
                        const bool both = col + 1 < ncol;
                        const int c = t.col0 + col;
                        const cpx<R>* src = t.bwd ? (kk < f.s ? W : X) : rnd;
                        LoadUnit<R, V>(v[i], src + (int64_t)at[i] * k + c, pair, both);
                        if (!t.bwd) {
                            if (f.P0) LoadUnit<R, V>(p0[i], f.P0 + (int64_t)kk * k + c, pair, both);
                            if (f.P1) LoadUnit<R, V>(p1[i], f.P1 + (int64_t)kk * k + c, pair, both);
                        }
                    }
                }
                if (b0 == 0 && gc >= C::kChunks &&
                    !WaitWarp(&S.rhsEmpty[cb], ((gc / C::kChunks) - 1) & 1, S, w.status)) return;
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int e = lt + (b0 + i) * kLoadThreads;
                    if (e < kUnits) {
#pragma unroll
                        for (int h = 0; h < V; ++h) StoreRhs(rhs, e * V + h, v[i].z[h] + p0[i].z[h] + p1[i].z[h]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.rhs[cb]);
        }
        for (int cs = 0; cs < t.carry; ++cs, ++gc) {
            const int cb = gc % C::kChunks;
            cpx<R>* dst = reinterpret_cast<cpx<R>*>(smem + C::kRhsOff + cb * C::kChunkBytes);
            if (gc >= C::kChunks && !WaitWarp(&S.rhsEmpty[cb], ((gc / C::kChunks) - 1) & 1, S, w.status)) return;
#pragma unroll 1
            for (int e0 = lt; e0 < kCarryUnits; e0 += kBatch * kLoadThreads) {
                Unit<R, V> p0[kBatch], p1[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int e = e0 + i * kLoadThreads;
                    const int r = t.row0 + cs * C::kCarryRows + e / kUnitsRow, col = (e % kUnitsRow) * V;
                    p0[i] = p1[i] = ZeroUnit<R, V>();
                    if (e < kCarryUnits && r >= f.s && r < f.s + f.u && col < ncol) {
                        const bool both = col + 1 < ncol;
                        const int64_t o = (int64_t)r * k + t.col0 + col;
                        if (f.P0) LoadUnit<R, V>(p0[i], f.P0 + o, pair, both);
                        if (f.P1) LoadUnit<R, V>(p1[i], f.P1 + o, pair, both);
                    }
                }
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int e = e0 + i * kLoadThreads;
                    if (e < kCarryUnits) {
#pragma unroll
                        for (int h = 0; h < V; ++h) dst[e * V + h] = p0[i].z[h] + p1[i].z[h];
                    }
                }
            }
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.rhs[cb]);
        }
        __syncwarp();
        if (lane == 0) umma::MbarArrive(&S.tileEmpty[qs]);
    }
}

// ------------------------------------------------------------------ compute

typedef unsigned long long u64;

__device__ __forceinline__ void Fma2(u64& d, u64 a, u64 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// (re, im) -> (-im, re)
__device__ __forceinline__ u64 Rot(u64 a) {
    u64 r;
    asm("{\n\t.reg .f32 x, y;\n\tmov.b64 {x, y}, %1;\n\tneg.f32 y, y;\n\tmov.b64 %0, {y, x};\n\t}" : "=l"(r) : "l"(a));
    return r;
}
__device__ __forceinline__ ulonglong2 Lds128(const unsigned char* p) {
    return *reinterpret_cast<const ulonglong2*>(p);
}

// Complex accumulators of a thread: packed (re, im) singles, or doubles.
template <typename R> struct Acc;
template <> struct Acc<float> {
    u64 v;
    __device__ __forceinline__ c32 Get() const {
        return mk(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
    }
    __device__ __forceinline__ void Set(c32 z) {
        v = (u64)__float_as_uint(z.re) | ((u64)__float_as_uint(z.im) << 32);
    }
};
template <> struct Acc<double> {
    z64 v;
    __device__ __forceinline__ z64 Get() const { return v; }
    __device__ __forceinline__ void Set(z64 z) { v = z; }
};

// Row of thread row i inside its warp's rows.
template <typename R, int NC, bool kBwd>
__device__ __forceinline__ int RowIn(int i, int rg) {
    using C = Cfg<R, NC>;
    if (!kBwd && sizeof(R) == 4) return (i >> 1) * 2 * C::RG + 2 * rg + (i & 1);
    return i * C::RG + rg;
}

// One K column: acc[i][j] += x[i] b_j, y[i] the rotated x[i].  The two products
// of one sum are kept apart: an FMA pair that depends on itself stalls.
template <int NC>
__device__ __forceinline__ void Products(const unsigned char* rhs, const u64 (&x)[4], const u64 (&y)[4],
                                         Acc<float> (&acc)[Cfg<float, NC>::RPT][Cfg<float, NC>::CPT]) {
    using C = Cfg<float, NC>;
    constexpr int J = C::CPT < 4 ? C::CPT : 4;
#pragma unroll
    for (int j0 = 0; j0 < C::CPT; j0 += J) {
        ulonglong2 b[J];
#pragma unroll
        for (int j = 0; j < J; ++j) b[j] = Lds128(rhs + (j0 + j) * C::CG * 16);
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) Fma2(acc[i][j0 + j].v, x[i], b[j].x);
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) Fma2(acc[i][j0 + j].v, y[i], b[j].y);
    }
}

// acc += this thread's rows and columns of one stage; wrow: first row of the
// warp inside the tile, kb: first K column of the warp's group.
template <int NC, bool kBwd>
__device__ __forceinline__ void StageProduct(const unsigned char* slot, const unsigned char* rhs, int wrow, int kb, int rg,
                                             int cg, Acc<float> (&acc)[Cfg<float, NC>::RPT][Cfg<float, NC>::CPT]) {
    using C = Cfg<float, NC>;
    rhs += cg * 16;
    if (!kBwd) {
        const unsigned char* a = slot + (wrow + 2 * rg) * 8;
#pragma unroll(C::KPG <= 4 ? 4 : 2)
        for (int kc = kb; kc < kb + C::KPG; ++kc) {
            u64 x[4], y[4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const ulonglong2 v = Lds128(a + kc * (C::kRows * 8) + p * 2 * C::RG * 8);
                x[2 * p] = v.x;
                x[2 * p + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = Rot(x[i]);
            Products<NC>(rhs + kc * NC * 16, x, y, acc);
        }
    } else {
        const int sw = (wrow + rg) & 7;
#pragma unroll(C::KPG <= 4 ? 2 : 1)
        for (int kc = kb; kc < kb + C::KPG; kc += 2) {
            ulonglong2 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                x[i] = Lds128(slot + (wrow + i * C::RG + rg) * 128 +
                              (((kc >> 1) ^ (C::RG >= 8 ? sw : ((sw + i * C::RG) & 7))) * 16));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                u64 a[4], y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] = h ? x[i].y : x[i].x;
                    y[i] = Rot(a[i]);
                }
                Products<NC>(rhs + (kc + h) * NC * 16, a, y, acc);
            }
        }
    }
}

template <int NC, bool kBwd>
__device__ __forceinline__ void StageProduct(const unsigned char* slot, const unsigned char* rhs, int wrow, int kb, int rg,
                                             int cg, Acc<double> (&acc)[Cfg<double, NC>::RPT][Cfg<double, NC>::CPT]) {
    using C = Cfg<double, NC>;
    rhs += cg * 16;
#pragma unroll(C::KPG <= 4 ? 4 : 2)
    for (int kc = kb; kc < kb + C::KPG; ++kc) {
        z64 x[C::RPT];
#pragma unroll
        for (int i = 0; i < C::RPT; ++i) {
            const int row = wrow + i * C::RG + rg;
            const unsigned char* p = kBwd ? slot + (kc >> 3) * (kGBytes / 2) + row * 128 + (((kc & 7) ^ (row & 7)) * 16)
                                          : slot + kc * (C::kRows * 16) + row * 16;
            x[i] = *reinterpret_cast<const z64*>(p);
        }
        constexpr int J = C::CPT < 4 ? C::CPT : 4;
#pragma unroll
        for (int j0 = 0; j0 < C::CPT; j0 += J) {
            z64 b[J];
#pragma unroll
            for (int j = 0; j < J; ++j) b[j] = *reinterpret_cast<const z64*>(rhs + (kc * NC + (j0 + j) * C::CG) * 16);
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int i = 0; i < C::RPT; ++i) {
                    z64& a = acc[i][j0 + j].v;
                    a.re = fma(x[i].re, b[j].re, a.re);
                    a.im = fma(x[i].re, b[j].im, a.im);
                }
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int i = 0; i < C::RPT; ++i) {
                    z64& a = acc[i][j0 + j].v;
                    a.re = fma(-x[i].im, b[j].im, a.re);
                    a.im = fma(x[i].im, b[j].re, a.im);
                }
        }
    }
}

// Writes the finished sums of a tile (compute threads of K group 0).
template <typename R, int NC, bool kBwd>
__device__ __forceinline__ void StoreTile(const FlowTile& t, const FlowFront<R>& f, const cpx<R>* dinv, const int* idx,
                                          int k, int wrow, int rg, int cg,
                                          const Acc<R> (&acc)[Cfg<R, NC>::RPT][Cfg<R, NC>::CPT],
                                          const FlowWork& w) {
    using C = Cfg<R, NC>;
    const int left = (kBwd ? f.s : f.s + f.u) - t.row0, pivots = f.s - t.row0, col0 = t.col0 + cg;
    cpx<R>* const own = static_cast<cpx<R>*>(kBwd ? w.x : w.w) + (int64_t)(f.ndOff + t.row0) * k;
    cpx<R>* const Pp = f.Pp;
#pragma unroll
    for (int i = 0; i < C::RPT; ++i) {
        const int row = wrow + RowIn<R, NC, kBwd>(i, rg);
        const bool pivot = kBwd || row < pivots;
        cpx<R>* dst = pivot ? own + row * k : Pp + (int64_t)idx[row] * k;
        const cpx<R> d = !kBwd && pivot ? dinv[row] : mk<R>(1, 0);
#pragma unroll
        for (int j = 0; j < C::CPT; ++j) {
            const cpx<R> v = acc[i][j].Get();
            if (row < left && col0 + j * C::CG < k) dst[col0 + j * C::CG] = !kBwd && pivot ? v * d : v;
        }
    }
}

// The grid's entries of a backward tile, after the solution that other tiles
// wait for has been released.  An entry is written once per launch, so an
// addition that does not return is the same as one that does; loaded, added to
// and stored before the release they made each backward level 1 us longer.
template <typename R, int NC>
__device__ __forceinline__ void StoreGrid(const FlowTile& t, const FlowFront<R>& f, const int* idx, int k, int wrow, int rg,
                                          int cg, const Acc<R> (&acc)[Cfg<R, NC>::RPT][Cfg<R, NC>::CPT], z64* B,
                                          const PanelIO& io) {
    using C = Cfg<R, NC>;
    const int left = f.s - t.row0, col0 = t.col0 + cg;
    const bool accumulate = io.outAccumulate;
    const int64_t ldk = io.ldk;
#pragma unroll
    for (int i = 0; i < C::RPT; ++i) {
        const int row = wrow + RowIn<R, NC, true>(i, rg);
        const int at = row < left ? idx[row] : -1;
        z64* const dst = B + at * ldk;
#pragma unroll
        for (int j = 0; j < C::CPT; ++j) {
            const int col = col0 + j * C::CG;
            if (at < 0 || col >= k) continue;
            const z64 v = ccast<double>(acc[i][j].Get());
            if (accumulate) {
                asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(&dst[col].re), "d"(v.re) : "memory");
                asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(&dst[col].im), "d"(v.im) : "memory");
            } else {
                dst[col] = v;
            }
        }
    }
}

// One tile: its stages (g: stages consumed so far, gc: chunks), the sum over
// the K groups and splits, and the write-out.
template <typename R, int NC, bool kBwd>
__device__ __forceinline__ bool ComputeTile(const FlowTile& t, const FlowFront<R>& f, int qs, int k, int& g, int& gc,
                                            unsigned char* smem, Sync<R>& S, z64* B, const PanelIO& io,
                                            const FlowWork& w) {
    using C = Cfg<R, NC>;
    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int rg = lane / C::CG, cg = lane % C::CG;
    const int kg = warp / C::RW, wrow = (warp % C::RW) * C::kWarpRows;
    const int M = kBwd ? f.s : f.s + f.u;
    Acc<R> acc[C::RPT][C::CPT];
#pragma unroll
    for (int i = 0; i < C::RPT; ++i)
#pragma unroll
        for (int j = 0; j < C::CPT; ++j) acc[i][j].Set(mk<R>(0, 0));
    const int r0 = t.row0 + wrow, r1 = r0 + C::kWarpRows - 1;
    bool ok = true;
    for (int s0 = 0; ok && s0 < t.nst; s0 += C::CH, ++gc) {
        const int cb = gc % C::kChunks;
        ok = WaitWarp(&S.rhs[cb], (gc / C::kChunks) & 1, S, w.status);
        if (!ok) break;
        const unsigned char* rhs = smem + C::kRhsOff + cb * C::kChunkBytes;
        const int s1 = min(t.nst, s0 + C::CH);
        for (int st = s0; st < s1; ++st, ++g, rhs += kStageK * NC * 16) {
            const int slot = g % C::kSlots;
            ok = WaitWarp(&S.tma[slot], (g / C::kSlots) & 1, S, w.status);
            if (!ok) break;
            // inv(L11) is lower triangular: stages past the warp's last row
            // (forward) or before its first (backward) are zero for all its rows
            const int kBase = t.k0 + st * kStageK;
            if (r0 < M && (kBwd ? kBase + kStageK > r0 : kBase <= r1))
                StageProduct<NC, kBwd>(smem + slot * kGBytes, rhs, wrow, kg * C::KPG, rg, cg, acc);
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.empty[slot]);
        }
        if (ok && lane == 0) umma::MbarArrive(&S.rhsEmpty[cb]);
    }
    if (!kBwd) {
        for (int cs = 0; ok && cs < t.carry; ++cs, ++gc) {
            const int cb = gc % C::kChunks;
            ok = WaitWarp(&S.rhs[cb], (gc / C::kChunks) & 1, S, w.status);
            if (!ok) break;
            const cpx<R>* src = reinterpret_cast<const cpx<R>*>(smem + C::kRhsOff + cb * C::kChunkBytes);
            if (kg == 0) {
#pragma unroll
                for (int i = 0; i < C::RPT; ++i) {
                    const int row = wrow + RowIn<R, NC, kBwd>(i, rg) - cs * C::kCarryRows;
                    if (row < 0 || row >= C::kCarryRows) continue;
#pragma unroll
                    for (int j = 0; j < C::CPT; ++j)
                        acc[i][j].Set(acc[i][j].Get() + src[row * NC + j * C::CG + cg]);
                }
            }
            __syncwarp();
            if (lane == 0) umma::MbarArrive(&S.rhsEmpty[cb]);
        }
    }
    constexpr int kGroup0 = C::RW * 32;
    // every compute thread goes on or leaves here: they share the barriers below
    if constexpr (C::KG == 1) {
        if (umma::NamedBarrierOr(1, kComputeThreads, !ok)) return false;
    } else {
        cpx<R>* red = reinterpret_cast<cpx<R>*>(smem + C::kRedOff);
        const int at = (warp % C::RW) * 32 + lane;
        if (kg > 0) {
#pragma unroll
            for (int i = 0; i < C::RPT; ++i)
#pragma unroll
                for (int j = 0; j < C::CPT; ++j)
                    red[((kg - 1) * C::RPT * C::CPT + i * C::CPT + j) * kGroup0 + at] = acc[i][j].Get();
        }
        if (umma::NamedBarrierOr(1, kComputeThreads, !ok)) return false;
        if (kg == 0) {
#pragma unroll
            for (int h = 0; h < C::KG - 1; ++h)
#pragma unroll
                for (int i = 0; i < C::RPT; ++i)
#pragma unroll
                    for (int j = 0; j < C::CPT; ++j)
                        acc[i][j].Set(acc[i][j].Get() +
                                      red[(h * C::RPT * C::CPT + i * C::CPT + j) * kGroup0 + at]);
        }
    }
    bool finish = true;
    if (t.nsplit > 1) {
        // partials in the threads' own layout, summed in split order by the
        // last CTA to arrive
        cpx<R>* part = static_cast<cpx<R>*>(w.partials);
        auto at = [&](int sp, int a) { return part + ((int64_t)(t.slot + sp) * C::RPT * C::CPT + a) * kGroup0 + threadIdx.x; };
        if (kg == 0) {
#pragma unroll
            for (int i = 0; i < C::RPT; ++i)
#pragma unroll
                for (int j = 0; j < C::CPT; ++j) *at(t.split, i * C::CPT + j) = acc[i][j].Get();
        }
        umma::NamedBarrier(1, kComputeThreads);
        if (threadIdx.x == 0) {
            int before;
            asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(before) : "l"(w.counters + t.counter) : "memory");
            const bool last = before == t.nsplit - 1;
            if (last) w.counters[t.counter] = 0;  // ready for the next launch
            S.isLast = last;
        }
        umma::NamedBarrier(1, kComputeThreads);
        finish = S.isLast;
        if (finish && kg == 0) {
#pragma unroll
            for (int i = 0; i < C::RPT; ++i)
#pragma unroll
                for (int j = 0; j < C::CPT; ++j) acc[i][j].Set(mk<R>(0, 0));
            constexpr int kAcc = C::RPT * C::CPT, kFly = kAcc >= 16 ? 1 : 16 / kAcc;  // splits in flight
            for (int sp = 0; sp < t.nsplit; sp += kFly) {
                cpx<R> v[kFly][kAcc];
#pragma unroll
                for (int h = 0; h < kFly; ++h)
#pragma unroll
                    for (int a = 0; a < kAcc; ++a)
                        v[h][a] = sp + h < t.nsplit ? LoadCg(at(sp + h, a)) : mk<R>(0, 0);
#pragma unroll
                for (int h = 0; h < kFly; ++h)
#pragma unroll
                    for (int a = 0; a < kAcc; ++a)
                        acc[a / C::CPT][a % C::CPT].Set(acc[a / C::CPT][a % C::CPT].Get() + v[h][a]);
            }
        }
    }
    if (finish && kg == 0) StoreTile<R, NC, kBwd>(t, f, S.dinv[qs], S.idx[qs], k, wrow, rg, cg, acc, w);
    umma::NamedBarrier(1, kComputeThreads);  // also: the reduction scratch and isLast are rewritten next
    if (finish && threadIdx.x == 0) AddRelease(w.done + t.signal);
    if constexpr (kBwd) {
        if (finish && kg == 0) StoreGrid<R, NC>(t, f, S.idx[qs], k, wrow, rg, cg, acc, B, io);
    }
    return true;
}

template <typename R, int NC>
__device__ void ComputeRole(int k, unsigned char* smem, Sync<R>& S, z64* B, const PanelIO& io, const FlowWork& w) {
    PdlWait();
    int g = 0, gc = 0;
    for (int q = 0;; ++q) {
        const int qs = q % kQueue;
        bool ok = WaitWarp(&S.tileFull[qs], (q / kQueue) & 1, S, w.status);
        const TileCtx<R>& ctx = S.queue[qs];
        // every compute thread leaves together: they share named barriers
        if (umma::NamedBarrierOr(2, kComputeThreads, !ok)) return;
        if (ctx.t.front < 0) return;
        ok = ctx.t.bwd ? ComputeTile<R, NC, true>(ctx.t, ctx.f, qs, k, g, gc, smem, S, B, io, w)
                       : ComputeTile<R, NC, false>(ctx.t, ctx.f, qs, k, g, gc, smem, S, B, io, w);
        if (!ok) return;
        __syncwarp();
        if ((threadIdx.x & 31) == 0) umma::MbarArrive(&S.tileEmpty[qs]);
    }
}

// ------------------------------------------------------------------ kernels

template <typename R, int NC>
__global__ void __launch_bounds__(kThreads, 2) sweep_flow_kernel(const FlowFront<R>* __restrict__ fr,
                                                                 const FlowTile* __restrict__ tiles, int n, int k,
                                                                 z64* __restrict__ B, const __grid_constant__ PanelIO io,
                                                                 const __grid_constant__ FlowWork w) {
    using C = Cfg<R, NC>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ Sync<R> S;
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int i = 0; i < C::kSlots; ++i) {
            umma::MbarInit(&S.tma[i], 1);
            umma::MbarInit(&S.empty[i], kComputeWarps);
        }
        for (int i = 0; i < C::kChunks; ++i) {
            umma::MbarInit(&S.rhs[i], kLoadWarps);
            umma::MbarInit(&S.rhsEmpty[i], kComputeWarps);
        }
        for (int i = 0; i < kQueue; ++i) {
            umma::MbarInit(&S.tileFull[i], 1);
            umma::MbarInit(&S.tileEmpty[i], kLoadWarps + kComputeWarps);
        }
        S.abort = 0;
        S.issued = 0;
        umma::FenceMbarInit();
    }
    __syncthreads();
    if (tid < kLoad0) ComputeRole<R, NC>(k, smem, S, B, io, w);
    else if (tid < kProd0) LoaderRole<R, NC>(k, smem, S, io, w);
    else ProducerRole<R, NC>(fr, tiles, n, smem, S, w);
    __syncthreads();
    // Every role has returned.  When one gave up, copies that nobody waited for may
    // be in flight, whether or not the producer was done: the last one into every
    // slot lands (bounded) before the CTA exits.  S.abort is no longer written.
    if (*reinterpret_cast<volatile int*>(&S.abort)) {
        if (tid == kProd0) DrainCopies<C::kSlots>(S);
        __syncthreads();
    }
    LeaveFlow(w, &S.lastCta);
}

// The panel's right-hand sides in the subproblem's nested-dissection order,
// rounded to the factors' precision: the planes' own entries with the sweep's
// panel coupling folded in.  The rows of the artificial padding are zero and
// stay zero; they are not written.
//
// Bound by memory: points in natural order, so that the grid is read in long
// runs (16 k bytes per point) and rows of 8 k or 16 k bytes are scattered; a
// thread keeps its columns (kVec of them, 16 bytes of the result in complex
// single), two points in flight.  With rows in the subproblem's order, padding
// included, and a 64-bit division per entry it took 26 us at 96 x 96, k = 32, and
// 20 us at 116 x 116, k = 16 (mean over a sweep's panel solves); now 16 and 13 us.
template <typename R, int kVec>
__global__ void __launch_bounds__(256) flow_gather_kernel(const z64* __restrict__ B, cpx<R>* __restrict__ rnd, int own,
                                                          int k, int units, const __grid_constant__ PanelIO io) {
    PdlWait();
    PdlTrigger();  // after the wait: the tree kernel may copy factors as soon as it starts
    const StencilParams& sp = io.sp;
    const int rows = 256 / units, row = threadIdx.x / units, r = (blockIdx.y * units + threadIdx.x % units) * kVec;
    if (row >= rows || r >= k) return;
#pragma unroll 2
    for (int i = blockIdx.x * rows + row; i < own; i += gridDim.x * rows) {
        const int first = io.padding * io.nxy, plane = i / io.nxy, xy = i - plane * io.nxy;
        const int at = __ldg(io.natToNd + first + i);
        const int v = io.vOffset + io.padding + plane;
        const z64* b = B + (xy + (int64_t)(io.nz - 1 - v) * io.nxy) * io.ldk + r;
        const int64_t up = (int64_t)io.nxy * io.ldk;  // the plane before in v
        z64 val[kVec];
        if (io.inMode != 2) {
#pragma unroll
            for (int c = 0; c < kVec; ++c) val[c] = b[c];
            if (io.inMode == 1 && v == io.lowV) {
                const z64 coef = sp.ihz2 * (sp.s1[xy % io.nx + 1] * sp.s2[xy / io.nx + 1] * (sp.is3[v] + sp.is3[v + 1]));
#pragma unroll
                for (int c = 0; c < kVec; ++c) val[c] += coef * b[up + c];
            }
        } else if (v == io.highV) {
            const z64 coef = sp.ihz2 * (sp.s1[xy % io.nx + 1] * sp.s2[xy / io.nx + 1] * (sp.is3[v + 2] + sp.is3[v + 1]));
#pragma unroll
            for (int c = 0; c < kVec; ++c) val[c] = coef * b[c - up];
        } else {
#pragma unroll
            for (int c = 0; c < kVec; ++c) val[c] = mk(0.0, 0.0);
        }
        cpx<R>* const dst = rnd + (int64_t)at * k + r;
        if constexpr (kVec == 2) {
            const c32 a = ccast<float>(val[0]), c = ccast<float>(val[1]);
            *reinterpret_cast<float4*>(dst) = make_float4(a.re, a.im, c.re, c.im);
        } else {
            *dst = ccast<R>(val[0]);
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 g_flowEncode = nullptr;
int g_flowSMs = 0;

template <typename R, int NC>
void LaunchNc(const FlowFront<R>* fr, const FlowTile* tiles, int n, int k, z64* B, const PanelIO& io, const FlowWork& w,
              cudaStream_t st) {
    const int grid = n < 2 * g_flowSMs ? n : 2 * g_flowSMs;
    LaunchPdl(sweep_flow_kernel<R, NC>, dim3(grid), dim3(kThreads), Cfg<R, NC>::kSmem, st, fr, tiles, n, k, B, io, w);
}

template <typename R, int NC>
void PrepareNc() {
    CUDA_CHECK(cudaFuncSetAttribute(sweep_flow_kernel<R, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)Cfg<R, NC>::kSmem));
}

}  // namespace

int FlowCols(int k, double stages) {
    int nc = 1;
    while (nc < k && nc < kFlowMaxCols / 2) nc *= 2;
    if (k <= nc) return nc;
    constexpr double kWideStages = 700;
    const int narrow = (int)CeilDiv(k, nc);
    return narrow % 2 == 0 && narrow * stages >= kWideStages ? kFlowMaxCols : nc;
}

template <typename R>
int FlowCarryChunks(int nc) {
    return nc >= 32 ? Cfg<R, 32>::kCarry : 1;
}

int FlowSlots() { return 2 * g_flowSMs; }

template <typename R>
void PrepareFlowKernels() {
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    CUDA_CHECK(cudaDeviceGetAttribute(&g_flowSMs, cudaDevAttrMultiProcessorCount, dev));
    PrepareNc<R, 1>();
    PrepareNc<R, 2>();
    PrepareNc<R, 4>();
    PrepareNc<R, 8>();
    PrepareNc<R, 16>();
    PrepareNc<R, 32>();
    if (!g_flowEncode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !fn) throw PspError(kCudaError, "cuTensorMapEncodeTiled is unavailable");
        g_flowEncode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
}

template <typename R>
void EncodeFlowMaps(const cpx<R>* G, int s, int u, int ldg, void* out) {
    // G as a (s+u) x s array of 8-byte words (one or two per entry), column
    // stride ldg (even, so every column starts on a 16-byte boundary)
    constexpr int wpe = (int)(sizeof(cpx<R>) / 8);
    const cuuint64_t dims[2] = {(cuuint64_t)wpe * (s + u), (cuuint64_t)s};
    const cuuint64_t strides[1] = {(cuuint64_t)ldg * sizeof(cpx<R>)};
    const cuuint32_t unit[2] = {1, 1};
    const cuuint32_t boxes[2][2] = {{128, (cuuint32_t)kStageK}, {16, (cuuint32_t)FlowRows<R>()}};
    CUtensorMap* maps = static_cast<CUtensorMap*>(out);
    for (int b = 0; b < 2; ++b) {
        const CUresult r = g_flowEncode(&maps[b], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<cpx<R>*>(G), dims, strides,
                                        boxes[b], unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                        b ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) throw PspError(kCudaError, "cuTensorMapEncodeTiled failed for a sweep front");
    }
}

template <typename R>
void LaunchFlowGather(const z64* B, cpx<R>* rnd, int own, int k, const PanelIO& io, cudaStream_t st) {
    // two columns of complex single are 16 bytes when rows are
    const int vec = sizeof(R) == 4 && k % 2 == 0 ? 2 : 1, units = std::min(k / vec, 256);
    const dim3 grid(std::min<unsigned>(CeilDiv(own, 256 / units), 16 * g_flowSMs), CeilDiv(k / vec, units));
    if (vec == 2) LaunchPdl(flow_gather_kernel<R, sizeof(R) == 4 ? 2 : 1>, grid, dim3(256), 0, st, B, rnd, own, k, units, io);
    else LaunchPdl(flow_gather_kernel<R, 1>, grid, dim3(256), 0, st, B, rnd, own, k, units, io);
}

template <typename R>
void LaunchFlow(const FlowFront<R>* fr, const FlowTile* tiles, int n, int k, int cols, z64* B, const PanelIO& io,
                const FlowWork& w, cudaStream_t st) {
    if (n <= 0) return;
    switch (cols) {
        case 1: LaunchNc<R, 1>(fr, tiles, n, k, B, io, w, st); break;
        case 2: LaunchNc<R, 2>(fr, tiles, n, k, B, io, w, st); break;
        case 4: LaunchNc<R, 4>(fr, tiles, n, k, B, io, w, st); break;
        case 8: LaunchNc<R, 8>(fr, tiles, n, k, B, io, w, st); break;
        case 16: LaunchNc<R, 16>(fr, tiles, n, k, B, io, w, st); break;
        default: LaunchNc<R, 32>(fr, tiles, n, k, B, io, w, st); break;
    }
}

#define PSP_FLOW_INSTANTIATE(R)                                                                                       \
    template int FlowCarryChunks<R>(int);                                                                             \
    template void PrepareFlowKernels<R>();                                                                            \
    template void EncodeFlowMaps<R>(const cpx<R>*, int, int, int, void*);                                             \
    template void LaunchFlowGather<R>(const z64*, cpx<R>*, int, int, const PanelIO&, cudaStream_t);                   \
    template void LaunchFlow<R>(const FlowFront<R>*, const FlowTile*, int, int, int, z64*, const PanelIO&,            \
                                const FlowWork&, cudaStream_t);

PSP_FLOW_INSTANTIATE(double)
PSP_FLOW_INSTANTIATE(float)

}  // namespace psp_b200
