// Device parts shared by the two kernels that walk an elimination tree in one
// launch (sweep_flow.cu: CUDA cores; sweep_flow_tc.cu: tensor cores).
#pragma once
#include "kernels.cuh"
#include "umma.cuh"

namespace psp_b200 {
namespace flow {

template <typename R>
struct alignas(16) TileCtx {
    FlowTile t;
    FlowFront<R> f;
};
constexpr int kTileWords = sizeof(FlowTile) / 16, kFrontWords = sizeof(FlowFront<float>) / 16;
constexpr int kCtxWords = kTileWords + kFrontWords;
static_assert(sizeof(FlowFront<float>) == sizeof(FlowFront<double>) && kCtxWords <= 32, "copied in 16-byte words");

// Repeats a test until it holds, the CTA gave up, or the wait has run out (which
// gives up).
template <typename Sync, typename Test>
__device__ __forceinline__ bool WaitUntil(const Test& test, Sync& S, int* status) {
    if (test()) return true;
    const uint64_t t0 = umma::GlobalTimerNs();
    for (;;) {
        if (test()) return true;
        if (*reinterpret_cast<volatile int*>(&S.abort)) return false;
        if (umma::GlobalTimerNs() - t0 > umma::kWaitLimitNs) break;
    }
    *reinterpret_cast<volatile int*>(&S.abort) = 1;
    atomicOr(status, 2);
    return false;
}

// Bounded wait on one phase of an mbarrier; false once this or another role of
// the CTA (S.abort) gave up.
template <typename Sync>
__device__ __forceinline__ bool Wait(uint64_t* mbar, uint32_t parity, Sync& S, int* status) {
    return WaitUntil([&] { return umma::MbarTryWait(mbar, parity); }, S, status);
}

// The same by a whole warp, which goes on or gives up together.
template <typename Sync>
__device__ __forceinline__ bool WaitWarp(uint64_t* mbar, uint32_t parity, Sync& S, int* status) {
    return __all_sync(~0u, Wait(mbar, parity, S, status));
}

__device__ __forceinline__ int LoadAcquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Whether both counters of a pair have reached what a tile needs.
__device__ __forceinline__ bool CountsReached(const int* pair, int need0, int need1) {
    int a, b;
    asm volatile("ld.acquire.gpu.global.v2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "l"(pair) : "memory");
    return a >= need0 && b >= need1;
}

// Whether the fronts that a tile reads are finished, tested once (`wait` false) or
// waited for (bounded); by a whole warp.  Every lane acquires the counters itself:
// a vote passes an answer on but orders no memory, and a warp barrier after it
// made the sweeps of small grids 1 to 2 % slower.
template <typename Sync>
__device__ __forceinline__ bool TileReady(const FlowTile& t, bool wait, Sync& S, const FlowWork& w) {
    if (t.dep < 0) return true;
    auto reached = [&] { return CountsReached(w.done + t.dep, t.need0, t.need1); };
    return __all_sync(~0u, wait ? WaitUntil(reached, S, w.status) : reached());
}

// Global data written by other CTAs of this launch: through L2.
__device__ __forceinline__ c32 LoadCg(const c32* p) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    return mk(v.x, v.y);
}
__device__ __forceinline__ z64 LoadCg(const z64* p) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return mk(v.x, v.y);
}

// V consecutive columns of a row; `pair`: rows are 16-byte aligned (even k).
template <typename R, int V>
struct Unit {
    cpx<R> z[V];
};
template <typename R, int V>
__device__ __forceinline__ void LoadUnit(Unit<R, V>& u, const cpx<R>* p, bool pair, bool both) {
    if constexpr (V == 2) {
        if (pair) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
            u.z[0] = mk(v.x, v.y);
            u.z[1] = mk(v.z, v.w);
        } else {
            u.z[0] = LoadCg(p);
            if (both) u.z[1] = LoadCg(p + 1);
        }
    } else {
        u.z[0] = LoadCg(p);
    }
}
template <typename R, int V>
__device__ __forceinline__ Unit<R, V> ZeroUnit() {
    Unit<R, V> u;
#pragma unroll
    for (int i = 0; i < V; ++i) u.z[i] = mk<R>(0, 0);
    return u;
}

// Grid point (in the slab that io addresses) of row `col` of the subproblem's
// ordering; -1 on the artificial padding.
__device__ __forceinline__ int NaturalRow(const PanelIO& io, int col) {
    const int pn = __ldg(io.ndToNat + col);
    const int vl = pn / io.nxy, xy = pn - vl * io.nxy;
    return vl < io.padding ? -1 : xy + (io.nz - 1 - (io.vOffset + vl)) * io.nxy;
}

__device__ __forceinline__ void AddRelease(int* p) {
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p) : "memory");
}

// A tiled 2-D tensor copy (no multicast) of the box at coordinates (x, y) of the
// tensor map at `tmap` (global memory, 64-byte aligned) into this CTA's shared
// memory, completing as transaction bytes on `mbar`; elements outside the tensor
// are zero-filled.  x times the element size must be a multiple of 16 bytes.
// Its lines leave L2 first: a panel's factors are larger than what L2 would
// keep of them until they are read again, and the right-hand sides and index
// maps of the solve should stay there.
__device__ __forceinline__ void TmaLoadStream(void* dst, const void* tmap, int x, int y, uint64_t* mbar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], "
        "[%1, {%2, %3}], [%4], %5;" ::"r"(umma::SmemAddr(dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(umma::SmemAddr(mbar)), "l"(policy)
        : "memory");
}

// This CTA's tiles, by an atomic ticket (one warp).  Take() fetches the words of the
// next tile and of its front, one 16-byte word per lane (front < 0: the list is done).
// It takes the ticket when the copies of the tile before have been issued, and no
// earlier: a CTA that runs ahead of its tiles by no more than its ring of stages
// should hold no ticket that another CTA could start sooner.
template <typename R>
struct TileSource {
    const int4* tiles;
    const int4* fronts;
    int* ctrl;
    int n, tk;
    int4 ctx;

    __device__ __forceinline__ TileSource(const FlowFront<R>* fr, const FlowTile* tl, int n_, int* ctrl_)
        : tiles(reinterpret_cast<const int4*>(tl)), fronts(reinterpret_cast<const int4*>(fr)), ctrl(ctrl_), n(n_) {
        Take();
    }
    __device__ __forceinline__ bool Done() const { return tk >= n; }
    __device__ __forceinline__ void Take() {
        const int lane = threadIdx.x & 31;
        tk = __shfl_sync(~0u, lane == 0 ? atomicAdd(ctrl, 1) : 0, 0);
        ctx = lane < kTileWords && tk < n ? __ldg(tiles + (int64_t)tk * kTileWords + lane) : make_int4(-1, 0, 0, 0);
        const int front = __shfl_sync(~0u, ctx.x, 0);
        if (lane >= kTileWords && lane < kCtxWords && tk < n)
            ctx = __ldg(fronts + (int64_t)front * kFrontWords + lane - kTileWords);
    }
};

// After a role gave up: waits (bounded) until the last copy into each of the ring's
// slots has landed, so none is in flight when the CTA exits.
template <int kSlots, typename Sync>
__device__ __forceinline__ void DrainCopies(Sync& S) {
    for (int s = 0; s < kSlots && s < S.issued; ++s)
        umma::MbarWaitBounded(&S.tma[s], ((S.issued - 1 - s) / kSlots) & 1, nullptr);
}

// At the end of a CTA: the last one leaves the ticket and the counters at zero.
// The arrivals of split tiles are back at zero by themselves (the last arrival
// resets its counter) unless a wait ran out: a CTA that gave up never arrives, and
// a count left behind would make a later launch sum partials that are not there.
__device__ __forceinline__ void LeaveFlow(const FlowWork& w, int* lastCta) {
    if (threadIdx.x == 0) {
        __threadfence();
        *lastCta = atomicAdd(w.ctrl + 1, 1) == (int)gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (*lastCta) {
        for (int i = threadIdx.x; i < w.numDone; i += blockDim.x) w.done[i] = 0;
        if (*reinterpret_cast<volatile int*>(w.status) & 2)
            for (int i = threadIdx.x; i < w.numCounters; i += blockDim.x) w.counters[i] = 0;
        if (threadIdx.x < 2) w.ctrl[threadIdx.x] = 0;
    }
}

}  // namespace flow
}  // namespace psp_b200
