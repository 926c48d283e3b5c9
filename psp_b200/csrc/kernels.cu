// CUDA-core kernels of the solve: on-the-fly 7-point PML stencil, batched
// complex GEMM over task lists, frontal LDL^T building blocks and the multi-RHS
// GMRES vector ops.  (The panel solves are in sweep_flow.cu and sweep_flow_tc.cu.)
#include <algorithm>

#include "kernels.cuh"
#include "umma.cuh"

namespace psp_b200 {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double LoadCg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ z64 LoadCg(const z64* p) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return mk(v.x, v.y);
}

// Face and centre terms of one stencil row (initialize_finalize.hpp:527-587
// and 589-651).  s3M and the three s3 reciprocals come from either the global
// or the panel's artificial table; omega is omega (+ i*damping for panels).
struct Terms {
    z64 c, xL, xR, yL, yR, vL, vR;
};

__device__ __forceinline__ Terms StencilAt(const StencilParams& sp, int x, int y, z64 s3M, z64 is3L, z64 is3M,
                                           z64 is3R, z64 omega, double alpha) {
    const z64 s1M = sp.s1[x + 1], s2M = sp.s2[y + 1];
    const z64 cx = s2M * s3M, cy = s1M * s3M, cz = s1M * s2M;
    Terms t;
    t.xL = sp.ihx2 * (cx * (sp.is1[x] + sp.is1[x + 1]));
    t.xR = sp.ihx2 * (cx * (sp.is1[x + 2] + sp.is1[x + 1]));
    t.yL = sp.ihy2 * (cy * (sp.is2[y] + sp.is2[y + 1]));
    t.yR = sp.ihy2 * (cy * (sp.is2[y + 2] + sp.is2[y + 1]));
    t.vL = sp.ihz2 * (cz * (is3L + is3M));
    t.vR = sp.ihz2 * (cz * (is3R + is3M));
    const z64 w = mk(omega.re / alpha, omega.im / alpha);
    t.c = (t.xL + t.xR + t.yL + t.yR + t.vL + t.vR) - (w * w) * (cz * s3M);
    return t;
}

// ---------------------------------------------------------------- stencil apply

// A block applies the operator to up to kApplyTX points of a row (`px`, chosen by
// ApplyPoints): one thread per point for the coefficients (products and quotients of
// the stretch tables), then one per column and point, all seven entries in flight.  Eight blocks per
// SM hide the first part behind the second.  Bound by memory: 140 x 140 x 80,
// k = 32 (0.8 GB in, 0.8 GB out, b in every second launch): 0.45 ms with 64
// points on 256 threads, most of them idle through the coefficients, now 0.42 ms
// (4.8 TB/s); two or four planes per block with the column in registers have
// fewer warps in flight and take 0.44 and 0.69 ms.
constexpr int kApplyTX = 128;

// out(e, (A x) at entry e of the row piece); `base` is the first of the piece's px
// points in x's storage, `ready` runs before the first use of x.
template <typename Ready, typename Out>
__device__ __forceinline__ void ApplyRow(const z64* __restrict__ x, const double* __restrict__ vel,
                                         const StencilParams& sp, int k, int px, int x0, int yy, int zz, int64_t base,
                                         const Ready& ready, const Out& out) {
    __shared__ z64 coef[kApplyTX][7];
    const int nx = sp.nx, ny = sp.ny, nz = sp.nz;
    const int64_t nxy = (int64_t)nx * ny;
    const int npts = min(px, nx - x0);
    const int v = nz - 1 - zz;
    if ((int)threadIdx.x < npts) {
        const int xx = x0 + threadIdx.x;
        const Terms t = StencilAt(sp, xx, yy, sp.s3[v + 1], sp.is3[v], sp.is3[v + 1], sp.is3[v + 2],
                                  mk(sp.omega, 0.0), vel[xx + yy * (int64_t)nx + zz * nxy]);
        z64* c = coef[threadIdx.x];
        c[0] = t.c;
        c[1] = -t.xL;
        c[2] = -t.xR;
        c[3] = -t.yL;
        c[4] = -t.yR;
        c[5] = -t.vL;
        c[6] = -t.vR;
    }
    ready();
    __syncthreads();
    const int64_t sx = k, sy = (int64_t)nx * k, sz = nxy * k;
    const z64* const row = x + base * k;
    for (int e = threadIdx.x; e < npts * k; e += kApplyTX) {
        const int p = e / k, xx = x0 + p;
        const z64 none = mk(0.0, 0.0);
        const z64* q = row + e;
        const z64 c = q[0];
        const z64 xl = xx > 0 ? q[-sx] : none, xr = xx + 1 < nx ? q[sx] : none;
        const z64 yl = yy > 0 ? q[-sy] : none, yr = yy + 1 < ny ? q[sy] : none;
        const z64 zr = zz + 1 < nz ? q[sz] : none, zl = zz > 0 ? q[-sz] : none;
        const z64* f = coef[p];
        z64 acc = f[0] * c;
        if (xx > 0) cfma(acc, f[1], xl);
        if (xx + 1 < nx) cfma(acc, f[2], xr);
        if (yy > 0) cfma(acc, f[3], yl);
        if (yy + 1 < ny) cfma(acc, f[4], yr);
        if (zz + 1 < nz) cfma(acc, f[5], zr);  // v-1 neighbour
        if (zz > 0) cfma(acc, f[6], zl);       // v+1 neighbour
        out(e, acc);
    }
}

// Planes zFirst ..; storage from plane zSlab.
__global__ void __launch_bounds__(kApplyTX, 8) helmholtz_apply_kernel(const z64* __restrict__ x, z64* __restrict__ y,
                                                                      const z64* __restrict__ b,
                                                                      const double* __restrict__ vel, StencilParams sp,
                                                                      int k, int px, int zFirst, int zSlab) {
    const int x0 = blockIdx.x * px, yy = blockIdx.y, zz = zFirst + (int)blockIdx.z;
    const int64_t base = x0 + yy * (int64_t)sp.nx + (zz - zSlab) * ((int64_t)sp.nx * sp.ny);
    ApplyRow(x, vel, sp, k, px, x0, yy, zz, base, [] {}, [&](int e, z64 v) {
        const int64_t idx = base * k + e;
        y[idx] = b ? b[idx] - v : v;
    });
}

// One step of B := A B: planes zApply .. of A B go to `ring` (plane z in slot
// z mod ringPlanes), planes zCopy .. of it, of an earlier step, to B.  The
// stencil reads one plane beyond its slab on either side, which no step before
// the next has overwritten.  Bound by memory: 4 x 16 bytes per entry.
__global__ void __launch_bounds__(kApplyTX, 8) helmholtz_in_place_kernel(z64* __restrict__ B, z64* __restrict__ ring,
                                                                         const double* __restrict__ vel,
                                                                         StencilParams sp, int k, int px, int zApply,
                                                                         int numApply, int zCopy, int ringPlanes) {
    const int x0 = blockIdx.x * px, yy = blockIdx.y;
    const bool apply = (int)blockIdx.z < numApply;
    const int zz = apply ? zApply + (int)blockIdx.z : zCopy + (int)blockIdx.z - numApply;
    const int64_t nxy = (int64_t)sp.nx * sp.ny, row = x0 + yy * (int64_t)sp.nx, base = row + zz * nxy;
    z64* const slot = ring + (row + zz % ringPlanes * nxy) * k;
    auto ready = [] {
        PdlWait();
        PdlTrigger();
    };
    if (apply) {
        ApplyRow(B, vel, sp, k, px, x0, yy, zz, base, ready, [&](int e, z64 v) { slot[e] = v; });
    } else {
        ready();
        const int n = min(px, sp.nx - x0) * k;
        for (int e = threadIdx.x; e < n; e += 4 * kApplyTX) {
            z64 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (e + i * kApplyTX < n) v[i] = LoadCg(slot + e + i * kApplyTX);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (e + i * kApplyTX < n) B[base * k + e + i * kApplyTX] = v[i];
        }
    }
}

// ---------------------------------------------------------------- velocity gradient

__global__ void __launch_bounds__(kThreads) velocity_gradient_kernel(const z64* __restrict__ U,
                                                                     const z64* __restrict__ Z,
                                                                     const double* __restrict__ vel, StencilParams sp,
                                                                     int k, double* __restrict__ grad, int accumulate) {
    const int64_t nxy = (int64_t)sp.nx * sp.ny, n = nxy * sp.nz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int xx = (int)(i % sp.nx), yy = (int)((i / sp.nx) % sp.ny), zz = (int)(i / nxy);
        const int v = sp.nz - 1 - zz;
        const double a = vel[i];
        const z64 s = sp.s1[xx + 1] * sp.s2[yy + 1] * sp.s3[v + 1];
        const z64 dA = (2.0 * sp.omega * sp.omega / (a * a * a)) * s;
        z64 acc = mk(0.0, 0.0);
        for (int r = 0; r < k; ++r) cfma(acc, Z[i * k + r], U[i * k + r]);
        const double g = -(dA * acc).re;
        grad[i] = accumulate ? grad[i] + g : g;
    }
}

// ---------------------------------------------------------------- batched GEMM

// 64 x 64 tiles, 4 x 4 entries per thread, K in stages of 8 through a ring of
// three that asynchronous copies fill two stages ahead; the tile of C, copied
// meanwhile, waits in shared memory as each thread's own entries.  A thread
// scales the entries of A that it copied itself, so one barrier per stage
// orders the copies, the scaling and the ring.
//
// Bound by FP64 (64 multiply-adds per cycle and SM) at long K and by the traffic of C
// (128 KB per tile) at short K, which the fronts' trees mostly have: factoring a
// 50 x 50 x 50 grid's panels in FP64 took 19.7 ms at 4.7 TFLOP/s with loads, barriers
// and products one after the other, now 11.0 ms at 8.4 TFLOP/s.
constexpr int kGemmTile = 64, kGemmK = 8, kGemmStages = 3, kGemmThreads = 256, kGemmT = 4;
constexpr int kGemmPad = kGemmTile + 1;
template <typename R>
constexpr size_t kGemmSmem = (2 * kGemmStages * kGemmK * kGemmPad + kGemmT * kGemmT * kGemmThreads) * sizeof(cpx<R>);

template <typename R>
__device__ __forceinline__ void CopyEntry(cpx<R>* dst, const cpx<R>* src, bool ok) {
    if constexpr (sizeof(cpx<R>) == 16) umma::CpAsync16(dst, src, ok ? 16u : 0u);
    else umma::CpAsync8(dst, src, ok ? 8u : 0u);
}

template <typename R>
__global__ void __launch_bounds__(kGemmThreads, 2)
    gemm_kernel(const GemmOp<R>* __restrict__ ops, const GemmTile* __restrict__ tiles) {
    constexpr int BM = kGemmTile, BK = kGemmK, T = kGemmT, TX = BM / T;
    extern __shared__ __align__(16) unsigned char gemmSmem[];
    cpx<R>* const As = reinterpret_cast<cpx<R>*>(gemmSmem);
    cpx<R>* const Bs = As + kGemmStages * BK * kGemmPad;
    cpx<R>* const Cs = Bs + kGemmStages * BK * kGemmPad + threadIdx.x;  // own entries
    const GemmTile tl = tiles[blockIdx.x];
    const GemmOp<R>& op = ops[tl.op];
    const int tid = threadIdx.x, row0 = tl.tm * BM, col0 = tl.tn * BM;
    const int M = op.M, N = op.N;
    int kbeg = 0, kend = op.K;
    if (op.triA == 1) kend = min(kend, row0 + BM);
    if (op.triA == 2) kbeg = max(kbeg, row0);
    if (op.triB == 1) kbeg = max(kbeg, col0);
    if (op.triB == 2) kend = min(kend, col0 + BM);
    kbeg = (kbeg / BK) * BK;
    const int ns = kend > kbeg ? (kend - kbeg + BK - 1) / BK : 0;
    // this thread's two entries of a stage of A and of B: their place in the
    // tile, the first one's address, the steps to the second and the next stage
    const bool tA = op.transA, tB = op.transB;
    const cpx<R>* const Aany = op.A;
    const cpx<R>* const Bany = op.B;
    const cpx<R>* const d = op.d;
    const int ar = tA ? tid / BK : tid % BM, ak = tA ? tid % BK : tid / BM;
    const int ar1 = tA ? ar + BM / 2 : ar, ak1 = tA ? ak : ak + BK / 2;
    const int bc = tB ? tid % BM : tid / BK, bk = tB ? tid / BM : tid % BK;
    const int bc1 = tB ? bc : bc + BM / 2, bk1 = tB ? bk + BK / 2 : bk;
    const int64_t aStep = tA ? BK : BK * op.lda, aNext = tA ? BM / 2 * op.lda : BK / 2 * op.lda;
    const int64_t bStep = tB ? BK * op.ldb : BK, bNext = tB ? BK / 2 * op.ldb : BM / 2 * op.ldb;
    const cpx<R>* aP = tA ? Aany + (kbeg + ak) + (row0 + ar) * op.lda : Aany + (row0 + ar) + (kbeg + ak) * op.lda;
    const cpx<R>* bP = tB ? Bany + (col0 + bc) + (kbeg + bk) * op.ldb : Bany + (kbeg + bk) + (col0 + bc) * op.ldb;
    const bool a0 = row0 + ar < M, a1 = row0 + ar1 < M, b0 = col0 + bc < N, b1 = col0 + bc1 < N;
    auto issue = [&](int st, int buf) {
        if (st < ns) {
            const int k0 = kbeg + st * BK;
            cpx<R>* a = As + buf * BK * kGemmPad;
            cpx<R>* b = Bs + buf * BK * kGemmPad;
            const bool ok0 = a0 && k0 + ak < kend, ok1 = a1 && k0 + ak1 < kend;
            const bool ok2 = b0 && k0 + bk < kend, ok3 = b1 && k0 + bk1 < kend;
            CopyEntry(a + ak * kGemmPad + ar, ok0 ? aP : Aany, ok0);
            CopyEntry(a + ak1 * kGemmPad + ar1, ok1 ? aP + aNext : Aany, ok1);
            CopyEntry(b + bk * kGemmPad + bc, ok2 ? bP : Bany, ok2);
            CopyEntry(b + bk1 * kGemmPad + bc1, ok3 ? bP + bNext : Bany, ok3);
            aP += aStep;
            bP += bStep;
        }
    };
    const int tx = tid % TX, ty = tid / TX;  // rows tx + 16 i, columns ty + 16 j
    const bool useBeta = (op.beta_re != R(0) || op.beta_im != R(0)), lowerC = op.lowerC;
    const cpx<R>* const C0 = op.C + (row0 + tx) + (int64_t)(col0 + ty) * op.ldc;
    auto writes = [&](int i, int j) {
        const int r = row0 + tx + i * TX, c = col0 + ty + j * TX;
        return r < M && c < N && !(lowerC && r < c);
    };
    auto issueC = [&] {
        if (!useBeta) return;
#pragma unroll
        for (int j = 0; j < T; ++j)
#pragma unroll
            for (int i = 0; i < T; ++i)
                if (writes(i, j)) CopyEntry(Cs + (j * T + i) * kGemmThreads, C0 + i * TX + j * TX * op.ldc, true);
    };
    issue(0, 0);
    umma::CpAsyncCommit();
    issue(1, 1);
    umma::CpAsyncCommit();
    const cpx<R> one = mk<R>(1, 0);
    auto scale = [&](int k) { return d && k < kend ? d[k] : one; };
    cpx<R> d0 = scale(kbeg + ak), d1 = scale(kbeg + ak1);
    cpx<R> acc[T][T];
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
        for (int j = 0; j < T; ++j) acc[i][j] = mk<R>(0, 0);
    int buf = 0;
    for (int st = 0; st < ns; ++st) {
        umma::CpAsyncWait<1>();
        cpx<R>* const a = As + buf * BK * kGemmPad;
        const cpx<R>* const b = Bs + buf * BK * kGemmPad;
        if (d) {
            cpx<R>& v0 = a[ak * kGemmPad + ar];
            cpx<R>& v1 = a[ak1 * kGemmPad + ar1];
            v0 = v0 * d0;
            v1 = v1 * d1;
            d0 = scale(kbeg + (st + 1) * BK + ak);
            d1 = scale(kbeg + (st + 1) * BK + ak1);
        }
        __syncthreads();  // the stage is here and scaled, and the one before is done with
        issue(st + 2, buf == 0 ? 2 : buf - 1);
        if (st == 0) issueC();
        umma::CpAsyncCommit();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            cpx<R> av[T], bv[T];
#pragma unroll
            for (int i = 0; i < T; ++i) av[i] = a[kk * kGemmPad + tx + i * TX];
#pragma unroll
            for (int j = 0; j < T; ++j) bv[j] = b[kk * kGemmPad + ty + j * TX];
#pragma unroll
            for (int i = 0; i < T; ++i)
#pragma unroll
                for (int j = 0; j < T; ++j) cfma(acc[i][j], av[i], bv[j]);
        }
        if (++buf == kGemmStages) buf = 0;
    }
    if (ns == 0) issueC();
    umma::CpAsyncWaitAll();
    const cpx<R> alpha = mk(op.alpha_re, op.alpha_im), beta = mk(op.beta_re, op.beta_im);
    cpx<R>* const out0 = op.C + (row0 + tx) + (int64_t)(col0 + ty) * op.ldc;
#pragma unroll
    for (int j = 0; j < T; ++j)
#pragma unroll
        for (int i = 0; i < T; ++i) {
            if (!writes(i, j)) continue;
            cpx<R> out = alpha * acc[i][j];
            if (useBeta) out += beta * Cs[(j * T + i) * kGemmThreads];
            out0[i * TX + j * TX * op.ldc] = out;
        }
}

// ---------------------------------------------------------------- front assembly

template <typename R>
__global__ void __launch_bounds__(kThreads) assemble_kernel(const FactorFront<R>* __restrict__ fronts,
                                                            const int* __restrict__ list, AssemblyParams ap) {
    const FactorFront<R> f = fronts[list[blockIdx.x]];
    const StencilParams& sp = ap.sp;
    const int nx = sp.nx, nxy = sp.nx * sp.ny;
    const int* ndToNat = ap.tabs.ndToNat[f.cls];
    const int* nbr = ap.tabs.nbrRows[f.cls];
    const int64_t ld = f.s + f.u;
    const z64 omega = mk(sp.omega, ap.damping);
    const z64* s3a = ap.s3a + f.s3aOff;
    const z64* is3a = ap.is3a + f.s3aOff;
    for (int j = threadIdx.x; j < f.s; j += blockDim.x) {
        const int col = f.ndOff + j;
        const int pn = ndToNat[col];
        const int xy = pn % nxy, vl = pn / nxy;
        const int x = xy % nx, y = xy / nx;
        const int z = sp.nz - 1 - (f.vOffset + vl);
        const double alpha = ap.vel[xy + (int64_t)z * nxy];
        const Terms t = StencilAt(sp, x, y, s3a[vl + 1], is3a[vl], is3a[vl + 1], is3a[vl + 2], omega, alpha);
        cpx<R>* colp = f.L + j * ld;
        colp[j] = ccast<R>(t.c);
        const z64 vals[6] = {t.xL, t.xR, t.yL, t.yR, t.vL, t.vR};
        const int* rows = nbr + (int64_t)col * 6;
#pragma unroll
        for (int n = 0; n < 6; ++n) {
            const int row = rows[n];
            if (row >= 0) colp[row] = ccast<R>(-vals[n]);
        }
    }
}

// ---------------------------------------------------------------- extend-add

template <typename R>
__global__ void __launch_bounds__(kThreads) extend_add_kernel(const FactorFront<R>* __restrict__ fronts,
                                                              const int2* __restrict__ tasks) {
    const int2 task = tasks[blockIdx.x];
    const FactorFront<R> ch = fronts[task.x];
    const FactorFront<R> p = fronts[ch.parent];
    const int b1 = min(task.y + 32, ch.u);
    const int64_t ldp = p.s + p.u;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nw = blockDim.x / 32;
    for (int b = task.y + warp; b < b1; b += nw) {
        const int rb = ch.rel[b];
        const cpx<R>* ucol = ch.U + (int64_t)b * ch.u;
        if (rb < p.s) {
            cpx<R>* dst = p.L + rb * ldp;
            for (int a = b + lane; a < ch.u; a += 32) dst[ch.rel[a]] += ucol[a];
        } else {
            cpx<R>* dst = p.U + (int64_t)(rb - p.s) * p.u - p.s;
            for (int a = b + lane; a < ch.u; a += 32) dst[ch.rel[a]] += ucol[a];
        }
    }
}

// ---------------------------------------------------------------- LDL^T blocks

// LDL^T of the diagonal block at (J, J): unit L, pivots D, and inv(L_JJ) written
// into G's diagonal block, all in registers:
// lane = row, a warp has every eighth column.  Step j publishes column j,
// still unscaled; every thread forms the row's multiplier l from it, subtracts
// l times column j's entries from its columns right of j, and l times row j of
// the inverse (a shuffle away) from its columns of the inverse up to j.
//
// Bound by the latency of the 32 steps: one barrier, one read of the column and
// one reciprocal each.  With the block in shared memory, two barriers per step
// and the inverse afterwards by one thread per column, a launch took 54 us
// (complex single; 51 us FP64), now 26 (31) us.
template <typename R>
__global__ void __launch_bounds__(kThreads) ldl_diag_kernel(const FactorFront<R>* __restrict__ fronts,
                                                            const int* __restrict__ list, int J, int* status) {
    constexpr int kWarps = kThreads / 32, kCols = kNB / kWarps;
    static_assert(kNB == 32, "lane = row");
    __shared__ cpx<R> column[2][kNB];
    const FactorFront<R>& f = fronts[list[blockIdx.x]];
    const int b = min(kNB, f.s - J);
    const int64_t ld = f.s + f.u, lg = f.ldg;
    cpx<R>* const Lb = f.L + J + J * ld;
    cpx<R>* const Gb = f.G + J + J * lg;
    cpx<R>* const D = f.D + J;
    const int i = threadIdx.x & 31, warp = threadIdx.x / 32;
    const cpx<R> zero = mk<R>(0, 0), one = mk<R>(1, 0);
    cpx<R> A[kCols], X[kCols];  // columns warp + 8 q
#pragma unroll
    for (int q = 0; q < kCols; ++q) {
        const int c = warp + kWarps * q;
        A[q] = i < b && i >= c ? Lb[i + c * ld] : zero;
        X[q] = i == c ? one : zero;
    }
#pragma unroll
    for (int q0 = 0; q0 < kCols; ++q0)
#pragma unroll 1
        for (int w0 = 0; w0 < kWarps; ++w0) {
            const int j = q0 * kWarps + w0;
            if (j >= b) break;
            if (warp == w0) column[j & 1][i] = A[q0];
            __syncthreads();
            const cpx<R> own = column[j & 1][i], d = column[j & 1][j];
            const cpx<R> l = own * cinv(d);
            if (threadIdx.x == 0) {
                if ((d.re == R(0) && d.im == R(0)) || !(d.re == d.re) || !(d.im == d.im)) atomicOr(status, 1);
                D[j] = d;
            }
            if (warp == w0 && i > j) A[q0] = l;
#pragma unroll
            for (int q = 0; q < kCols; ++q) {
                const int c = warp + kWarps * q;
                const cpx<R> x = mk<R>(__shfl_sync(~0u, X[q].re, j), __shfl_sync(~0u, X[q].im, j));
                if (i > j) {
                    if (c <= j) X[q] -= l * x;
                    else if (i >= c) A[q] -= l * column[j & 1][c];
                }
            }
        }
#pragma unroll
    for (int q = 0; q < kCols; ++q) {
        const int c = warp + kWarps * q;
        if (i >= b || c >= b) continue;
        Lb[i + c * ld] = i > c ? A[q] : i == c ? one : zero;
        Gb[i + c * lg] = X[q];
    }
}

// L[r, J:J+b] := F[r, J:J+b] inv(L_JJ)^T inv(D_J) for a row tile below the block.
template <typename R>
__global__ void __launch_bounds__(kThreads) ldl_trsm_kernel(const FactorFront<R>* __restrict__ fronts,
                                                            const int2* __restrict__ tasks, int J) {
    constexpr int RT = kTrsmRows;
    __shared__ cpx<R> Li[kNB][kNB + 1];
    __shared__ cpx<R> Dinv[kNB];
    __shared__ cpx<R> Ar[RT][kNB + 1];
    const int2 task = tasks[blockIdx.x];
    const FactorFront<R> f = fronts[task.x];
    const int b = min(kNB, f.s - J);
    const int64_t ld = f.s + f.u;
    const int r0 = task.y;
    const int rows = min(RT, f.s + f.u - r0);
    const int tid = threadIdx.x;
    for (int e = tid; e < b * b; e += blockDim.x) {
        const int i = e % b, j = e / b;
        Li[i][j] = f.G[(J + i) + (J + j) * (int64_t)f.ldg];
    }
    if (tid < b) Dinv[tid] = cinv(f.D[J + tid]);
    for (int e = tid; e < rows * b; e += blockDim.x) {
        const int i = e % rows, m = e / rows;
        Ar[i][m] = f.L[(r0 + i) + (J + m) * ld];
    }
    __syncthreads();
    for (int e = tid; e < rows * b; e += blockDim.x) {
        const int i = e % rows, c = e / rows;
        cpx<R> acc = mk<R>(0, 0);
        for (int m = 0; m <= c; ++m) cfma(acc, Ar[i][m], Li[c][m]);
        f.L[(r0 + i) + (J + c) * ld] = acc * Dinv[c];
    }
}

// ---------------------------------------------------------------- GMRES vectors

// Per-column reductions: blocks of up to kReduceThreads threads (column x
// point), kReduceUnroll points of each thread in flight, at most two blocks per
// SM; the last block to finish adds the blocks' sums, in block order, with all
// of its threads.  Bound by memory at large grids and by latency at small ones:
// 2 x 512 threads x 4 points x 2 vectors x 16 bytes per SM cover HBM's latency,
// and 296 block sums of up to 512 columns-per-thread slots are a handful of
// loads per thread, where a second launch that added 1184 of them one after the
// other took longer than the pass over the vectors.
constexpr int kReduceMaxBlocks = 296;
constexpr int kReduceThreads = 512;
constexpr int kReduceUnroll = 4;

// Sum over this block's threads of a column; the result is in ty == 0.
template <typename T>
__device__ __forceinline__ T BlockColumnSum(T acc, T* red) {
    const int at = threadIdx.y * blockDim.x + threadIdx.x;
    red[at] = acc;
    __syncthreads();
    for (int s = blockDim.y / 2; s > 0; s >>= 1) {
        if (threadIdx.y < s) red[at] += red[at + s * blockDim.x];
        __syncthreads();
    }
    return red[threadIdx.x];
}

// acc of every thread of the grid -> out[column] (its square root on request).
// `ticket` is zero before and after the launch.
template <typename T, typename Finish>
__device__ __forceinline__ void GridColumnSum(T acc, T* red, T* partial, int* ticket, const Finish& finish) {
    __shared__ int last;
    const int tx = threadIdx.x, ty = threadIdx.y, k = blockDim.x, nblocks = gridDim.x;
    acc = BlockColumnSum(acc, red);
    if (nblocks > 1) {
        if (ty == 0) {
            partial[blockIdx.x * (int64_t)k + tx] = acc;
            __threadfence();
        }
        __syncthreads();
        if (tx == 0 && ty == 0) {
            const int before = atomicAdd(ticket, 1);
            last = before == nblocks - 1;
            if (last) *ticket = 0;
            __threadfence();
        }
        __syncthreads();
        if (!last) return;
        acc = T();
#pragma unroll 8
        for (int b = ty; b < nblocks; b += blockDim.y) acc += LoadCg(partial + b * (int64_t)k + tx);
        acc = BlockColumnSum(acc, red);
    }
    if (ty == 0) finish(tx, acc);
}

// w -= hprev vprev per column (when there is a vprev), then out = <vnext, w>
// per column (kNorm false) or |w| (kNorm true).
template <bool kUpdate, bool kNorm>
__global__ void __launch_bounds__(1024) mgs_step_kernel(z64* __restrict__ w, const z64* __restrict__ vprev,
                                                        const z64* __restrict__ hprev, const z64* __restrict__ vnext,
                                                        int64_t npoints, int k, void* partial, int* ticket, void* out) {
    extern __shared__ z64 redc[];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const z64 h = kUpdate ? hprev[tx] : mk(0.0, 0.0);
    z64 acc = mk(0.0, 0.0);
    const int64_t stride = (int64_t)gridDim.x * blockDim.y, step = stride * k;
    int64_t p = blockIdx.x * (int64_t)blockDim.y + ty, e = p * k + tx;
    auto point = [&](int64_t at, z64 wv, z64 vp, z64 vn) {
        if (kUpdate) {
            wv -= h * vp;
            w[at] = wv;
        }
        if (kNorm) acc.re += cabs2(wv);
        else acc += mk(vn.re * wv.re + vn.im * wv.im, vn.re * wv.im - vn.im * wv.re);  // conj(v) w
    };
    for (; p + (kReduceUnroll - 1) * stride < npoints; p += kReduceUnroll * stride, e += kReduceUnroll * step) {
        z64 wv[kReduceUnroll], vp[kReduceUnroll], vn[kReduceUnroll];
#pragma unroll
        for (int i = 0; i < kReduceUnroll; ++i) {
            wv[i] = w[e + i * step];
            if (kUpdate) vp[i] = vprev[e + i * step];
            if (!kNorm) vn[i] = vnext[e + i * step];
        }
#pragma unroll
        for (int i = 0; i < kReduceUnroll; ++i) point(e + i * step, wv[i], vp[i], vn[i]);
    }
    for (; p < npoints; p += stride, e += step)
        point(e, w[e], kUpdate ? vprev[e] : acc, kNorm ? acc : vnext[e]);
    if (kNorm) {
        double* norm = static_cast<double*>(out);
        GridColumnSum(acc.re, reinterpret_cast<double*>(redc), static_cast<double*>(partial), ticket,
                      [&](int r, double v) { norm[r] = sqrt(v); });
    } else {
        z64* dot = static_cast<z64*>(out);
        GridColumnSum(acc, redc, static_cast<z64*>(partial), ticket, [&](int r, z64 v) { dot[r] = v; });
    }
}

__global__ void scale_columns_kernel(const z64* __restrict__ w, const double* __restrict__ s, z64* __restrict__ v,
                                     int64_t n, int k) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e % k);
        const double inv = 1.0 / s[r];
        v[e] = inv * w[e];
    }
}

__global__ void combine_kernel(const z64* __restrict__ x0, const z64* __restrict__ V, int64_t vstride,
                               const z64* __restrict__ y, int j1, z64* __restrict__ x, int64_t n, int k) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e % k);
        z64 acc = x0[e];
        for (int i = 0; i < j1; ++i) cfma(acc, y[i * k + r], V[i * vstride + e]);
        x[e] = acc;
    }
}

inline dim3 ReduceBlockDim(int k) {
    int ty = 1;
    while (ty * 2 * k <= kReduceThreads) ty *= 2;
    return dim3(k, ty);
}

unsigned ElementwiseGrid(int64_t n) { return (unsigned)std::min<int64_t>(CeilDiv(n, kThreads), 148 * 16); }

}  // namespace

// ---------------------------------------------------------------- host launchers

// Points of a row per block: kApplyTX and a rest, or, where a launch would end on a
// few long blocks, equal pieces: of at most kApplyTX points when it has less than
// four waves of blocks (a wave is 8 per SM), of at most 32 when these have 3000
// entries and more (from 24 columns on) or are less than half a wave.
// 128 points and a rest -> equal pieces of up to 128 -> of up to 32 (us; 64 points on
// 256 threads before): 129 x 40 x 40, k = 16: 50 -> 45 -> 49 (51), k = 64: 143 -> 120 ->
// 115 (120); two planes of 127 x 40, k = 64: 36 -> 36 -> 22 (23), k = 16: 21 -> 21 -> 17
// (19); 250 x 30 x 30, k = 48: 106 -> 106 -> 99 (100).  With more waves long pieces are
// the better ones, and the short rest fills the gaps: 140 x 140 x 80, k = 8: 133 -> 136 ->
// 167 (177), 220 x 220 x 40, k = 16: 252 -> 265 -> 306 (298).
int ApplyPoints(int nx, int ny, int planes, int k) {
    constexpr int64_t kWave = 8 * 148;
    const int64_t blocks = (int64_t)CeilDiv(nx, kApplyTX) * ny * planes;
    if (blocks >= 4 * kWave) return kApplyTX;
    const int most = k >= 24 || blocks < kWave / 2 ? 32 : kApplyTX;
    return (int)CeilDiv(nx, CeilDiv(nx, most));
}

void LaunchHelmholtzApply(const z64* x, z64* y, const z64* b, const double* vel, const StencilParams& sp, int k,
                          cudaStream_t st) {
    LaunchHelmholtzApplyPlanes(x, y, b, vel, sp, k, 0, sp.nz, 0, st);
}

void LaunchHelmholtzApplyPlanes(const z64* x, z64* y, const z64* b, const double* vel, const StencilParams& sp,
                                int k, int zFirst, int zCount, int zSlab, cudaStream_t st) {
    const int px = ApplyPoints(sp.nx, sp.ny, zCount, k);
    dim3 grid(CeilDiv(sp.nx, px), sp.ny, zCount);
    helmholtz_apply_kernel<<<grid, kApplyTX, 0, st>>>(x, y, b, vel, sp, k, px, zFirst, zSlab);
    CUDA_LAUNCH_CHECK();
}

// Planes of one step of the in-place apply.  Up to kInPlaceRing bytes (0.6 % of
// the device's memory) A B is one step and its copy: 400 MB take 320 us, against
// 426, 414 us in slabs of 32, 64 MB, whose launches cost more than their shorter
// way through L2 saves.  Larger grids go in slabs of a third of that.
constexpr size_t kInPlaceRing = size_t(1) << 30;
int InPlaceSlabPlanes(const StencilParams& sp, int k) {
    const size_t plane = (size_t)sp.nx * sp.ny * k * sizeof(z64);
    return plane * sp.nz <= kInPlaceRing ? sp.nz : (int)std::max<size_t>(1, kInPlaceRing / 3 / plane);
}

size_t InPlaceApplyBytes(const StencilParams& sp, int k) {
    const size_t plane = (size_t)sp.nx * sp.ny * k * sizeof(z64);
    return plane * std::min(sp.nz, 3 * InPlaceSlabPlanes(sp, k));
}

void LaunchHelmholtzInPlace(z64* B, void* ring, const double* vel, const StencilParams& sp, int k, cudaStream_t st) {
    const int planes = InPlaceSlabPlanes(sp, k), slabs = (int)CeilDiv(sp.nz, planes);
    const int ringPlanes = std::min(sp.nz, 3 * planes);
    const int behind = slabs > 1 ? 2 : 1;
    const int px = ApplyPoints(sp.nx, sp.ny, planes, k);
    auto count = [&](int s) { return s < 0 || s >= slabs ? 0 : std::min(planes, sp.nz - s * planes); };
    for (int s = 0; s < slabs + behind; ++s) {
        const int na = count(s), nc = count(s - behind);
        if (na + nc == 0) continue;
        LaunchPdl(helmholtz_in_place_kernel, dim3(CeilDiv(sp.nx, px), sp.ny, na + nc), dim3(kApplyTX), 0, st, B,
                  static_cast<z64*>(ring), vel, sp, k, px, s * planes, na, (s - behind) * planes, ringPlanes);
        CUDA_LAUNCH_CHECK();
    }
}

void LaunchVelocityGradient(const z64* U, const z64* Z, const double* vel, const StencilParams& sp, int k,
                            double* grad, int accumulate, cudaStream_t st) {
    const int64_t n = (int64_t)sp.nx * sp.ny * sp.nz;
    velocity_gradient_kernel<<<ElementwiseGrid(n), kThreads, 0, st>>>(U, Z, vel, sp, k, grad, accumulate);
    CUDA_LAUNCH_CHECK();
}

template <typename R>
void AppendGemmTiles(const GemmOp<R>& op, int opIndex, std::vector<GemmTile>& tiles) {
    constexpr int BM = kGemmTile, BN = kGemmTile;
    if (op.M <= 0 || op.N <= 0) return;
    const int tmN = (int)CeilDiv(op.M, BM), tnN = (int)CeilDiv(op.N, BN);
    for (int tn = 0; tn < tnN; ++tn)
        for (int tm = 0; tm < tmN; ++tm) {
            if (op.lowerC && tm * BM + BM - 1 < tn * BN) continue;
            tiles.push_back(GemmTile{opIndex, tm, tn});
        }
}

void PrepareGemmKernels() {
    CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kGemmSmem<double>));
    CUDA_CHECK(cudaFuncSetAttribute(gemm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kGemmSmem<float>));
}

template <typename R>
void LaunchGemm(const GemmOp<R>* ops, const GemmTile* tiles, int numTiles, cudaStream_t st) {
    if (numTiles <= 0) return;
    gemm_kernel<R><<<numTiles, kGemmThreads, kGemmSmem<R>, st>>>(ops, tiles);
    CUDA_LAUNCH_CHECK();
}

template <typename R>
void LaunchAssemble(const FactorFront<R>* fronts, const int* list, int n, const AssemblyParams& ap,
                    cudaStream_t st) {
    if (n <= 0) return;
    assemble_kernel<R><<<n, kThreads, 0, st>>>(fronts, list, ap);
    CUDA_LAUNCH_CHECK();
}

template <typename R>
void LaunchExtendAdd(const FactorFront<R>* fronts, const int2* tasks, int n, cudaStream_t st) {
    if (n <= 0) return;
    extend_add_kernel<R><<<n, kThreads, 0, st>>>(fronts, tasks);
    CUDA_LAUNCH_CHECK();
}

template <typename R>
void LaunchLdlDiag(const FactorFront<R>* fronts, const int* list, int n, int J, int* status, cudaStream_t st) {
    if (n <= 0) return;
    ldl_diag_kernel<R><<<n, kThreads, 0, st>>>(fronts, list, J, status);
    CUDA_LAUNCH_CHECK();
}

template <typename R>
void LaunchLdlTrsm(const FactorFront<R>* fronts, const int2* tasks, int n, int J, cudaStream_t st) {
    if (n <= 0) return;
    ldl_trsm_kernel<R><<<n, kThreads, 0, st>>>(fronts, tasks, J);
    CUDA_LAUNCH_CHECK();
}

int ReduceBlocks(int64_t npoints, int k) {
    const dim3 bd = ReduceBlockDim(k);
    return (int)std::max<int64_t>(1, std::min<int64_t>(CeilDiv(npoints, bd.y), kReduceMaxBlocks));
}

void LaunchNorms(const z64* w, int64_t npoints, int k, void* partial, int* ticket, double* out, cudaStream_t st) {
    const dim3 bd = ReduceBlockDim(k);
    mgs_step_kernel<false, true><<<ReduceBlocks(npoints, k), bd, sizeof(z64) * bd.x * bd.y, st>>>(
        const_cast<z64*>(w), nullptr, nullptr, nullptr, npoints, k, partial, ticket, out);
    CUDA_LAUNCH_CHECK();
}

void LaunchMgsStep(z64* w, const z64* vPrev, const z64* hPrev, const z64* vNext, int64_t npoints, int k, void* partial,
                   int* ticket, z64* out, cudaStream_t st) {
    const dim3 bd = ReduceBlockDim(k);
    const auto kernel = vPrev ? mgs_step_kernel<true, false> : mgs_step_kernel<false, false>;
    kernel<<<ReduceBlocks(npoints, k), bd, sizeof(z64) * bd.x * bd.y, st>>>(w, vPrev, hPrev, vNext, npoints, k, partial,
                                                                          ticket, out);
    CUDA_LAUNCH_CHECK();
}

void LaunchMgsNorm(z64* w, const z64* vPrev, const z64* hPrev, int64_t npoints, int k, void* partial, int* ticket,
                   double* out, cudaStream_t st) {
    const dim3 bd = ReduceBlockDim(k);
    mgs_step_kernel<true, true><<<ReduceBlocks(npoints, k), bd, sizeof(z64) * bd.x * bd.y, st>>>(
        w, vPrev, hPrev, nullptr, npoints, k, partial, ticket, out);
    CUDA_LAUNCH_CHECK();
}

void LaunchScaleColumns(const z64* w, const double* s, z64* v, int64_t npoints, int k, cudaStream_t st) {
    const int64_t n = npoints * k;
    scale_columns_kernel<<<ElementwiseGrid(n), kThreads, 0, st>>>(w, s, v, n, k);
    CUDA_LAUNCH_CHECK();
}

void LaunchCombine(const z64* x0, const z64* V, int64_t vstride, const z64* y, int j1, z64* x, int64_t npoints,
                   int k, cudaStream_t st) {
    const int64_t n = npoints * k;
    combine_kernel<<<ElementwiseGrid(n), kThreads, 0, st>>>(x0, V, vstride, y, j1, x, n, k);
    CUDA_LAUNCH_CHECK();
}

#define PSP_INSTANTIATE(R)                                                                                      \
    template void AppendGemmTiles<R>(const GemmOp<R>&, int, std::vector<GemmTile>&);                \
    template void LaunchGemm<R>(const GemmOp<R>*, const GemmTile*, int, cudaStream_t);              \
    template void LaunchAssemble<R>(const FactorFront<R>*, const int*, int, const AssemblyParams&,             \
                                    cudaStream_t);                                                             \
    template void LaunchExtendAdd<R>(const FactorFront<R>*, const int2*, int, cudaStream_t);                   \
    template void LaunchLdlDiag<R>(const FactorFront<R>*, const int*, int, int, int*, cudaStream_t);           \
    template void LaunchLdlTrsm<R>(const FactorFront<R>*, const int2*, int, int, cudaStream_t);

PSP_INSTANTIATE(double)
PSP_INSTANTIATE(float)

}  // namespace psp_b200
