// Device kernels of the sweeping-preconditioned Helmholtz solve and the
// descriptors the host orchestration fills for them.  Every batched
// factorization kernel walks a task list, so one launch covers all fronts of one
// elimination-tree depth across every panel in flight; a panel solve's list
// covers the whole tree.
#pragma once
#include <vector>

#include "common.cuh"

namespace psp_b200 {

// ------------------------------------------------------------------ stencil

// 1-D PML tables live on the device with one guard entry on each side:
// table[i+1] holds the value at grid index i, i in [-1, n].
struct StencilParams {
    int nx, ny, nz;
    double ihx2, ihy2, ihz2;  // 1/(2 h^2) per axis
    double omega;
    const z64* s1; const z64* is1;  // s1Inv and its reciprocal (initialize_finalize.hpp:415-441)
    const z64* s2; const z64* is2;  // s2Inv (443-469)
    const z64* s3; const z64* is3;  // s3Inv on the global sweep coordinate v (471-497)
};

// y := A x, or y := b - A x when b != nullptr, for natural-order grids with
// k interleaved right-hand sides (Multiply, solve.hpp:613-679; the operator is
// FormGlobalRow, initialize_finalize.hpp:527-587, evaluated on the fly).
void LaunchHelmholtzApply(const z64* x, z64* y, const z64* b, const double* vel, const StencilParams& sp, int k,
                          cudaStream_t st);
// The same on planes [zFirst, zFirst + zCount) of slabs whose first stored
// plane is zSlab (x must hold the existing planes next to the range).
void LaunchHelmholtzApplyPlanes(const z64* x, z64* y, const z64* b, const double* vel, const StencilParams& sp,
                                int k, int zFirst, int zCount, int zSlab, cudaStream_t st);

// B := A B by slabs of planes; `ring` holds InPlaceApplyBytes.
size_t InPlaceApplyBytes(const StencilParams& sp, int k);
void LaunchHelmholtzInPlace(z64* B, void* ring, const double* vel, const StencilParams& sp, int k, cudaStream_t st);

// grad[i] (+)= -Re( dA_ii/dvel_i * sum_r Z[i,r] U[i,r] ) for natural-order
// [N][k] grids: the velocity gradient of a real misfit whose forward fields
// are U and whose adjoint fields (A Z = conj of the misfit's field gradient)
// are Z.  dA_ii/dvel_i = 2 omega^2 / vel_i^3 * s1 s2 s3 differentiates the
// centre term of FormGlobalRow (initialize_finalize.hpp:567-568); the
// operator is complex symmetric, so Z reuses the forward factors.
void LaunchVelocityGradient(const z64* U, const z64* Z, const double* vel, const StencilParams& sp, int k,
                            double* grad, int accumulate, cudaStream_t st);

// ------------------------------------------------------------------ batched GEMM

// C = alpha * op(A) * diag(d) * op(B) + beta * C, complex, no conjugation.
// lowerC restricts the update to row >= col.  triA/triB describe structural
// zeros: triA 1 -> op(A)[r][k] = 0 for k > r, 2 -> for k < r;
// triB 1 -> op(B)[k][c] = 0 for k < c, 2 -> for k > c.
template <typename R>
struct GemmOp {
    const cpx<R>* A;
    const cpx<R>* B;
    cpx<R>* C;
    const cpx<R>* d;
    int64_t lda, ldb, ldc;
    int M, N, K;
    int transA, transB, lowerC, triA, triB;
    R alpha_re, alpha_im, beta_re, beta_im;
};
struct GemmTile {
    int op, tm, tn;
};

// Appends the output tiles of `op` (index opIndex) to `tiles`.
template <typename R>
void AppendGemmTiles(const GemmOp<R>& op, int opIndex, std::vector<GemmTile>& tiles);
template <typename R>
void LaunchGemm(const GemmOp<R>* ops, const GemmTile* tiles, int numTiles, cudaStream_t st);
void PrepareGemmKernels();  // launch attributes (the current device's)

// Tensor-core (tcgen05, split TF32) form of the complex-single batched GEMM
// (factor_tc.cu) for ops with real alpha and beta: same op semantics, 128 x
// 64 output tiles, each a self-contained record (operand pointers at the
// tile's origin and the start of its K range), so the kernel reads one
// record per tile and no op table.  A pipeline wait that times out sets the
// value 2 in *status and leaves its tile unwritten.
constexpr int kGemmTcRows = 128, kGemmTcCols = 64;
struct GemmTcTile {
    const c32* A;  // op(A)(row0, kb)
    const c32* B;  // op(B)(kb, col0)
    const c32* d;  // d + kb, or null
    c32* C;        // C(row0, col0)
    int lda, ldb, ldc;
    int m, n, nk;  // rows and columns of the tile inside the op, K extent
    int diag;      // lowerC: only tile-relative r - c >= diag is written
    int flags;     // bit 0 transA, bit 1 transB
    float alpha, beta;
};
// Whether `op` can take tensor-core tiles (real alpha and beta).
bool GemmTcEligible(const GemmOp<float>& op);
void PrepareFactorTcKernels();
void AppendGemmTilesTc(const GemmOp<float>& op, std::vector<GemmTcTile>& tiles);
void LaunchGemmTc(const GemmTcTile* tiles, int numTiles, int* status, cudaStream_t st);

// ------------------------------------------------------------------ factorization

constexpr int kNB = 32;  // column block of the frontal LDL^T

// Leading dimension of a front's persistent factor G: s + u rounded up to
// even, so that every column starts on a 16-byte boundary for bulk copies
// (the padding row is zero).
__host__ __device__ inline int GLeadingDim(int s, int u) { return (s + u + 1) & ~1; }
// Nonzeros of a front's G.
inline double GNonzeros(double s, double u) { return (s + u) * s - s * (s - 1) / 2; }

// One front of one panel during the factorization (cliq::LDL replacement).
template <typename R>
struct FactorFront {
    cpx<R>* L;      // transient (s+u) x s frontal columns, ld = s+u
    cpx<R>* G;      // persistent (s+u) x s: [inv(L11); -L21 inv(L11)], ld = ldg
    cpx<R>* D;      // persistent pivots, s entries
    cpx<R>* U;      // u x u Schur complement (update matrix), ld = u
    cpx<R>* T;      // inversion scratch
    const int* rel; // u entries: row of each structure index in the parent front
    int s, u;
    int ldg;        // leading dimension of G: s+u rounded up to even (16-byte aligned columns)
    int parent;     // index of the parent in the same descriptor array (-1 for a root)
    int cls;        // panel class (tables below)
    int ndOff;      // first ND index of the node in its class ordering
    int vOffset;    // global sweep coordinate of the padded subproblem's first plane
    int s3aOff;     // offset of the panel's artificial-PML table
};

struct ClassTables {
    const int* ndToNat[3];
    const int* nbrRows[3];
};

struct AssemblyParams {
    StencilParams sp;
    const double* vel;    // natural-order velocity
    const z64* s3a;       // artificial s3Inv per panel, vSize+2 entries each
    const z64* is3a;
    double damping;
    ClassTables tabs;
};

template <typename R>
void LaunchAssemble(const FactorFront<R>* fronts, const int* list, int n, const AssemblyParams& ap,
                    cudaStream_t st);
// tasks: (child front, first update column)
template <typename R>
void LaunchExtendAdd(const FactorFront<R>* fronts, const int2* tasks, int n, cudaStream_t st);
template <typename R>
void LaunchLdlDiag(const FactorFront<R>* fronts, const int* list, int n, int J, int* status, cudaStream_t st);
// tasks: (front, first row of a kTrsmRows-row tile below the diagonal block)
constexpr int kTrsmRows = 32;
template <typename R>
void LaunchLdlTrsm(const FactorFront<R>* fronts, const int2* tasks, int n, int J, cudaStream_t st);

// ------------------------------------------------------------------ panel solves

struct PanelIO {
    const int* ndToNat;
    const int* natToNd;
    int nxy, nx, nz;
    int ldk;         // row stride (complex entries per point) of the natural-order grid
    int padding;     // leading planes of the subproblem that are artificial padding
    int vOffset;     // global v of the subproblem's first plane
    int lowV, highV; // global v range of the panel's own planes
    int inMode;      // 0: B_i; 1: B_i - A_{i,i-1} B_{i-1}; 2: -A_{i,i+1} B_{i+1} only
    int outAccumulate;
    StencilParams sp;
};

// One panel solve as two launches (sweep_flow.cu): the panel's right-hand
// sides in the subproblem's ordering, then the whole elimination tree, forward
// and backward, as one ordered tile list (cliq::Solve replacement).

constexpr int kFlowStageK = 16;    // K columns per stage of a tile
constexpr int kFlowMaxCols = 32;   // right-hand sides per tile
constexpr size_t kFlowMapBytes = 256;  // the two TMA maps of one front
constexpr int kTcRows = 128;       // rows of a tensor-core tile (UMMA M)
// Right-hand sides from which the tensor-core kernel is the faster one: its
// time hardly depends on their number (96 x 96 x 76: 11.3 ms per sweep at 1 to 4,
// 11.8 at 8), the CUDA-core kernel takes 7.5, 8.7 and 12.1 ms at 1, 2 and 4.
constexpr int kFlowTcMinCols = 3;
// Rows of a tile: a stage of G is 16 KB.
template <typename R>
constexpr int FlowRows() { return 1024 / (int)sizeof(cpx<R>); }

// One front of the panel being solved (copied in 16-byte words).
template <typename R>
struct alignas(16) FlowFront {
    const cpx<R>* D;      // pivots
    cpx<R>* Pp;           // the parent's plane [s+u][k] that this front's update rows go to
    const cpx<R>* P0;     // the planes its own children write (null: no child, or one without pivots);
    const cpx<R>* P1;     // rows a child does not write are zero
    const int* rel;       // u entries: row of each update row in the parent
    const int* lower;     // u indices of the front's structure in the subproblem's ordering
    const void* map;      // TMA maps of G (forward, backward; 128 bytes each)
    int s, u, ndOff, pad;
};

// One tile: rows row0 .. of front `front`, columns col0 .., K range [k0, ke)
// in nst stages (and `carry` chunks of the children's updates of its update
// rows); split `split` of `nsplit`.  It may start once done[dep] >= need0 and
// done[dep + 1] >= need1 (dep even; -1: it waits for nothing) and adds one to
// done[signal] when its output is written.
struct alignas(16) FlowTile {
    int front, row0, col0, k0;
    int ke, nst, dep, need0;
    int need1, signal, slot, counter;
    short split, nsplit, carry, bwd;
    int pad[2];
};

struct FlowWork {
    void* rnd;       // [nSub][k] the panel's right-hand sides
    void* w;         // [nSub][k] inv(D) Y
    void* x;         // [nSub][k] solution
    void* partials;  // split-K partial tiles
    int* counters;   // arrivals of split tiles (zero between launches)
    int* done;       // finished tiles per front and direction, in pairs (8-byte aligned; zero between launches)
    int* ctrl;       // ticket, finished CTAs (zero between launches)
    int* status;     // bit 2: a wait timed out
    int numDone, numCounters;
};

// Columns of a tile of the CUDA-core kernel for k right-hand sides: the power of
// two that holds them up to 16, else 16, or 32 (kFlowMaxCols) where that is the
// faster one.  `stages`: stages of one panel solve per CTA that runs at once
// and column tile.  A tile of 32 columns takes twice as long per stage, and half of
// it is idle when the 16-column tiles are odd in number; it reads G half as often,
// which pays where wide levels, not the chain of levels, are most of the time.
// Sweeps with 32 instead of 16 columns, time against stages * ceil(k / 16): FP64
// k = 17 to 32: +36 % at 32, +8 % at 270, +1 % at 640, -1 % at 750, -5 % at 1780;
// k = 64: +33 % at 64, +3 % at 540, -1 % at 740, -6 % at 3560; k = 33 to 48: +22 % and
// more everywhere; complex single crosses between 500 and 900.
int FlowCols(int k, double stages);
template <typename R>
int FlowCarryChunks(int cols);
// CTAs that run at once.
int FlowSlots();
template <typename R>
void PrepareFlowKernels();
// The two TMA maps (256 bytes, 64-byte aligned host memory) of a front's factor.
template <typename R>
void EncodeFlowMaps(const cpx<R>* G, int s, int u, int ldg, void* out);
template <typename R>
void LaunchFlowGather(const z64* B, cpx<R>* rnd, int own, int k, const PanelIO& io, cudaStream_t st);
template <typename R>
void LaunchFlow(const FlowFront<R>* fr, const FlowTile* tiles, int n, int k, int cols, z64* B, const PanelIO& io,
                const FlowWork& w, cudaStream_t st);
// The same tile list on the tensor cores (sweep_flow_tc.cu; complex single,
// `cols` 16 or 32 right-hand sides per tile).
void PrepareFlowTcKernels();
int FlowTcSlots();
void LaunchFlowTc(const FlowFront<float>* fr, const FlowTile* tiles, int n, int k, int cols, z64* B, const PanelIO& io,
                  const FlowWork& w, cudaStream_t st);

// ------------------------------------------------------------------ GMRES vectors

// Per-RHS reductions over natural-order [N][k] vectors, one launch each: the
// blocks' sums land in `partial` (gridDim x k) and the last block to finish adds
// them in block order (`ticket`: zero before, and again after, every launch).
int ReduceBlocks(int64_t npoints, int k);
// out[r] := |w[:, r]|
void LaunchNorms(const z64* w, int64_t npoints, int k, void* partial, int* ticket, double* out, cudaStream_t st);
// w -= hPrev (.) vPrev (if vPrev), out[r] := conj(vNext[:, r]) . w[:, r]
void LaunchMgsStep(z64* w, const z64* vPrev, const z64* hPrev, const z64* vNext, int64_t npoints, int k, void* partial,
                   int* ticket, z64* out, cudaStream_t st);
// w -= hPrev (.) vPrev, out[r] := |w[:, r]|
void LaunchMgsNorm(z64* w, const z64* vPrev, const z64* hPrev, int64_t npoints, int k, void* partial, int* ticket,
                   double* out, cudaStream_t st);
// v := w / s (per RHS, s real)
void LaunchScaleColumns(const z64* w, const double* s, z64* v, int64_t npoints, int k, cudaStream_t st);
// x := x0 + sum_i y[i,r] V_i[:,r]
void LaunchCombine(const z64* x0, const z64* V, int64_t vstride, const z64* y, int j1, z64* x, int64_t npoints,
                   int k, cudaStream_t st);

}  // namespace psp_b200
