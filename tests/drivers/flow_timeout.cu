// One front, one row tile whose K range is split in two.  The second half waits
// for a front that nothing finishes: the kernel gives up within its limit, reports
// it in the status word and leaves its ticket and the fronts' counters at zero.
#include <complex>
#include <cstdio>
#include <cstring>
#include <vector>

#include "kernels.cuh"

using namespace psp_b200;

#define CHECK(x)                                                                              \
    do {                                                                                      \
        const cudaError_t e_ = (x);                                                           \
        if (e_ != cudaSuccess) {                                                              \
            std::printf("%s: %s\n", #x, cudaGetErrorString(e_));                              \
            return 1;                                                                         \
        }                                                                                     \
    } while (0)

template <typename T>
static T* Device(size_t n, const T* src = nullptr) {
    T* p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
    if (src) cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice);
    else cudaMemset(p, 0, n * sizeof(T));
    return p;
}

template <typename R>
static int Run(int k, bool tc) {
    typedef std::complex<R> C;
    constexpr int s = FlowRows<R>(), half = s / 2, kCounters = 3, kDone = 4, kFlag = 3;
    const int cols = tc ? (k > 16 ? 32 : 16) : FlowCols(k);
    // G = [inv(L11)], lower triangular, and the panel's right-hand sides
    std::vector<C> G((size_t)s * s), rhs((size_t)s * k);
    unsigned seed = 12345;
    auto next = [&] { seed = seed * 1664525u + 1013904223u; return (R)((int)(seed >> 8) % 2001 - 1000) / 1000; };
    for (int j = 0; j < s; ++j)
        for (int i = j; i < s; ++i) G[i + (size_t)j * s] = i == j ? C(1, 0) : C(next(), next());
    for (C& v : rhs) v = C(next(), next());
    std::vector<C> D(s, C(4, 0));

    cpx<R>* dG = Device<cpx<R>>(G.size(), reinterpret_cast<const cpx<R>*>(G.data()));
    alignas(64) unsigned char maps[kFlowMapBytes];
    EncodeFlowMaps<R>(dG, s, 0, s, maps);
    FlowFront<R> front;
    std::memset(&front, 0, sizeof(front));
    front.D = Device<cpx<R>>(s, reinterpret_cast<const cpx<R>*>(D.data()));
    front.rel = front.lower = Device<int>(1);
    front.map = Device<unsigned char>(kFlowMapBytes, maps);
    front.s = s;
    FlowTile tile[2];
    std::memset(tile, 0, sizeof(tile));
    for (int sp = 0; sp < 2; ++sp) {
        FlowTile& t = tile[sp];
        t.k0 = sp * half;
        t.ke = t.k0 + half;
        t.nst = half / kFlowStageK;
        t.dep0 = t.dep1 = -1;
        t.split = (short)sp;
        t.nsplit = 2;
    }
    tile[1].dep0 = kFlag;  // nothing finishes this front
    tile[1].need0 = 1;
    FlowWork w;
    std::memset(&w, 0, sizeof(w));
    w.rnd = Device<cpx<R>>(rhs.size(), reinterpret_cast<const cpx<R>*>(rhs.data()));
    w.w = Device<cpx<R>>(rhs.size());
    w.x = Device<cpx<R>>(rhs.size());
    w.partials = Device<cpx<R>>((size_t)2 * s * cols);
    w.counters = Device<int>(kCounters);
    w.ctrl = Device<int>(2 + kDone);
    w.done = w.ctrl + 2;
    w.status = Device<int>(1);
    w.numDone = kDone;
    PanelIO io;
    std::memset(&io, 0, sizeof(io));
    const FlowFront<R>* dFront = Device<FlowFront<R>>(1, &front);
    FlowTile* dTile = Device<FlowTile>(2, tile);
    CHECK(cudaGetLastError());

    auto launch = [&] {
        if constexpr (sizeof(R) == 4) {
            if (tc) return LaunchFlowTc(dFront, dTile, 2, k, cols, nullptr, io, w, 0);
        }
        LaunchFlow<R>(dFront, dTile, 2, k, nullptr, io, w, 0);
    };
    auto atRest = [&](int wantStatus) {
        int ctrl[2 + kDone], status;
        cudaMemcpy(ctrl, w.ctrl, sizeof(ctrl), cudaMemcpyDeviceToHost);
        cudaMemcpy(&status, w.status, sizeof(status), cudaMemcpyDeviceToHost);
        bool ok = status == wantStatus;
        for (int v : ctrl) ok = ok && v == 0;
        if (!ok) std::printf("status %d, ticket %d, done %d\n", status, ctrl[0], ctrl[2]);
        return ok;
    };
    launch();
    CHECK(cudaDeviceSynchronize());
    if (!atRest(2)) return 1;
    return 0;
}

int main() {
    PrepareFlowKernels<double>();
    PrepareFlowKernels<float>();
    PrepareFlowTcKernels();
    int bad = 0;
    for (int k : {1, 5, 16}) {
        if (Run<double>(k, false)) { std::printf("complex double, k = %d\n", k); bad = 1; }
        if (Run<float>(k, false)) { std::printf("complex single, k = %d\n", k); bad = 1; }
    }
    for (int k : {5, 20})
        if (Run<float>(k, true)) { std::printf("tensor cores, k = %d\n", k); bad = 1; }
    std::printf(bad ? "failed\n" : "ok\n");
    return bad;
}
