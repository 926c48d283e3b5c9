// One front, one row tile whose K range is split in two.  First the second half
// waits for a front that nothing finishes: the kernel gives up within its limit,
// reports it in the status word and leaves every counter at zero.  Then the same
// buffers solve the tile.
#include <cmath>
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
static int Run(int k, int cols, bool tc) {
    typedef std::complex<R> C;
    constexpr int s = FlowRows<R>(), half = s / 2, kCounters = 3, kDone = 4, kFlag = 2;
    // G = [inv(L11)], lower triangular, and the panel's right-hand sides
    std::vector<C> G((size_t)s * s), rhs((size_t)s * k), got((size_t)s * k);
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
        t.dep = -1;
        t.split = (short)sp;
        t.nsplit = 2;
    }
    tile[1].dep = kFlag;  // nothing finishes this front
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
    w.numCounters = kCounters;
    PanelIO io;
    std::memset(&io, 0, sizeof(io));
    const FlowFront<R>* dFront = Device<FlowFront<R>>(1, &front);
    FlowTile* dTile = Device<FlowTile>(2, tile);
    CHECK(cudaGetLastError());

    auto launch = [&] {
        if constexpr (sizeof(R) == 4) {
            if (tc) return LaunchFlowTc(dFront, dTile, 2, k, cols, nullptr, io, w, 0);
        }
        LaunchFlow<R>(dFront, dTile, 2, k, cols, nullptr, io, w, 0);
    };
    auto atRest = [&](int wantStatus) {
        int counters[kCounters], ctrl[2 + kDone], status;
        cudaMemcpy(counters, w.counters, sizeof(counters), cudaMemcpyDeviceToHost);
        cudaMemcpy(ctrl, w.ctrl, sizeof(ctrl), cudaMemcpyDeviceToHost);
        cudaMemcpy(&status, w.status, sizeof(status), cudaMemcpyDeviceToHost);
        bool ok = status == wantStatus;
        for (int v : counters) ok = ok && v == 0;
        for (int v : ctrl) ok = ok && v == 0;
        if (!ok) std::printf("status %d, split counter %d, ticket %d, done %d\n", status, counters[0], ctrl[0], ctrl[2]);
        return ok;
    };
    launch();
    CHECK(cudaDeviceSynchronize());
    if (!atRest(2)) return 1;

    tile[1].dep = -1;
    CHECK(cudaMemcpy(dTile, tile, sizeof(tile), cudaMemcpyHostToDevice));
    CHECK(cudaMemset(w.status, 0, sizeof(int)));
    launch();
    CHECK(cudaDeviceSynchronize());
    if (!atRest(0)) return 1;
    CHECK(cudaMemcpy(got.data(), w.w, got.size() * sizeof(C), cudaMemcpyDeviceToHost));
    // s products per sum, each rounded (and added) to at most s units of the
    // last place of the terms' sum of magnitudes
    const double tol = (sizeof(R) == 4 ? 1.2e-7 : 2.3e-16) * s;
    for (int i = 0; i < s; ++i)
        for (int c = 0; c < k; ++c) {
            std::complex<double> sum = 0;
            double mag = 0;
            for (int j = 0; j <= i; ++j) {
                const std::complex<double> p = std::complex<double>(G[i + (size_t)j * s]) *
                                               std::complex<double>(rhs[(size_t)j * k + c]);
                sum += p;
                mag += std::abs(p);
            }
            const double err = std::abs(std::complex<double>(got[(size_t)i * k + c]) - sum / 4.0);
            if (!(err <= tol * mag)) {
                std::printf("row %d column %d: off by %g of %g\n", i, c, err, mag);
                return 1;
            }
        }
    return 0;
}

int main() {
    PrepareFlowKernels<double>();
    PrepareFlowKernels<float>();
    PrepareFlowTcKernels();
    int bad = 0;
    const int columns[][2] = {{1, 1}, {5, 8}, {16, 16}, {20, 32}};  // right-hand sides, of a tile
    for (const auto& c : columns) {
        if (Run<double>(c[0], c[1], false)) { std::printf("complex double, k = %d\n", c[0]); bad = 1; }
        if (Run<float>(c[0], c[1], false)) { std::printf("complex single, k = %d\n", c[0]); bad = 1; }
        if (c[1] >= 16 && Run<float>(c[0], c[1], true)) { std::printf("tensor cores, k = %d\n", c[0]); bad = 1; }
    }
    if (Run<float>(5, 16, true)) { std::printf("tensor cores, k = 5\n"); bad = 1; }
    std::printf(bad ? "failed\n" : "ok\n");
    return bad;
}
