// The cluster form of the later MOOD passes (csrc/mood_cluster.cuh) run on the
// CPU, a lane a fiber: warp, block and cluster barriers are kept, and between
// barriers the warps run in a chosen order.  Lists are sets and counters are
// counts, so every order gives the same state; the program runs the kernel in
// several and compares.  The test writes cluster_order_gen.h: the few helpers
// of kernels.cu that the kernel calls, then the kernel's source with its
// assembly and its __shared__ variable replaced by the functions below.
#include <ucontext.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <random>
#include <vector>

#include <cuda_runtime.h>
#undef __launch_bounds__
#undef __noinline__
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)

namespace emu {
constexpr int BLOCKS = 2, THREADS = 512, WARPS = BLOCKS * THREADS / 32;
struct Barrier {
    int size, arrived = 0;
    long gen = 0;
    unsigned long long in[32], out[2][32];  // a warp's exchanged values
};
struct Lane {
    ucontext_t ctx;
    std::vector<char> stack = std::vector<char>(96 << 10);
    uint3 tid, bid;
    const long* gen = nullptr;  // waits while *gen == seen
    long seen = 0;
    bool done = false;
};
Lane lanes[BLOCKS * THREADS];
Barrier warps[WARPS], blocks[BLOCKS], cluster;
ucontext_t home;
Lane* cur;
std::unique_ptr<char[]> shared[BLOCKS];

const unsigned long long* meet(Barrier& b, int who = 0, unsigned long long v = 0) {
    const long g = b.gen;
    if (b.size == 32) b.in[who] = v;
    if (++b.arrived == b.size) {
        if (b.size == 32) std::memcpy(b.out[g & 1], b.in, sizeof b.in);
        b.arrived = 0;
        b.gen++;
    } else {
        cur->gen = &b.gen;
        cur->seen = g;
        swapcontext(&cur->ctx, &home);
    }
    return b.out[g & 1];
}
const unsigned long long* warp_meet(unsigned long long v) {
    const int i = (int)(cur - lanes);
    return meet(warps[i / 32], i % 32, v);
}
// every lane to its end; order: the warps, the first the most urgent
void run(void (*body)(), const std::vector<int>& order) {
    for (Barrier& w : warps) w = Barrier{32};
    for (Barrier& b : blocks) b = Barrier{THREADS};
    cluster = Barrier{BLOCKS * THREADS};
    for (int i = 0; i < BLOCKS * THREADS; i++) {
        Lane& l = lanes[i];
        l.tid = uint3{(unsigned)(i % THREADS), 0, 0};
        l.bid = uint3{(unsigned)(i / THREADS), 0, 0};
        l.gen = nullptr;
        l.done = false;
        getcontext(&l.ctx);
        l.ctx.uc_stack.ss_sp = l.stack.data();
        l.ctx.uc_stack.ss_size = l.stack.size();
        l.ctx.uc_link = &home;
        makecontext(&l.ctx, body, 0);
    }
    for (;;) {
        bool ran = false, left = false;
        for (int w : order) {
            for (int i = 32 * w; i < 32 * w + 32; i++) {
                Lane& l = lanes[i];
                left = left || !l.done;
                if (l.done || (l.gen && *l.gen == l.seen)) continue;
                l.gen = nullptr;
                cur = &l;
                swapcontext(&home, &l.ctx);
                if (!l.gen) l.done = true;  // it came back without a barrier
                ran = true;
            }
            if (ran) break;  // the most urgent warp that can run
        }
        if (!left) return;
        if (!ran) {
            std::printf("lanes wait at different barriers\n");
            std::exit(3);
        }
    }
}
}  // namespace emu

#define threadIdx (emu::cur->tid)
#define blockIdx (emu::cur->bid)
#define PDL_ENTRY()
static unsigned __ballot_sync(unsigned, bool p) {
    const unsigned long long* v = emu::warp_meet(p);
    unsigned m = 0;
    for (int i = 0; i < 32; i++) m |= v[i] ? 1u << i : 0u;
    return m;
}
static bool __any_sync(unsigned, bool p) { return __ballot_sync(0, p) != 0; }
template <typename T>
static T __shfl_sync(unsigned, T x, int from) {
    unsigned long long u = 0;
    std::memcpy(&u, &x, sizeof x);
    u = emu::warp_meet(u)[from & 31];
    std::memcpy(&x, &u, sizeof x);
    return x;
}
static int __reduce_min_sync(unsigned, int x) {
    const unsigned long long* v = emu::warp_meet((unsigned)x);
    for (int i = 0; i < 32; i++) x = (int)v[i] < x ? (int)v[i] : x;
    return x;
}
static void __syncwarp() { emu::warp_meet(0); }
static void __syncthreads() { emu::meet(emu::blocks[blockIdx.x]); }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int __ffs(int x) { return __builtin_ffs(x); }
template <typename T>
static T __ldg(const T* p) { return *p; }
template <typename T>
static T atomicAdd(T* p, T v) { return *p += v, *p - v; }
template <typename T>
static T atomicOr(T* p, T v) { T o = *p; *p |= v; return o; }
static int atomicExch(int* p, int v) { int o = *p; *p = v; return o; }
static void __threadfence() {}
static void cudaGraphSetConditional(cudaGraphConditionalHandle, unsigned) {}
static long long __double_as_longlong(double x) { long long u; std::memcpy(&u, &x, 8); return u; }
static int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static int __double2loint(double x) { return (int)__double_as_longlong(x); }
static double __hiloint2double(int h, int l) {
    const unsigned long long u = ((unsigned long long)(unsigned)h << 32) | (unsigned)l;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
static double __drcp_rn(double x) { return 1.0 / x; }
template <typename T>
static T min(T a, T b) { return b < a ? b : a; }
template <typename T>
static T max(T a, T b) { return a < b ? b : a; }
static void emu_cluster_sync() { emu::meet(emu::cluster); }
static unsigned emu_cluster_nctaid() { return emu::BLOCKS; }
template <typename T>
static T& emu_shared() {
    auto& s = emu::shared[blockIdx.x];
    if (!s) s.reset(new char[sizeof(T)]);
    return *reinterpret_cast<T*>(s.get());
}

#include "engine.h"
using std::fmax;
using std::fmin;
#include "cluster_order_gen.h"

using namespace hosono;
namespace {
constexpr int N = 24, R = 2, NG = R + 2, NT = N + 2 * NG, PITCH = 32, PLANE = PITCH * NT;
constexpr int TILES = (NT + 7) / 8;

// one instance after the dense pass 1: the stage input, first-order fluxes,
// and the cells detect lowered
struct Stage {
    std::vector<double> dbl = std::vector<double>(PLANE * 42);
    std::vector<uint8_t> byt = std::vector<uint8_t>(PLANE * 13);
    std::vector<double> pv = std::vector<double>(13 * 3 * 4 * R), qw = std::vector<double>(3 * R);
    std::vector<int2> lists[7];
    int counts[8] = {};
    InstDev dev{};
    InstState st{};
    BatchFlags flags{};
    int2 instTiles = make_int2(0, TILES);
    Batch B{};
    void make(int cap) {
        Geo& G = dev.geo;
        G = Geo{N, N, NG, NT, NT, PITCH, PLANE, R, 1, 13, 3, 1.0 / N, 1.0 / N, 1.0 / N, 1.0 / N};
        dev.phys = Phys{1.4, 1e-12, 1e-12, 1e-12, 0};
        std::mt19937 gen(7);
        auto uni = [&](double a, double b) { return a + (b - a) * (gen() / 4294967296.0); };
        for (int k = 0; k < (int)pv.size(); k += 13) {  // any weights of sum one
            double s = 0;
            for (int e = 0; e < 13; e++) s += pv[k + e] = uni(0.0, e == 6 ? 8.0 : 1.0);
            for (int e = 0; e < 13; e++) pv[k + e] /= s;
        }
        for (int q = 0; q < 2; q++) qw[q] = 0.5;
        for (int q = 0; q < 3; q++) qw[3 + q] = q == 1 ? 8.0 / 18 : 5.0 / 18;
        double* q = dbl.data();
        for (int r = 0; r < 3; r++, q += 8 * PLANE) dev.U[r] = q;
        dev.FX = q;
        dev.FY = q + 8 * PLANE;
        dev.CTX = q + 16 * PLANE;
        dev.CTY = q + 17 * PLANE;
        dev.pv = pv.data();
        dev.qw = qw.data();
        uint8_t* b = byt.data();
        uint8_t** planes[] = {(uint8_t**)&dev.scheme[0], (uint8_t**)&dev.scheme[1], &dev.rrRec, &dev.rec, &dev.recF, &dev.recB,
                              &dev.recFB, &dev.fail, &dev.nextPass, &dev.dirty, &dev.lowered, &dev.innerCount, &dev.detMask};
        for (uint8_t** p : planes) *p = b, b += PLANE;
        for (int j = 0; j < NT; j++)
            for (int i = 0; i < NT; i++) {
                const int c = j * PITCH + i, si = (i - NG + N) % N, sj = (j - NG + N) % N;
                std::mt19937 h(1 + si + N * sj);
                const bool in = (si - 12) * (si - 12) + (sj - 12) * (sj - 12) < 40;
                const double rho = (in ? 3.0 : 1.0) * (1.0 + 0.3 * (h() / 4294967296.0)), p = in ? 20.0 : 1.0;
                const double u[8] = {rho, 0.3 * rho, -0.2 * rho, 0.1 * rho, p / 0.4 + 0.07 * rho + 0.07, 0.2, 0.3, 0.1};
                for (int v = 0; v < 8; v++) dev.U[0][v * PLANE + c] = u[v];
                dev.scheme[0][c] = R;
                dev.rrRec[c] = R * 0x55;
                dev.detMask[c] = kstrict::DM_SHOCK;
            }
        for (int j = 1; j < NT; j++)
            for (int i = 1; i < NT; i++)
                for (int dir = 0; dir < 2; dir++) {
                    const int c = j * PITCH + i, cl = dir == XDIR ? c - 1 : c - PITCH;
                    double a[8], u[8], F[8];
                    for (int v = 0; v < 8; v++) a[v] = dev.U[0][v * PLANE + cl], u[v] = dev.U[0][v * PLANE + c];
                    hllc(dev.phys, a, u, dir, F);
                    for (int v = 0; v < 8; v++) (dir == XDIR ? dev.FX : dev.FY)[v * PLANE + c] = F[v];
                    (dir == XDIR ? dev.CTX : dev.CTY)[c] = F[dir == XDIR ? MAGY : MAGX];
                }
        for (auto& l : lists) l.assign(2 * TILES * 256, make_int2(0, 0));
        B.dev = &dev;
        B.st = &st;
        B.flags = &flags;
        int2** to[] = {&B.L.rec, &B.L.rec2, &B.L.face, &B.L.recF, &B.L.low, &B.L.next, &B.L.casc};
        for (int l = 0; l < 7; l++) *to[l] = lists[l].data();
        B.L.counts = counts;
        B.L.cap = TILES * 256;
        B.mcMax = 800;
        B.maxInst = 1;
        B.instTiles = &instTiles;
        st.live = st.stepping = st.stageActive = 1;
        st.dtdx = st.dtdy = 0.05;
        st.passCap = cap;
        int* low = reinterpret_cast<int*>(B.L.low);
        for (int j = NG + 2; j < NG + 20; j += 2) {
            low[st.nDetect] = j * PITCH + NG + (5 * j) % N;
            dev.lowered[low[st.nDetect++]] = 1;
        }
    }
};
Stage* now;
void body() { kstrict::k_mood_passes<false>(now->B, ROLE_STATE, ROLE_A, 0, 0); }
}  // namespace

int main(int argc, char** argv) {
    const int cap = argc > 1 ? std::atoi(argv[1]) : 1000;
    std::unique_ptr<Stage> first;
    for (int kind = 0; kind < 5; kind++) {
        // the cluster's first warp first, then last, then anywhere
        std::vector<int> order(emu::WARPS);
        for (int w = 0; w < emu::WARPS; w++) order[w] = kind == 1 ? emu::WARPS - 1 - w : w;
        std::mt19937 gen(kind);
        if (kind > 1)
            for (int w = emu::WARPS - 1; w > 0; w--) std::swap(order[w], order[gen() % (w + 1)]);
        std::unique_ptr<Stage> s(new Stage);
        s->make(cap);
        now = s.get();
        emu::run(body, order);
        const InstState& S = s->st;
        std::printf("order %d: %d passes, %lld lowered, error %d\n", kind, S.passes, (long long)S.detectTotal, S.error);
        if (!first) {
            first = std::move(s);
            if (first->st.passes < 3 || first->st.detectTotal < 40) return 4;  // too little work to tell
            continue;
        }
        if (std::memcmp(&S, &first->st, sizeof S)) return 5;
        if (std::memcmp(s->dbl.data(), first->dbl.data(), s->dbl.size() * 8)) return 6;
        if (!S.error && std::memcmp(s->byt.data(), first->byt.data(), s->byt.size())) return 7;
    }
    return 0;
}
