// mood_cluster.cuh -- the short parts of a forward-Euler stage, one thread-
// block cluster per instance (included by kernels.cu): pass 1's face cascade
// (k_mood_faces) and, after the dense pass-1 update, every later MOOD pass
// (k_mood_passes; timeStep.f90:86-128).
//
// What bounds them: nothing but latency.  A later pass of a small solve
// touches a few hundred cells; as a chain of grid-wide kernels it cost nine
// launches (and four per cascade iteration) of 3-20 us each.  Here a pass is four
// phases between hardware cluster barriers, and each item is split over
// lanes so that a lane's chain is short: a cell's face states over 32 lanes
// (4 faces x 8 variables: 13 loads at R = 2 instead of 104), a face's fluxes
// over 8 lanes, an updated cell over 8 (its variables), a lowered cell's
// flags over 13 (its diamond).  The lists are per instance (segments of the
// batch's lists that start at the instance's first tile), and hold cell
// indices; a flag's first setter appends its cell, so nothing scans the grid.
// Orders differ from the chain's, values do not: every list is a set, and
// each item's arithmetic is the chain's, statement by statement.
//
// Flags: a pass reads recompute / recomputeFLICD in one pair of planes (rec,
// recF or recB, recFB) and its flag rebuild sets the other, so the old flags
// are cleared in the same phase.  Between stages all of them, nextPass, fail,
// lowered and DM_CASC are zero, and so are the counters.
//
// Every branch around a barrier is taken on values all blocks of the cluster
// read alike: a counter is changed only in phases a barrier away from its
// last read.
#pragma once

constexpr int MC_THREADS = 512, MC_WARPS = MC_THREADS / 32;
enum : int { MC_FAIL = 0, MC_NEXT = 2, MC_REC = 4, MC_RECF = 6 };  // InstState::mc, two of each
constexpr int MC_FS = 72;                 // doubles per face of a warp's exchange buffer (64 + 8 against bank conflicts)
constexpr int MC_BUF = 4 * MC_FS;         // a warp's exchange buffer
constexpr int MC_PV = 25 * 4 * 4 * 3;     // prediction vectors of the largest radius
constexpr int MC_QW = 4 * 3;

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_nctaid() {
    unsigned n;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;\n" : "=r"(n));
    return n;
}
// a counter as the last phase left it (past L1)
__device__ __forceinline__ int mc_ld(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

struct Mc {
    const InstDev& d;
    InstState& S;
    const double* __restrict__ U;  // the stage input (read only while the kernel runs)
    const Phys P;                  // hydro flag, gamma, floors
    int8_t* sch;
    int *fail, *next, *rec[2], *recF[2], *low, *casc;  // the instance's lists
    uint8_t *pRec[2], *pRecF[2];                       // flag planes
    double* buf;                                       // this warp's exchange buffer
    const double* spv;                                 // prediction vectors and weights in shared memory
    const double* sqw;
    int gw, nw, lane;  // warp of the cluster, warps of the cluster
    bool lead;         // the cluster's first thread
};
__device__ __forceinline__ int cell_j(const Geo& G, int c) { return c / G.pitch; }

// append the items of the lanes with pred (every lane of the warp calls)
__device__ __forceinline__ void mc_append(int* list, int* counter, bool pred, int item, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    int base = 0;
    const int leader = __ffs(m) - 1;
    if (lane == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) list[base + __popc(m & ((1u << lane) - 1))] = item;
}
// set plane[c]; true for the thread that changed it from zero (the byte is
// set through its 32-bit word, so exactly one thread sees it change)
__device__ __forceinline__ bool mc_first(uint8_t* plane, long long c) {
    const unsigned sh = 8u * (unsigned)(c & 3);
    const unsigned old = atomicOr(reinterpret_cast<unsigned*>(plane + (c - (c & 3))), 1u << sh);
    return ((old >> sh) & 0xffu) == 0;
}
// the radius-2 diamond by lane: the centre, its cross, then the outer ring
__device__ __forceinline__ int diamond_di(int l) { return (int)((0x2204113322132ull >> (4 * l)) & 15) - 2; }
__device__ __forceinline__ int diamond_dj(int l) { return (int)((0x0422131313222ull >> (4 * l)) & 15) - 2; }

// Face states of variable v around cell c at radius RR and quadrature points
// 0..nq-1: sum_k pv(k, q) * U(v, stencil_k), k ascending from zero
// (reconstruct.f90:109-124), one lane per variable.
template <int RR>
__device__ __forceinline__ void mc_gp(const double* __restrict__ Uv, int pitch, int c, const double* pvf, int qs, int nq,
                                      double out[4]) {
    constexpr int NS = 1 + 2 * RR * (RR + 1);
    double u[NS];
    int k = 0;
#pragma unroll
    for (int a = -RR; a <= RR; a++)
#pragma unroll
        for (int b = -RR; b <= RR; b++)
            if (iabs_c(a) + iabs_c(b) <= RR) u[k++] = __ldg(Uv + c + b * pitch + a);
#pragma unroll 1
    for (int q = 0; q < nq; q++) {
        double s = 0.0;
#pragma unroll
        for (int t = 0; t < NS; t++) s = s + pvf[q * qs + t] * u[t];
        // nq is a run-time count: store by selects, out stays in registers
        out[0] = q == 0 ? s : out[0];
        out[1] = q == 1 ? s : out[1];
        out[2] = q == 2 ? s : out[2];
        out[3] = q == 3 ? s : out[3];
    }
}
__device__ __forceinline__ void mc_face_states(const Mc& m, int rr, int c, int f, int v, int nq, double out[4]) {
    const Geo& G = m.d.geo;
    const double* Uv = m.U + v * G.plane;
    if (rr == 0) {  // the first-order copy
        out[0] = out[1] = out[2] = out[3] = __ldg(Uv + c);
        return;
    }
    const double* pvf = m.spv + G.nsMax * (G.nqMax * (f + 4 * (rr - 1)));
    if (rr == 1)
        mc_gp<1>(Uv, G.pitch, c, pvf, G.nsMax, nq, out);
    else if (rr == 2)
        mc_gp<2>(Uv, G.pitch, c, pvf, G.nsMax, nq, out);
    else
        mc_gp<3>(Uv, G.pitch, c, pvf, G.nsMax, nq, out);
}

// Re-reconstruct the n cells of `list` (reconstruct_faceValsWithGP's inner
// pass, reconstruct.f90:80-139), one warp per cell: lane 8 f + v sums
// variable v of face f, then lane 8 f + q tests the state at point q.
// Inadmissible cells go on the fail list.  fromNext: clear the cell's mark.
__device__ __forceinline__ void mc_recon(const Mc& m, const int* list, int n, bool fromNext, int* failCount) {
    const Geo& G = m.d.geo;
    const int f = m.lane >> 3, v = m.lane & 7;
    for (int e = m.gw; e < n; e += m.nw) {
        const int c = list[e];
        const int j = cell_j(G, c), i = c - j * G.pitch;
        if (i < G.g - 2 || j < G.g - 2 || i > G.g + G.nx + 1 || j > G.g + G.ny + 1) continue;  // uniform over the warp
        const int nb = f == NORTH ? c + G.pitch : f == SOUTH ? c - G.pitch : f == EAST ? c + 1 : c - 1;
        const int rr = min((int)m.sch[c], (int)m.sch[nb]);
        const int rN = __shfl_sync(0xffffffffu, rr, 0), rS = __shfl_sync(0xffffffffu, rr, 8);
        const int rE = __shfl_sync(0xffffffffu, rr, 16), rW = __shfl_sync(0xffffffffu, rr, 24);
        if (m.lane == 0) {
            m.d.rrRec[c] = (uint8_t)(rN | (rS << 2) | (rE << 4) | (rW << 6));
            if (fromNext) m.d.nextPass[c] = 0;
        }
        if (rr > 0) {
            double o[4] = {0.0, 0.0, 0.0, 0.0};
            mc_face_states(m, rr, c, f, v, rr + 1, o);
#pragma unroll
            for (int q = 0; q < 4; q++) m.buf[f * MC_FS + q * 8 + v] = o[q];
        }
        __syncwarp();
        bool bad = false;
        if (rr > 0 && v <= rr) {
            double u[NCONS];
#pragma unroll
            for (int w = 0; w < NCONS; w++) u[w] = m.buf[f * MC_FS + v * 8 + w];
            bad = !admissible(u[DENS], cons2pres(m.P, u));
        }
        const bool any = __any_sync(0xffffffffu, bad);
        mc_append(m.fail, failCount, any && m.lane == 0, c, m.lane);
        __syncwarp();
    }
}

// The serial lowering loop of reconstruct.f90:146-169 for the n cells of the
// fail list, one warp per cell (order independent: a cell lowers only its own
// scheme; every flag write sets): gridBlock_lowerOrder (gridBlock.f90:194-235)
// and the cross marked for the next inner pass.  withF: recomputeFLICD too
// (in pass 1 it is set everywhere).
__device__ __forceinline__ void mc_lower(const Mc& m, int n, int cur, bool withF, int* nextCount) {
    const Geo& G = m.d.geo;
    const int l = m.lane;
    const int di = l < 13 ? diamond_di(l) : 0, dj = l < 13 ? diamond_dj(l) : 0;
    for (int e = m.gw; e < n; e += m.nw) {
        const int c = m.fail[e];
        const int j = cell_j(G, c), i = c - j * G.pitch;
        bool first = false;
        if (l == 0) {
            const int s = m.sch[c];
            m.sch[c] = (int8_t)(s - 1 > 0 ? s - 1 : 0);
            m.d.fail[c] = 0;
            const int mask = m.d.detMask[c];
            first = !(mask & DM_CASC);
            if (first) m.d.detMask[c] = (uint8_t)(mask | DM_CASC);
        }
        mc_append(m.casc, &m.S.nCasc, first, c, l);
        const int ii = i + di, jj = j + dj, cn = c + dj * G.pitch + di;
        const bool in = l < 13 && ii >= 0 && jj >= 0 && ii < G.nxt && jj < G.nyt;
        const bool range = ii >= G.g - 2 && jj >= G.g - 2 && ii <= G.g + G.nx + 1 && jj <= G.g + G.ny + 1;
        mc_append(m.rec[cur], &m.S.mc[MC_REC + cur], in && l < 5 && mc_first(m.pRec[cur], cn), cn, l);
        mc_append(m.next, nextCount, in && l < 5 && range && mc_first(m.d.nextPass, cn), cn, l);
        if (withF) mc_append(m.recF[cur], &m.S.mc[MC_RECF + cur], in && mc_first(m.pRecF[cur], cn), cn, l);
    }
}

// The face cascade (reconstruct.f90:143-171) from nF failing cells; returns
// the lowerings.  All blocks enter with the same nF, a barrier after the
// fail list was filled.
__device__ __forceinline__ int mc_cascade(const Mc& m, int nF, int cur, bool withF, int* iters) {
    int sum = 0;
    for (int it = 0; nF > 0; it++) {
        int* nextCount = &m.S.mc[MC_NEXT + (it & 1)];
        mc_lower(m, nF, cur, withF, nextCount);
        sum += nF;
        ++*iters;
        cluster_sync();
        const int nN = mc_ld(nextCount);
        mc_recon(m, m.next, nN, true, &m.S.mc[MC_FAIL + ((it + 1) & 1)]);
        if (m.lead) m.S.mc[MC_FAIL + (it & 1)] = 0;  // read before the last barrier
        cluster_sync();
        nF = mc_ld(&m.S.mc[MC_FAIL + ((it + 1) & 1)]);
        if (m.lead) *nextCount = 0;
    }
    return sum;
}

// getFluxes_ (getFluxes.f90:16-90) next to the n cells of the recompute list,
// one warp per cell, 8 lanes per face: lane 8 f + v sums variable v of both
// face states of face f, lane 8 f + q solves the Riemann problem of point q,
// lane 8 f + v adds the Gauss sum of flux v in quadrature order.  A cell
// takes its west and south faces, and the east or north one where the cell
// beyond is not flagged.  Face states are rebuilt at the radius each side was
// last reconstructed with (rrRec), the quadrature uses the face's current
// radius (riemannSolver.f90:23-47), as in flux_list.
__device__ __forceinline__ void mc_flux(const Mc& m, const int* list, int n, const uint8_t* pRec) {
    const Geo& G = m.d.geo;
    const int f = m.lane >> 3, v = m.lane & 7;
    const bool x = f == EAST || f == WEST;
    const int fL = x ? EAST : NORTH, fR = x ? WEST : SOUTH;
    // variable v's place in face coordinates (physics.cuh)
    const int vf = x ? v : v == MOMX || v == MAGX ? v + 1 : v == MOMY || v == MAGY ? v - 1 : v;
    for (int e = m.gw; e < n; e += m.nw) {
        const int c = list[e];
        const int cf = f == EAST ? c + 1 : f == NORTH ? c + G.pitch : c;  // the face's right / upper cell
        const int cl = x ? cf - 1 : cf - G.pitch;
        const int j = cell_j(G, cf), i = cf - j * G.pitch;
        bool act = i >= G.g - 1 && j >= G.g - 1 && i <= G.g + G.nx + 1 && j <= G.g + G.ny + 1;
        if (act && cf != c) act = pRec[cf] == 0;
        int rr = 0;
        if (act) {
            rr = min((int)m.sch[cf], (int)m.sch[cl]);
            const int rrL = (m.d.rrRec[cl] >> (2 * fL)) & 3, rrR = (m.d.rrRec[cf] >> (2 * fR)) & 3;
            double o[4] = {0.0, 0.0, 0.0, 0.0};
            mc_face_states(m, rrL, cl, fL, v, rr + 1, o);
#pragma unroll
            for (int q = 0; q < 4; q++) m.buf[f * MC_FS + (2 * q) * 8 + vf] = o[q];
            mc_face_states(m, rrR, cf, fR, v, rr + 1, o);
#pragma unroll
            for (int q = 0; q < 4; q++) m.buf[f * MC_FS + (2 * q + 1) * 8 + vf] = o[q];
        }
        __syncwarp();
        double F[NCONS];
        const bool solve = act && v <= rr;
        if (solve) {
            double uL[NCONS], uR[NCONS];
#pragma unroll
            for (int w = 0; w < NCONS; w++) {
                uL[w] = m.buf[f * MC_FS + (2 * v) * 8 + w];
                uR[w] = m.buf[f * MC_FS + (2 * v + 1) * 8 + w];
            }
            hllc_face(m.P, uL, uR, F);
        }
        __syncwarp();
        if (solve) {
#pragma unroll
            for (int w = 0; w < NCONS; w++) m.buf[f * MC_FS + v * 8 + w] = F[w];
        }
        __syncwarp();
        if (act) {
            double s;
            if (rr == 0) {
                s = m.buf[f * MC_FS + vf];
            } else {
                s = 0.0;
                for (int q = 0; q <= rr; q++) s = s + m.sqw[q + G.nqMax * (rr - 1)] * m.buf[f * MC_FS + q * 8 + vf];
            }
            (x ? m.d.FX : m.d.FY)[v * G.plane + cf] = s;
            if (v == (x ? MAGY : MAGX)) (x ? m.d.CTX : m.d.CTY)[cf] = s;
        }
        __syncwarp();
    }
}

// FLICD, the update (timeStep.f90:107-118) and detect_ALL on the n cells of
// the recomputeFLICD list, 8 lanes per cell: lane v updates variable v (the
// MAGX and MAGY lanes also correct the cell's fluxes, as ct_cell does), the
// group's first lane runs the per-pass tests.
__device__ __forceinline__ void mc_update(const Mc& m, const int* list, int n, int uout, const uint8_t* pRecF) {
    const InstDev& d = m.d;
    const Geo& G = d.geo;
    const int v = m.lane & 7, base = m.lane & ~7;
    const double dt = m.S.dt;
    const double dtdx = dt / G.dx, dtdy = dt / G.dy;
    double* Uo = role_ptr(d, m.S.parity, uout);
    const double* fxy = d.FX + MAGY * G.plane;
    const double* fyx = d.FY + MAGX * G.plane;
    for (int e0 = m.gw * 4; e0 < n; e0 += m.nw * 4) {
        const int e = e0 + (m.lane >> 3);
        int c = 0;
        bool in = false, cell = false;
        if (e < n) {
            c = list[e];
            const int j = cell_j(G, c), i = c - j * G.pitch;
            in = i >= G.g && j >= G.g && i <= G.g + G.nx && j <= G.g + G.ny;
            cell = in && i < G.g + G.nx && j < G.g + G.ny;
        }
        double un = 0.0;
        double f0 = 0.0, f1 = 0.0, g0 = 0.0, g1 = 0.0;
        if (in && v == MAGY) {
            f0 = flicd_x_at(fxy, fyx, c, G.pitch);
            d.CTX[c] = f0;
            if (cell) f1 = pRecF[c + 1] ? flicd_x_at(fxy, fyx, c + 1, G.pitch) : d.CTX[c + 1];
        } else if (in && v == MAGX) {
            g0 = flicd_y_at(fxy, fyx, c, G.pitch);
            d.CTY[c] = g0;
            if (cell) g1 = pRecF[c + G.pitch] ? flicd_y_at(fxy, fyx, c + G.pitch, G.pitch) : d.CTY[c + G.pitch];
        } else if (cell) {
            const double* fx = d.FX + v * G.plane + c;
            const double* fy = d.FY + v * G.plane + c;
            f0 = fx[0];
            f1 = fx[1];
            g0 = fy[0];
            g1 = fy[G.pitch];
        }
        if (cell) {
            un = __ldg(m.U + v * G.plane + c) - dtdx * (f1 - f0) - dtdy * (g1 - g0);
            Uo[v * G.plane + c] = un;
        }
        double u[NCONS];
#pragma unroll
        for (int w = 0; w < NCONS; w++) u[w] = __shfl_sync(0xffffffffu, un, base + w);
        bool low = false;
        if (cell && v == 0 && m.sch[c] > 0) {
            low = detect_cell_at(m.P, d.detMask + c, m.U + DENS * G.plane, c, G.pitch, u);
            if (low) d.lowered[c] = 1;
        }
        mc_append(m.low, &m.S.nDetect, low, c, m.lane);
    }
}

// The flag rebuild after detect, from the lists: the cross and the diamond of
// every translate of each cell detect lowered (gridBlock_lowerOrder with
// boundaryConditions_applyMOOD's periodic sync) into the other pair of flag
// planes, and one scheme per translate class of each cell this pass lowered:
// the minimum over the class of (scheme - lowered)^+.  One warp per cell.  A
// class holds one interior cell, so at most one entry of the low list; that
// entry alone takes a class detect lowered, and the cascade's entries of
// other classes all write the same minimum, which a partly written class
// still has.  Clears the pass's own flags.
__device__ __forceinline__ void mc_flags(const Mc& m, int nLow, int nCasc, int cur, int nRec, int nRecF) {
    const InstDev& d = m.d;
    const Geo& G = d.geo;
    const int l = m.lane;
    const int di = l < 13 ? diamond_di(l) : 0, dj = l < 13 ? diamond_dj(l) : 0;
    const int reach = G.bc == 1 ? 1 : 0;
    const int tb = l < 9 ? l / 3 - 1 : 2, tt = l < 9 ? l % 3 - 1 : 2;  // this lane's translate
    for (int e = m.gw; e < nLow + nCasc; e += m.nw) {
        const bool fromLow = e < nLow;
        const int c = fromLow ? m.low[e] : m.casc[e - nLow];
        const int j = cell_j(G, c), i = c - j * G.pitch;
        const int jo = j + tb * G.ny, io = i + tt * G.nx;
        const bool mem = l < 9 && iabs_c(tb) <= reach && iabs_c(tt) <= reach && jo >= 0 && io >= 0 && jo < G.nyt &&
                         io < G.nxt;
        const int co = jo * G.pitch + io;
        int s = 127, lo = 0;
        if (mem) {
            s = m.sch[co];
            lo = d.lowered[co];
        }
        const bool classLow = __any_sync(0xffffffffu, lo != 0);
        if (mem) s = max(s - lo, 0);
        s = __reduce_min_sync(0xffffffffu, s);
        if (fromLow || !classLow) {
            if (mem) m.sch[co] = (int8_t)s;
        }
        if (!fromLow) {
            if (l == 0) d.detMask[c] &= (uint8_t)~DM_CASC;
            continue;
        }
        unsigned members = __ballot_sync(0xffffffffu, mem);
        while (members) {
            const int t = __ffs(members) - 1;
            members &= members - 1;
            const int ii = i + (t % 3 - 1) * G.nx + di, jj = j + (t / 3 - 1) * G.ny + dj;
            const int cn = jj * G.pitch + ii;
            const bool in = l < 13 && ii >= 0 && jj >= 0 && ii < G.nxt && jj < G.nyt;
            mc_append(m.rec[cur ^ 1], &m.S.mc[MC_REC + (cur ^ 1)], in && l < 5 && mc_first(m.pRec[cur ^ 1], cn), cn, l);
            mc_append(m.recF[cur ^ 1], &m.S.mc[MC_RECF + (cur ^ 1)], in && mc_first(m.pRecF[cur ^ 1], cn), cn, l);
        }
    }
    for (int e = m.gw * 32 + l; e < nRec + nRecF; e += m.nw * 32) {
        if (e < nRec)
            m.pRec[cur][m.rec[cur][e]] = 0;
        else
            m.pRecF[cur][m.recF[cur][e - nRec]] = 0;
    }
}

// the instance's prediction vectors and weights into shared memory
__device__ __forceinline__ void mc_stage_tables(const InstDev& d, double* spv, double* sqw) {
    const Geo& G = d.geo;
    const int npv = G.nsMax * G.nqMax * 4 * G.R, nqw = G.nqMax * G.R;
    for (int e = threadIdx.x; e < npv; e += MC_THREADS) spv[e] = d.pv[e];
    for (int e = threadIdx.x; e < nqw; e += MC_THREADS) sqw[e] = d.qw[e];
    __syncthreads();
}
__device__ __forceinline__ Mc mc_context(const Batch& B, int k, int uin, double* smem) {
    const InstDev& d = B.dev[k];
    InstState& S = B.st[k];
    const long long seg = (long long)B.instTiles[k].x * (TILE_X * TILE_Y);
    const int rank = blockIdx.x % cluster_nctaid(), warp = threadIdx.x >> 5;
    Mc m{d, S, role_ptr(d, S.parity, uin), d.phys};
    m.sch = d.scheme[S.schemeSel];
    int* face = reinterpret_cast<int*>(B.L.face + 2 * seg);  // not used as a face list here
    m.fail = face;
    m.recF[1] = face + 2 * (long long)B.instTiles[k].y * (TILE_X * TILE_Y);
    m.next = reinterpret_cast<int*>(B.L.next + seg);
    m.rec[0] = reinterpret_cast<int*>(B.L.rec + seg);
    m.rec[1] = reinterpret_cast<int*>(B.L.rec2 + seg);
    m.recF[0] = reinterpret_cast<int*>(B.L.recF + seg);
    m.low = reinterpret_cast<int*>(B.L.low + seg);
    m.casc = reinterpret_cast<int*>(B.L.casc + seg);
    m.pRec[0] = d.rec;
    m.pRec[1] = d.recB;
    m.pRecF[0] = d.recF;
    m.pRecF[1] = d.recFB;
    m.buf = smem + warp * MC_BUF;
    m.spv = smem + MC_WARPS * MC_BUF;
    m.sqw = m.spv + MC_PV;
    m.gw = rank * MC_WARPS + warp;
    m.nw = cluster_nctaid() * MC_WARPS;
    m.lane = threadIdx.x & 31;
    m.lead = rank == 0 && threadIdx.x == 0;
    return m;
}
// A cluster is done (its first thread calls): the last one of the launch
// tells the graph, and the host, whether some instance is left to the chain.
__device__ __forceinline__ void mc_done(const Batch& B, bool left, int* out, cudaGraphConditionalHandle h, int set_handle) {
    if (left) atomicOr(&B.flags->mcBig, 1);
    __threadfence();
    if (atomicAdd(&B.flags->mcDone, 1) + 1 == B.maxInst) {
        B.flags->mcDone = 0;
        const int any = atomicExch(&B.flags->mcBig, 0);
        *out = any;
        if (set_handle) cudaGraphSetConditional(h, any ? 1u : 0u);
    }
}

// After pass 1: the stage's scalars, and the face cascade of the instances
// whose failing cells are few, with the fluxes next to the cells it
// re-reconstructed (in pass 1 that is the recompute list the cascade built).
__global__ void __launch_bounds__(MC_THREADS, 1) k_mood_faces(Batch B, int uin, cudaGraphConditionalHandle h,
                                                            int set_handle) { PDL_ENTRY();
    __shared__ double smem[MC_WARPS * MC_BUF + MC_PV + MC_QW];
    const int k = blockIdx.x / cluster_nctaid();
    InstState& S = B.st[k];
    const bool on = S.stepping != 0;
    const bool lead = blockIdx.x % cluster_nctaid() == 0 && threadIdx.x == 0;
    bool left = false;
    if (lead && k == 0) {  // the chain's lists, pass 1's tile counters and the grid barrier start over
        for (int w = 0; w < LIST_N; w++) B.L.counts[w] = 0;
        for (int r = 0; r < 4; r++) B.flags->p1Next[r] = 0;
        B.gbar[0] = 0;
    }
    if (on) {
        const int nF = mc_ld(&S.cFail);
        const bool big = B.mcMax < 0 || nF > B.mcMax;
        if (lead) {
            S.stageActive = 1;
            S.passes = 0;
            S.nInner = 0;
            S.nDetect = 0;
            S.anyFail = big && nF > 0;
            S.cascaded = 0;
            S.big = big;
            S.stages++;
        }
        left = big && nF > 0;
        if (nF > 0) {
            if (big) {
                cluster_sync();  // every block has read cFail
            } else {
                const Mc m = mc_context(B, k, uin, smem);
                mc_stage_tables(m.d, smem + MC_WARPS * MC_BUF, smem + MC_WARPS * MC_BUF + MC_PV);
                cluster_sync();  // every block has read cFail
                int iters = 0;
                const int lowered = mc_cascade(m, nF, 0, false, &iters);
                const int nRec = mc_ld(&S.mc[MC_REC]);
                mc_flux(m, m.rec[0], nRec, m.pRec[0]);
                cluster_sync();
                for (int e = m.gw * 32 + m.lane; e < nRec; e += m.nw * 32) m.pRec[0][m.rec[0][e]] = 0;
                if (lead) {
                    S.mc[MC_REC] = 0;
                    S.nInner = lowered;
                    S.cascadeIters += iters;
                }
            }
            if (lead) S.cFail = 0;
        }
    }
    if (lead) mc_done(B, left, &B.flags->anyCasc, h, set_handle);
}

// After the pass-1 update: the end of pass 1 and every later MOOD pass of the
// instances whose lowered cells are few.
__global__ void __launch_bounds__(MC_THREADS, 1) k_mood_passes(Batch B, int uin, int uout,
                                                             cudaGraphConditionalHandle h, int set_handle) {
    PDL_ENTRY();
    __shared__ double smem[MC_WARPS * MC_BUF + MC_PV + MC_QW];
    const int k = blockIdx.x / cluster_nctaid();
    InstState& S = B.st[k];
    const bool on = S.stepping != 0;
    const bool lead = blockIdx.x % cluster_nctaid() == 0 && threadIdx.x == 0;
    bool left = false;
    if (on) {
        int nLow = mc_ld(&S.nDetect), nCasc = mc_ld(&S.nCasc);
        left = S.big || nLow > B.mcMax;
        if (left) {
            if (lead) {
                S.big = 1;
                S.nCasc = 0;  // the dense flag rebuild clears the cascade's marks
            }
        } else {
            int inner = S.nInner, passes = 1, lastInner = inner, lastDetect = nLow;
            long long innerSum = inner, detectSum = nLow;
            int iters = 0;
            bool capped = false;
            if (nLow > 0 || nCasc > 0) {
                const Mc m = mc_context(B, k, uin, smem);
                mc_stage_tables(m.d, smem + MC_WARPS * MC_BUF, smem + MC_WARPS * MC_BUF + MC_PV);
                const int cap = S.passCap;
                cluster_sync();  // every block has read the scalars
                int cur = 0, nRec = 0, nRecF = 0;
                for (;;) {
                    mc_flags(m, nLow, nCasc, cur, nRec, nRecF);
                    if (nLow == 0) break;
                    cluster_sync();
                    for (int e = m.gw * 32 + m.lane; e < nLow; e += m.nw * 32) m.d.lowered[m.low[e]] = 0;
                    capped = passes >= cap;
                    if (capped) break;
                    // the counters read before the last barrier start over
                    if (lead) {
                        S.nDetect = 0;
                        S.nCasc = 0;
                        S.mc[MC_REC + cur] = 0;
                        S.mc[MC_RECF + cur] = 0;
                    }
                    cur ^= 1;
                    nRec = mc_ld(&S.mc[MC_REC + cur]);
                    mc_recon(m, m.rec[cur], nRec, false, &S.mc[MC_FAIL]);
                    cluster_sync();
                    inner = mc_cascade(m, mc_ld(&S.mc[MC_FAIL]), cur, true, &iters);
                    nRec = mc_ld(&S.mc[MC_REC + cur]);  // with the cascade's
                    nRecF = mc_ld(&S.mc[MC_RECF + cur]);
                    nCasc = mc_ld(&S.nCasc);
                    mc_flux(m, m.rec[cur], nRec, m.pRec[cur]);
                    cluster_sync();
                    mc_update(m, m.recF[cur], nRecF, uout, m.pRecF[cur]);
                    cluster_sync();
                    nLow = mc_ld(&S.nDetect);
                    passes++;
                    lastInner = inner;
                    lastDetect = nLow;
                    innerSum += inner;
                    detectSum += nLow;
                }
            }
            if (lead) {
                for (int w = 0; w < 8; w++) S.mc[w] = 0;
                S.nDetect = 0;
                S.nCasc = 0;
                S.nInner = 0;
                S.passes = passes;
                S.passesTotal += passes;
                S.innerTotal += innerSum;
                S.detectTotal += detectSum;
                S.lastInner = lastInner;
                S.lastDetect = lastDetect;
                S.cascadeIters += iters;
                S.stageActive = 0;
                if (capped) {
                    S.stepping = 0;
                    S.done = 1;
                    S.error = HOSONO_EMOODCAP;
                } else if (passes > S.maxPasses) {
                    S.maxPasses = passes;
                }
            }
        }
    }
    if (lead) mc_done(B, left, &B.flags->anyMood, h, set_handle);
}
