// mood_cluster.cuh -- the short parts of a forward-Euler stage, one thread-
// block cluster per instance (included by kernels.cu): pass 1's face cascade
// (k_mood_faces) and, after the dense pass-1 update, the later MOOD passes
// (k_mood_passes; timeStep.f90:86-128).
//
// What bounds them: latency.  A later pass of a small solve touches a few
// hundred cells; as a chain of grid-wide kernels it cost nine launches (and
// four per cascade iteration) of 3-20 us each, 75 us in all.  Here a pass is
// two phases between hardware cluster barriers (0.6 us each) -- reconstruct,
// test and solve the listed faces; update, detect and flag the listed cells --
// of three or four dependent L2 accesses (0.45 us each), one or two atomics
// and one Riemann solve (2.5 us alone on its scheduler): 13 us for a 64^2
// blast's 200 faces and 150 cells, 19 us for a 128^2 Orszag-Tang's 900 and 640.
// Each item is split over lanes so that a lane's chain is short: a cell's face
// states over 32 lanes (4 faces x 8 variables: 13 loads at R = 2 instead of
// 104), a face's over 8, an updated cell over 8 (its variables), a lowered
// cell's flags over 13 (its diamond).  The lists are per instance (segments of
// the batch's lists that start at the instance's first tile), and hold cell
// indices; a flag's first setter appends its cell, so nothing scans the grid.
// Orders differ from the chain's, values do not: every list is a set, and
// each item's arithmetic is the chain's, statement by statement.
//
// Flags: a pass reads recompute / recomputeFLICD in one pair of planes (rec,
// recF or recB, recFB) and its flag rebuild sets the other, so the old flags
// are cleared beside the next pass's first phase.  Between stages all of them,
// nextPass, fail, lowered and DM_CASC are zero, and so are the counters.
//
// Every branch around a barrier is taken on values all blocks of the cluster
// read alike: a counter is changed only in phases a barrier away from its
// last read, and started over only in phases a barrier away from its next
// addition, so counters come in pairs that the passes (cascade iterations)
// take in turn.  With cur a pass's half, and its phases flux (reconstruct, test,
// solve), then, if cells failed, the cascade's, then update, a barrier after
// each:
//   counter          added to in               read in               back to 0 in
//   LOW[cur]         update                    next flux             next update
//   REC, RECF[cur]   update before, cascade    flux, update          next flux
//   FACE[cur]        update before, cascade    flux, cascade         next flux; cascade, a barrier before its own
//   nCasc            cascade                   update                next flux
//   FAIL, NEXT[it]   flux or iteration it - 1  iteration it          iteration it, a barrier after its read
// (where the lowered cells are listed, their flags are set in a phase of their
// own after update, with a barrier to flux).
#pragma once

constexpr int MC_THREADS = 512, MC_WARPS = MC_THREADS / 32;
enum : int { MC_FAIL = 0, MC_NEXT = 2, MC_REC = 4, MC_RECF = 6, MC_FACE = 8, MC_LOW = 10 };  // InstState::mc, two of each
constexpr int MC_N = 12;                  // counters
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

// What every thread of a block needs, in shared memory: as registers it was
// spilled, and after a barrier spills come back from L2 one by one (a phase of
// a small solve took three times as long).
struct Mc {
    InstHead d;
    InstState* S;
    const double* U;  // the stage input (read only while the kernel runs)
    int8_t* sch;
    int *fail, *next, *rec[2], *recF[2], *low, *casc, *face;  // the instance's lists
    uint8_t *pRec[2], *pRecF[2];                              // flag planes
    double* Uo;                                               // the stage output
    double dtdx, dtdy;
    double bufs[MC_WARPS * MC_BUF];  // the warps' exchange buffers
    double pv[MC_PV], qw[MC_QW];     // prediction vectors and weights
    int faceC[4 * MC_WARPS];         // the block's faces: 2 * right cell + direction, and
    int faceI[4 * MC_WARPS];         // radius | flux << 2 | test left << 3 | test right << 4
};
struct McT {  // a thread's place
    int gw, nw, lane, warp;  // warp of the cluster, warps of the cluster
    bool lead;               // the cluster's first thread
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
// a list to append to, the lanes that do, and what
struct McApp {
    int* list;
    int* counter;
    bool pred;
    int item;
};
// the same on three lists, their counters' atomics in flight together
__device__ __forceinline__ void mc_append3(const McApp& a, const McApp& b, const McApp& c, int lane) {
    const unsigned ma = __ballot_sync(0xffffffffu, a.pred), mb = __ballot_sync(0xffffffffu, b.pred);
    const unsigned mc = __ballot_sync(0xffffffffu, c.pred);
    const unsigned own = lane == 0 ? ma : lane == 1 ? mb : lane == 2 ? mc : 0u;
    int base = 0;
    if (own) base = atomicAdd(lane == 0 ? a.counter : lane == 1 ? b.counter : c.counter, __popc(own));
    const int ba = __shfl_sync(0xffffffffu, base, 0), bb = __shfl_sync(0xffffffffu, base, 1);
    const int bc = __shfl_sync(0xffffffffu, base, 2);
    const unsigned below = (1u << lane) - 1;
    if (a.pred) a.list[ba + __popc(ma & below)] = a.item;
    if (b.pred) b.list[bb + __popc(mb & below)] = b.item;
    if (c.pred) c.list[bc + __popc(mc & below)] = c.item;
}
// set plane[c]; true for the thread that changed it from zero (the byte is
// set through its 32-bit word, so exactly one thread sees it change)
__device__ __forceinline__ bool mc_first(uint8_t* plane, long long c, int bit = 0) {
    const unsigned mask = 1u << (8u * (unsigned)(c & 3) + (unsigned)bit);
    return (atomicOr(reinterpret_cast<unsigned*>(plane + (c - (c & 3))), mask) & mask) == 0;
}
// the radius-2 diamond by lane: the centre, its cross, then the outer ring
__device__ __forceinline__ int diamond_di(int l) { return (int)((0x2204113322132ull >> (4 * l)) & 15) - 2; }
__device__ __forceinline__ int diamond_dj(int l) { return (int)((0x0422131313222ull >> (4 * l)) & 15) - 2; }

// Face states of variable v around cells c[0..NC) at radius RR and quadrature
// points 0..nq-1: sum_k pv(k, q) * U(v, stencil_k), k ascending from zero
// (reconstruct.f90:109-124), one lane per variable; pvf[s]: side s's prediction
// vector of the first point, points qs apart.  The loads of all sides are in
// flight together and their sums interleave.
template <int RR, int NC>
__device__ __forceinline__ void mc_gp(const double* __restrict__ Uv, int pitch, const int (&c)[NC],
                                      const double* const (&pvf)[NC], int qs, int nq, double (&out)[NC][4]) {
    constexpr int NS = 1 + 2 * RR * (RR + 1);
    double u[NC][NS];
#pragma unroll
    for (int n = 0; n < NC; n++) {
        int k = 0;
#pragma unroll
        for (int a = -RR; a <= RR; a++)
#pragma unroll
            for (int b = -RR; b <= RR; b++)
                if (iabs_c(a) + iabs_c(b) <= RR) u[n][k++] = __ldg(Uv + c[n] + b * pitch + a);
    }
#pragma unroll
    for (int q = 0; q <= RR; q++) {  // a face's radius is at least its quadrature's ...
#pragma unroll
        for (int n = 0; n < NC; n++) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < NS; k++) s = s + pvf[n][q * qs + k] * u[n][k];
            out[n][q] = s;
        }
    }
#pragma unroll
    for (int q = RR + 1; q < 4; q++) {  // ... unless a sync left it with an older, smaller one
        if (q >= nq) break;
#pragma unroll
        for (int n = 0; n < NC; n++) {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < NS; k++) s = s + pvf[n][q * qs + k] * u[n][k];
            out[n][q] = s;
        }
    }
}
__device__ __forceinline__ const double* mc_pv(Mc& m, const McT& t, int rr, int f) {
    return m.pv + m.d.geo.nsMax * (m.d.geo.nqMax * (f + 4 * (rr - 1)));
}
// one side, any radius; rr == 0 is the first-order copy
__device__ __forceinline__ void mc_face_states(Mc& m, const McT& t, int rr, int c, int f, int v, int nq, double (&o)[1][4]) {
    const Geo& G = m.d.geo;
    const double* Uv = m.U + v * G.plane;
    if (rr == 0) {
        o[0][0] = o[0][1] = o[0][2] = o[0][3] = __ldg(Uv + c);
        return;
    }
    const int cs[1] = {c};
    const double* const pvf[1] = {mc_pv(m, t, rr, f)};
    if (rr == 1)
        mc_gp<1, 1>(Uv, G.pitch, cs, pvf, G.nsMax, nq, o);
    else if (rr == 2)
        mc_gp<2, 1>(Uv, G.pitch, cs, pvf, G.nsMax, nq, o);
    else
        mc_gp<3, 1>(Uv, G.pitch, cs, pvf, G.nsMax, nq, o);
}

// The faces getFluxes_ recomputes next to a cell of the recompute list
// (getFluxes.f90:27-89), appended to the face list: the cell's west and south
// ones, and the east or north one where the cell beyond is not flagged
// (2 * cell + direction).  One warp per cell, lane 8 f decides face f.
__device__ __forceinline__ void mc_cell_faces(Mc& m, const McT& t, int c, const uint8_t* pRec, int* count) {
    const Geo& G = m.d.geo;
    const int f = t.lane >> 3;
    const bool x = f == EAST || f == WEST;
    const int cf = f == EAST ? c + 1 : f == NORTH ? c + G.pitch : c;  // the face's right / upper cell
    const int j = cell_j(G, cf), i = cf - j * G.pitch;
    bool act = (t.lane & 7) == 0 && i >= G.g - 1 && j >= G.g - 1 && i <= G.g + G.nx + 1 && j <= G.g + G.ny + 1;
    if (act && cf != c) act = pRec[cf] == 0;
    mc_append(m.face, count, act, 2 * cf + (x ? XDIR : YDIR), t.lane);
}

// Re-reconstruct the n cells of the next list (reconstruct_faceValsWithGP's
// inner pass, reconstruct.f90:80-139), one warp per cell: lane 8 f + v sums
// variable v of face f, then lane 8 f + q tests the state at point q.
// Inadmissible cells go on the fail list.
__device__ __forceinline__ void mc_recon(Mc& m, const McT& t, int n, int* failCount) {
    const Geo& G = m.d.geo;
    const int f = t.lane >> 3, v = t.lane & 7;
    double* buf = m.bufs + t.warp * MC_BUF;
    for (int e = t.gw; e < n; e += t.nw) {
        const int c = m.next[e];  // in the reconstruct range
        const int nb = f == NORTH ? c + G.pitch : f == SOUTH ? c - G.pitch : f == EAST ? c + 1 : c - 1;
        const int rr = min((int)m.sch[c], (int)m.sch[nb]);
        const int rN = __shfl_sync(0xffffffffu, rr, 0), rS = __shfl_sync(0xffffffffu, rr, 8);
        const int rE = __shfl_sync(0xffffffffu, rr, 16), rW = __shfl_sync(0xffffffffu, rr, 24);
        if (t.lane == 0) {
            m.d.rrRec[c] = (uint8_t)(rN | (rS << 2) | (rE << 4) | (rW << 6));
            m.d.nextPass[c] = 0;
        }
        if (rr > 0) {
            double o[1][4] = {{0.0, 0.0, 0.0, 0.0}};
            mc_face_states(m, t, rr, c, f, v, rr + 1, o);
#pragma unroll
            for (int q = 0; q < 4; q++) buf[f * MC_FS + q * 8 + v] = o[0][q];
        }
        __syncwarp();
        bool bad = false;
        if (rr > 0 && v <= rr) {
            double u[NCONS];
#pragma unroll
            for (int w = 0; w < NCONS; w++) u[w] = buf[f * MC_FS + v * 8 + w];
            bad = !admissible(u[DENS], cons2pres(m.d.phys, u));
        }
        const bool any = __any_sync(0xffffffffu, bad);
        mc_append(m.fail, failCount, any && t.lane == 0, c, t.lane);
        __syncwarp();
    }
}

// The serial lowering loop of reconstruct.f90:146-169 for the n cells of the
// fail list, one warp per cell (order independent: a cell lowers only its own
// scheme; every flag write sets): gridBlock_lowerOrder (gridBlock.f90:194-235)
// and the cross marked for the next inner pass.  withF: recomputeFLICD too
// (in pass 1 it is set everywhere).
__device__ __forceinline__ void mc_lower(Mc& m, const McT& t, int n, int cur, bool withF, int* nextCount) {
    const Geo& G = m.d.geo;
    const int l = t.lane;
    const int di = l < 13 ? diamond_di(l) : 0, dj = l < 13 ? diamond_dj(l) : 0;
    for (int e = t.gw; e < n; e += t.nw) {
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
        mc_append(m.casc, &m.S->nCasc, first, c, l);
        const int ii = i + di, jj = j + dj, cn = c + dj * G.pitch + di;
        const bool in = l < 13 && ii >= 0 && jj >= 0 && ii < G.nxt && jj < G.nyt;
        const bool range = ii >= G.g - 2 && jj >= G.g - 2 && ii <= G.g + G.nx + 1 && jj <= G.g + G.ny + 1;
        const bool r = in && l < 5 && mc_first(m.pRec[cur], cn);
        const bool n = in && l < 5 && range && mc_first(m.d.nextPass, cn);
        const bool rf = withF && in && mc_first(m.pRecF[cur], cn);
        mc_append3({m.rec[cur], &m.S->mc[MC_REC + cur], r, cn}, {m.next, nextCount, n, cn},
                   {m.recF[cur], &m.S->mc[MC_RECF + cur], rf, cn}, l);
    }
}

// The face cascade (reconstruct.f90:143-171) from nF failing cells; returns
// the lowerings.  All blocks enter with the same nF, a barrier after the
// fail list was filled.
__device__ __forceinline__ int mc_cascade(Mc& m, const McT& t, int nF, int cur, bool withF, int* iters) {
    int sum = 0;
    for (int it = 0; nF > 0; it++) {
        int* nextCount = &m.S->mc[MC_NEXT + (it & 1)];
        mc_lower(m, t, nF, cur, withF, nextCount);
        sum += nF;
        ++*iters;
        cluster_sync();
        const int nN = mc_ld(nextCount);
        mc_recon(m, t, nN, &m.S->mc[MC_FAIL + ((it + 1) & 1)]);
        if (t.lead) m.S->mc[MC_FAIL + (it & 1)] = 0;  // read before the last barrier
        cluster_sync();
        nF = mc_ld(&m.S->mc[MC_FAIL + ((it + 1) & 1)]);
        if (t.lead) *nextCount = 0;
    }
    return sum;
}

// the face list of the n cells of the recompute list from scratch (after a
// cascade, which flags more cells)
__device__ __forceinline__ void mc_faces(Mc& m, const McT& t, const int* list, int n, const uint8_t* pRec, int* count) {
    for (int e = t.gw; e < n; e += t.nw) mc_cell_faces(m, t, list[e], pRec, count);
}

// getFluxes_ (getFluxes.f90:16-90) on the n faces of the face list, 8 lanes
// per face: lane v sums variable v of both face states; then a thread of the
// block's first warps solves the Riemann problem of each face and point (a
// warp's own faces would keep eight to sixteen lanes of every warp busy); lane
// v adds the Gauss sum of flux v in quadrature order.  Face states are rebuilt at the radius each side was last
// reconstructed with (rrRec), the quadrature uses the face's current radius
// (riemannSolver.f90:23-47), as in flux_list.
// FIRST: the start of a later pass, reconstruct_faceValsWithGP's first inner
// pass (reconstruct.f90:80-139) in one with it: a side whose cell is on the
// recompute list takes the face's current radius and is tested (a cell that
// fails goes on the fail list, and the cascade's fluxes replace these); the
// list also holds the faces just outside the flux range, tested only.
__device__ __forceinline__ bool mc_in_recon(const Geo& G, int i, int j) {
    return i >= G.g - 2 && j >= G.g - 2 && i <= G.g + G.nx + 1 && j <= G.g + G.ny + 1;
}
__device__ __forceinline__ void mc_fail(Mc& m, int c) {
    if (mc_first(m.d.fail, c)) m.fail[atomicAdd(&m.S->mc[MC_FAIL], 1)] = c;
}
template <bool FIRST>
__device__ __forceinline__ void mc_flux(Mc& m, const McT& t, int n, int cur) {
    const Geo& G = m.d.geo;
    const int g8 = t.lane >> 3, v = t.lane & 7;
    double* buf = m.bufs + t.warp * MC_BUF + g8 * MC_FS;
    const int nq = G.nqMax;
    for (int b0 = 0; b0 < n; b0 += 4 * t.nw) {
        // a warp's faces of the round: over the warps first, up to four each
        const int e = b0 + t.gw + g8 * t.nw;
        const bool act = e < n;
        const int slot = g8 * MC_WARPS + t.warp;  // in the block: filled from 0 up
        int rr = 0, cf = 0, vf = v;
        bool x = true, flux = act;
        if (act) {
            const int it = m.face[e];
            cf = it >> 1;
            x = (it & 1) == XDIR;
            // variable v's place in face coordinates (physics.cuh)
            vf = x ? v : v == MOMX || v == MAGX ? v + 1 : v == MOMY || v == MAGY ? v - 1 : v;
            const int cl = x ? cf - 1 : cf - G.pitch;
            const int fL = x ? EAST : NORTH, fR = x ? WEST : SOUTH;
            rr = min((int)m.sch[cf], (int)m.sch[cl]);
            int rrL = (m.d.rrRec[cl] >> (2 * fL)) & 3, rrR = (m.d.rrRec[cf] >> (2 * fR)) & 3;
            bool recL = false, recR = false;
            if (FIRST) {
                const int j = cell_j(G, cf), i = cf - j * G.pitch;
                flux = i >= G.g - 1 && j >= G.g - 1 && i <= G.g + G.nx + 1 && j <= G.g + G.ny + 1;
                recL = m.pRec[cur][cl] != 0 && mc_in_recon(G, x ? i - 1 : i, x ? j : j - 1);
                recR = m.pRec[cur][cf] != 0 && mc_in_recon(G, i, j);
                rrL = recL ? rr : rrL;
                rrR = recR ? rr : rrR;
                if (v == 0) m.d.dirty[cf] = 0;  // the face's mark
            }
            if (v == 0) {
                m.faceC[slot] = it;
                m.faceI[slot] = rr | (flux ? 4 : 0) | (recL ? 8 : 0) | (recR ? 16 : 0);
            }
            const double* Uv = m.U + v * G.plane;
            if (flux && rrL == rrR && (rrL == 1 || rrL == 2)) {  // nearly every face
                double o[2][4] = {};
                const int cs[2] = {cl, cf};
                const double* const pvf[2] = {mc_pv(m, t, rrL, fL), mc_pv(m, t, rrL, fR)};
                if (rrL == 1)
                    mc_gp<1, 2>(Uv, G.pitch, cs, pvf, G.nsMax, rr + 1, o);
                else
                    mc_gp<2, 2>(Uv, G.pitch, cs, pvf, G.nsMax, rr + 1, o);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    buf[2 * q * 8 + vf] = o[0][q];
                    buf[(2 * q + 1) * 8 + vf] = o[1][q];
                }
            } else {
#pragma unroll 1
                for (int side = 0; side < 2; side++) {
                    if (!(flux || (side ? recR : recL))) continue;
                    double o[1][4] = {};
                    mc_face_states(m, t, side ? rrR : rrL, side ? cf : cl, side ? fR : fL, v, rr + 1, o);
#pragma unroll
                    for (int q = 0; q < 4; q++) buf[(2 * q + side) * 8 + vf] = o[0][q];
                }
            }
        }
        __syncthreads();
        // the block's Riemann problems on as few warps as hold them: the slots
        // are filled in the list's order, block after block
        const int nct = t.nw / MC_WARPS, left = n - b0 - t.gw % nct;
        const int faces = min(left > 0 ? (left + nct - 1) / nct : 0, 4 * MC_WARPS);
        if ((int)threadIdx.x < faces * nq) {
            const int k = (int)threadIdx.x / nq, q = (int)threadIdx.x - k * nq;
            const int info = m.faceI[k], rq = info & 3;
            double* st = m.bufs + (k % MC_WARPS) * MC_BUF + (k / MC_WARPS) * MC_FS + 16 * q;
            if (q <= rq) {
                bool badL = false, badR = false;
                double uL[NCONS], uR[NCONS];
#pragma unroll
                for (int w = 0; w < NCONS; w++) {
                    uL[w] = st[w];
                    uR[w] = st[8 + w];
                }
                if (info & 4) {
                    double F[NCONS];
                    bool admL, admR;
                    hllc_face(m.d.phys, uL, uR, F, admL, admR);
                    badL = !admL;
                    badR = !admR;
#pragma unroll
                    for (int w = 0; w < NCONS; w++) st[w] = F[w];
                } else if (FIRST) {  // a side that is not tested holds no state
                    if (info & 8) badL = !admissible(uL[DENS], cons2pres(m.d.phys, uL));
                    if (info & 16) badR = !admissible(uR[DENS], cons2pres(m.d.phys, uR));
                }
                if (FIRST && rq > 0) {
                    const int it = m.faceC[k], c = it >> 1;
                    if ((info & 8) && badL) mc_fail(m, (it & 1) == XDIR ? c - 1 : c - G.pitch);
                    if ((info & 16) && badR) mc_fail(m, c);
                }
            }
        }
        __syncthreads();
        if (act && flux) {
            double s;
            if (rr == 0) {
                s = buf[vf];
            } else {
                s = 0.0;
                for (int q = 0; q <= rr; q++) s = s + m.qw[q + G.nqMax * (rr - 1)] * buf[16 * q + vf];
            }
            (x ? m.d.FX : m.d.FY)[v * G.plane + cf] = s;
            if (v == (x ? MAGY : MAGX)) (x ? m.d.CTX : m.d.CTY)[cf] = s;
        }
        __syncthreads();  // the buffers are read before the next round fills them
    }
}
// the radii the cells of the recompute list were reconstructed with, one
// thread per cell (a face next to a listed cell does not read its entry)
__device__ __forceinline__ void mc_record(Mc& m, const McT& t, const int* list, int n) {
    const Geo& G = m.d.geo;
    // from the last warp down: the first ones have most faces to solve
    for (int e = (t.nw - 1 - t.gw) * 32 + t.lane; e < n; e += t.nw * 32) {
        const int c = list[e];
        const int j = cell_j(G, c), i = c - j * G.pitch;
        if (!mc_in_recon(G, i, j)) continue;
        const int s = m.sch[c];
        const int rN = min(s, (int)m.sch[c + G.pitch]), rS = min(s, (int)m.sch[c - G.pitch]);
        const int rE = min(s, (int)m.sch[c + 1]), rW = min(s, (int)m.sch[c - 1]);
        m.d.rrRec[c] = (uint8_t)(rN | (rS << 2) | (rE << 4) | (rW << 6));
    }
}

// A cell detect lowered sets its flags for the next pass: the cross and the
// diamond of each of its translates (gridBlock_lowerOrder with
// boundaryConditions_applyMOOD's periodic sync) in the other pair of planes,
// and marks the sixteen faces around the cross (bit dir of the `dirty` plane),
// each first setter appending to its list.  One warp; `members`: the
// translates in the array (bit 3 (tb + 1) + tt + 1).
__device__ __forceinline__ void mc_scatter(Mc& m, const McT& t, int i, int j, unsigned members, int cur) {
    const Geo& G = m.d.geo;
    const int l = t.lane;
    const int di = l < 13 ? diamond_di(l) : 0, dj = l < 13 ? diamond_dj(l) : 0;
    // face l < 16: along the direction dir = l / 8 -1, 0, 1, 2 in the cell's
    // own row, then 0, 1 in the rows on either side
    const int dir = (l >> 3) & 1, k8 = l & 7;
    const int along = k8 < 4 ? k8 - 1 : k8 & 1, across = k8 < 4 ? 0 : k8 < 6 ? 1 : -1;
    const int fi = dir == XDIR ? along : across, fj = dir == XDIR ? across : along;
    while (members) {
        const int k = __ffs(members) - 1;
        members &= members - 1;
        const int ci = i + (k % 3 - 1) * G.nx, cj = j + (k / 3 - 1) * G.ny;
        const int ii = ci + di, jj = cj + dj;
        const int cn = jj * G.pitch + ii;
        const bool in = l < 13 && ii >= 0 && jj >= 0 && ii < G.nxt && jj < G.nyt;
        // faces next to a cell of the reconstruct range
        const int xi = ci + fi, xj = cj + fj, xc = xj * G.pitch + xi;
        const bool fin = l < 16 && xi >= G.g - 2 && xj >= G.g - 2 && xi <= G.g + G.nx + 1 + (dir == XDIR ? 1 : 0) &&
                         xj <= G.g + G.ny + 1 + (dir == YDIR ? 1 : 0);
        const bool r = in && l < 5 && mc_first(m.pRec[cur ^ 1], cn);
        const bool rf = in && mc_first(m.pRecF[cur ^ 1], cn);
        const bool fc = fin && mc_first(m.d.dirty, xc, dir);
        mc_append3({m.rec[cur ^ 1], &m.S->mc[MC_REC + (cur ^ 1)], r, cn},
                   {m.recF[cur ^ 1], &m.S->mc[MC_RECF + (cur ^ 1)], rf, cn},
                   {m.face, &m.S->mc[MC_FACE + (cur ^ 1)], fc, 2 * xc + dir}, l);
    }
}
// this lane's translate of cell (i, j): whether it lies in the array, and its index
__device__ __forceinline__ bool mc_translate(Mc& m, const McT& t, int i, int j, int* co) {
    const Geo& G = m.d.geo;
    const int l = t.lane, reach = G.bc == 1 ? 1 : 0;
    const int tb = l < 9 ? l / 3 - 1 : 2, tt = l < 9 ? l % 3 - 1 : 2;
    const int jo = j + tb * G.ny, io = i + tt * G.nx;
    *co = jo * G.pitch + io;
    return l < 9 && iabs_c(tb) <= reach && iabs_c(tt) <= reach && jo >= 0 && io >= 0 && jo < G.nyt && io < G.nxt;
}

// FLICD, the update (timeStep.f90:107-118) and detect_ALL on the n cells of
// the recomputeFLICD list, 8 lanes per cell: lane v updates variable v (the
// MAGX and MAGY lanes also correct the cell's fluxes, as ct_cell does), the
// group's first lane runs the per-pass tests.  flags: no cell was lowered by
// the cascade in this pass, so the translates of a cell share its scheme and
// the flag rebuild needs nothing but the cell: it is done here, by the warp.
// Else (`low` list, `lowered` marks) mc_flags does it after a barrier.
__device__ __forceinline__ void mc_update(Mc& m, const McT& t, const int* list, int n, int cur, bool flags) {
    const InstHead& d = m.d;
    const Geo& G = d.geo;
    const uint8_t* pRecF = m.pRecF[cur];
    const int v = t.lane & 7, base = t.lane & ~7;
    const double* fxy = d.FX + MAGY * G.plane;
    const double* fyx = d.FY + MAGX * G.plane;
    for (int e0 = t.gw; e0 < n; e0 += t.nw * 4) {
        const int e = e0 + (t.lane >> 3) * t.nw;
        int c = 0, i = 0, j = 0;
        bool in = false, cell = false;
        if (e < n) {
            c = list[e];
            j = cell_j(G, c);
            i = c - j * G.pitch;
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
        const int sch = cell ? m.sch[c] : 0;
        int mask = 0;
        double rho[5] = {};
        if (cell && v == 0) {
            const double* r = m.U + DENS * G.plane + c;
            mask = d.detMask[c];
            rho[0] = __ldg(r);
            rho[1] = __ldg(r + 1);
            rho[2] = __ldg(r - 1);
            rho[3] = __ldg(r + G.pitch);
            rho[4] = __ldg(r - G.pitch);
        }
        if (cell) {
            un = __ldg(m.U + v * G.plane + c) - m.dtdx * (f1 - f0) - m.dtdy * (g1 - g0);
            m.Uo[v * G.plane + c] = un;
        }
        double u[NCONS];
#pragma unroll
        for (int w = 0; w < NCONS; w++) u[w] = __shfl_sync(0xffffffffu, un, base + w);
        bool low = false;
        if (cell && v == 0 && sch > 0) {
            const double msq = (0.0 + u[MOMX] * u[MOMX]) + u[MOMY] * u[MOMY] + u[MOMZ] * u[MOMZ];
            const double bsq = (0.0 + u[MAGX] * u[MAGX]) + u[MAGY] * u[MAGY] + u[MAGZ] * u[MAGZ];
            low = detect_decide(m.d.phys, mask, rho, NewState{u[DENS], msq, bsq, u[ENER]});
        }
        if (flags) {
            unsigned lows = __ballot_sync(0xffffffffu, low);
            if (lows && t.lane == 0) atomicAdd(&m.S->mc[MC_LOW + cur], __popc(lows));
            while (lows) {  // the warp takes its lowered cells in turn
                const int src = __ffs(lows) - 1;
                lows &= lows - 1;
                const int ci = __shfl_sync(0xffffffffu, i, src), cj = __shfl_sync(0xffffffffu, j, src);
                const int cs = __shfl_sync(0xffffffffu, sch, src);
                int co;
                const bool mem = mc_translate(m, t, ci, cj, &co);
                if (mem) m.sch[co] = (int8_t)(cs - 1);
                mc_scatter(m, t, ci, cj, __ballot_sync(0xffffffffu, mem), cur);
            }
        } else {
            if (low) d.lowered[c] = 1;
            mc_append(m.low, &m.S->mc[MC_LOW + cur], low, c, t.lane);
        }
    }
}

// The flag rebuild after detect, from the lists (pass 1, and passes whose
// cascade lowered cells): each lowered cell's flags, and one scheme per
// translate class of each cell the pass lowered, the minimum over the class
// of (scheme - lowered)^+.  One warp per cell.  A class holds one interior
// cell, so at most one entry of the low list; that entry alone takes a class
// detect lowered, and the cascade's entries of other classes all write the
// same minimum, which a partly written class still has.
__device__ __forceinline__ void mc_flags(Mc& m, const McT& t, int nLow, int nCasc, int cur) {
    const InstHead& d = m.d;
    const Geo& G = d.geo;
    for (int e = t.gw; e < nLow + nCasc; e += t.nw) {
        const bool fromLow = e < nLow;
        const int c = fromLow ? m.low[e] : m.casc[e - nLow];
        const int j = cell_j(G, c), i = c - j * G.pitch;
        int co;
        const bool mem = mc_translate(m, t, i, j, &co);
        int s = 127, lo = 0;
        if (mem) {
            s = m.sch[co];
            lo = d.lowered[co];
        }
        const bool classLow = __any_sync(0xffffffffu, lo != 0);
        if (mem) s = max(s - lo, 0);
        s = __reduce_min_sync(0xffffffffu, s);
        if (mem && (fromLow || !classLow)) m.sch[co] = (int8_t)s;
        if (!fromLow) {
            if (t.lane == 0) d.detMask[c] &= (uint8_t)~DM_CASC;
            continue;
        }
        mc_scatter(m, t, i, j, __ballot_sync(0xffffffffu, mem), cur);
    }
}
// the flags of a list's cells back to zero
__device__ __forceinline__ void mc_clear(Mc& m, const McT& t, uint8_t* plane, const int* list, int n) {
    for (int e = t.gw * 32 + t.lane; e < n; e += t.nw * 32) plane[list[e]] = 0;
}

// The cascade of a later pass, and every flux next to the cells it leaves on
// the recompute list; (lowerings, iterations).  Rare, so out of line: inlined
// it took registers from the common path.
static __device__ __noinline__ int2 mc_cascade_later(Mc* mp, McT t, int nFail, int cur) {
    Mc& m = *mp;
    int iters = 0;
    const int inner = mc_cascade(m, t, nFail, cur, true, &iters);
    const int nRec = mc_ld(&m.S->mc[MC_REC + cur]);
    if (t.lead) m.S->mc[MC_FACE + cur] = 0;  // the faces next to them, afresh
    cluster_sync();
    mc_faces(m, t, m.rec[cur], nRec, m.pRec[cur], &m.S->mc[MC_FACE + cur]);
    cluster_sync();
    mc_flux<false>(m, t, mc_ld(&m.S->mc[MC_FACE + cur]), cur);
    cluster_sync();
    return make_int2(inner, iters);
}

// fill the block's Mc for instance k (every thread calls)
__device__ __forceinline__ void mc_setup(const Batch& B, int k, int uin, int uout, Mc& m) {
    const InstDev& d = B.dev[k];
    const InstState& S = B.st[k];
    const Geo& G = d.geo;
    const int* src = reinterpret_cast<const int*>(static_cast<const InstHead*>(&d));
    int* dst = reinterpret_cast<int*>(&m.d);
    for (int e = threadIdx.x; e < (int)(sizeof(InstHead) / sizeof(int)); e += MC_THREADS) dst[e] = src[e];
    const int npv = G.nsMax * G.nqMax * 4 * G.R, nqw = G.nqMax * G.R;
    for (int e = threadIdx.x; e < npv; e += MC_THREADS) m.pv[e] = d.pv[e];
    for (int e = threadIdx.x; e < nqw; e += MC_THREADS) m.qw[e] = d.qw[e];
    if (threadIdx.x == 0) {
        const long long seg = (long long)B.instTiles[k].x * (TILE_X * TILE_Y);
        const long long cells = (long long)B.instTiles[k].y * (TILE_X * TILE_Y);
        m.S = B.st + k;
        m.U = role_ptr(d, S.parity, uin);
        m.Uo = role_ptr(d, S.parity, uout);
        m.dtdx = S.dtdx;
        m.dtdy = S.dtdy;
        m.sch = d.scheme[S.schemeSel];
        // the segment of the batch's face list holds 2 entries of 2 ints a cell
        int* face = reinterpret_cast<int*>(B.L.face + 2 * seg);
        m.fail = face;
        m.recF[1] = face + cells;
        m.face = face + 2 * cells;
        m.next = reinterpret_cast<int*>(B.L.next + seg);
        // both recompute lists in the batch's free one: the other holds the chain's
        // cells for its next pass when instances are handed over
        m.rec[0] = reinterpret_cast<int*>(rec_list(B, true) + seg);
        m.rec[1] = m.rec[0] + cells;
        m.recF[0] = reinterpret_cast<int*>(B.L.recF + seg);
        m.low = reinterpret_cast<int*>(B.L.low + seg);
        m.casc = reinterpret_cast<int*>(B.L.casc + seg);
        m.pRec[0] = d.rec;
        m.pRec[1] = d.recB;
        m.pRecF[0] = d.recF;
        m.pRecF[1] = d.recFB;
    }
    __syncthreads();
}
// the cluster's slot (-1: none)
__device__ __forceinline__ int mc_slot(const Batch& B) {
    const int n = blockIdx.x / cluster_nctaid();
    return B.mcSlots ? B.mcSlots[n] : n;
}
__device__ __forceinline__ McT mc_place() {
    McT t;
    const int rank = blockIdx.x % cluster_nctaid();
    t.warp = threadIdx.x >> 5;
    t.gw = t.warp * (int)cluster_nctaid() + rank;  // a short list spreads over every block
    t.nw = cluster_nctaid() * MC_WARPS;
    t.lane = threadIdx.x & 31;
    t.lead = rank == 0 && threadIdx.x == 0;
    return t;
}
// A cluster is done (its first thread calls): the last one of the launch
// tells the graph, and the host, whether some instance is left to the chain.
__device__ __forceinline__ void mc_done(const Batch& B, bool left, int* out, cudaGraphConditionalHandle h, int set_handle) {
    if (left) atomicOr(&B.flags->mcBig, 1);
    __threadfence();
    if (atomicAdd(&B.flags->mcDone, 1) + 1 == mc_clusters(B)) {
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
    __shared__ Mc m;
    const McT t = mc_place();
    const int slot = mc_slot(B), k = max(slot, 0);
    InstState& S = B.st[k];
    const bool on = slot >= 0 && S.stepping != 0;
    const bool lead = t.lead;
    bool left = false;
    if (lead && blockIdx.x == 0) {  // the chain's lists, pass 1's tile counters and the grid barrier start over
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
                mc_setup(B, k, uin, uin, m);
                cluster_sync();  // every block has read cFail
                int iters = 0;
                const int lowered = mc_cascade(m, t, nF, 0, false, &iters);
                const int nRec = mc_ld(&S.mc[MC_REC]);
                mc_faces(m, t, m.rec[0], nRec, m.pRec[0], &S.mc[MC_FACE]);
                cluster_sync();
                mc_clear(m, t, m.pRec[0], m.rec[0], nRec);
                mc_flux<false>(m, t, mc_ld(&S.mc[MC_FACE]), 0);
                cluster_sync();
                if (lead) {
                    S.mc[MC_REC] = 0;
                    S.mc[MC_FACE] = 0;
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
// instances whose lowered cells are few.  REST: in the chain's loop, the passes
// left of the instances it hands over (hand_over), from the lists k_handover
// made.
template <bool REST>
__global__ void __launch_bounds__(MC_THREADS, 1) k_mood_passes(Batch B, int uin, int uout,
                                                             cudaGraphConditionalHandle h, int set_handle) {
    PDL_ENTRY();
    __shared__ Mc m;
    const McT t = mc_place();
    const int slot = mc_slot(B), k = max(slot, 0);
    InstState& S = B.st[k];
    const bool on = slot >= 0 && S.stepping != 0 && (!REST || S.hand);
    const bool lead = t.lead;
    bool left = false;
    if (on) {
        int nLow = mc_ld(REST ? &S.cLow : &S.nDetect), nCasc = mc_ld(&S.nCasc);
        left = !REST && (S.big || nLow > B.mcMax);
        if (left) {
            if (lead) {
                S.big = 1;
                S.nCasc = 0;  // the dense flag rebuild clears the cascade's marks
            }
        } else {
            const int before = REST ? S.passes : 0;  // passes the chain has counted
            int inner = S.nInner, passes = REST ? before : 1, lastInner = inner, lastDetect = nLow;
            long long innerSum = inner, detectSum = REST ? 0 : nLow;
            int iters = 0;
            bool capped = false;
            if (nLow > 0 || nCasc > 0) {
                mc_setup(B, k, uin, uout, m);
                const int cap = S.passCap;
                if (REST) {
                    const int* cascRest = m.next + (long long)B.instTiles[k].y * (TILE_X * TILE_Y);
                    for (int e = t.gw * 32 + t.lane; e < nLow; e += t.nw * 32) m.low[e] = m.next[e];
                    for (int e = t.gw * 32 + t.lane; e < nCasc; e += t.nw * 32) m.casc[e] = cascRest[e];
                }
                cluster_sync();  // every block has read the scalars
                int cur = 0, nRec = 0, nRecF = 0;
                bool listed = true;  // the last pass's lowerings are on the low and cascade lists
                for (;;) {
                    if (listed) mc_flags(m, t, nLow, nCasc, cur);
                    if (nLow == 0) {
                        mc_clear(m, t, m.pRec[cur], m.rec[cur], nRec);
                        mc_clear(m, t, m.pRecF[cur], m.recF[cur], nRecF);
                        break;
                    }
                    capped = passes >= cap;
                    if (listed || capped) cluster_sync();  // capped: every block has read nLow
                    if (listed)
                        for (int e = t.gw * 32 + t.lane; e < nLow; e += t.nw * 32) m.d.lowered[m.low[e]] = 0;
                    if (capped) break;  // (the next stage's pass 1 clears the flag planes)
                    // the old flags, and the counters every block has read a
                    // barrier ago, start over
                    mc_clear(m, t, m.pRec[cur], m.rec[cur], nRec);
                    mc_clear(m, t, m.pRecF[cur], m.recF[cur], nRecF);
                    if (lead) {
                        S.nCasc = 0;
                        S.mc[MC_REC + cur] = 0;
                        S.mc[MC_RECF + cur] = 0;
                        S.mc[MC_FACE + cur] = 0;
                    }
                    cur ^= 1;
                    nRec = mc_ld(&S.mc[MC_REC + cur]);
                    mc_record(m, t, m.rec[cur], nRec);
                    mc_flux<true>(m, t, mc_ld(&S.mc[MC_FACE + cur]), cur);
                    cluster_sync();
                    const int nFail = mc_ld(&S.mc[MC_FAIL]);
                    if (lead) S.mc[MC_LOW + (cur ^ 1)] = 0;  // nLow was read before this barrier
                    inner = 0;
                    if (nFail > 0) {
                        const int2 r = mc_cascade_later(&m, t, nFail, cur);
                        inner = r.x;
                        iters += r.y;
                        nRec = mc_ld(&S.mc[MC_REC + cur]);  // with the cascade's
                    }
                    nRecF = mc_ld(&S.mc[MC_RECF + cur]);
                    nCasc = mc_ld(&S.nCasc);
                    listed = nCasc > 0;
                    mc_update(m, t, m.recF[cur], nRecF, cur, !listed);
                    cluster_sync();
                    nLow = mc_ld(&S.mc[MC_LOW + cur]);
                    passes++;
                    lastInner = inner;
                    lastDetect = nLow;
                    innerSum += inner;
                    detectSum += nLow;
                }
            }
            if (lead) {
                for (int w = 0; w < MC_N; w++) S.mc[w] = 0;
                S.nDetect = 0;
                S.nCasc = 0;
                S.nInner = 0;
                S.cLow = 0;
                S.hand = 0;
                S.passes = passes;
                S.passesTotal += passes - before;
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
