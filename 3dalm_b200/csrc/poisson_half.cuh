// One half of a Jacobi(3)-preconditioned BiCGStab iteration in one pass
// (run_pbicgstab, src/eq.h:333-473, fast arithmetic), for one thread block.
//
//   P half: p = r + beta (p - omega q)             (src/eq.h:355-365)
//           pp = M^-1 p: Jacobi from zero, 3 sweeps (src/eq.h:367-368)
//           q = A pp, <r0, q>                      (src/eq.h:369-371)
//   S half: s = r - alpha q                        (src/eq.h:373-377)
//           ss = M^-1 s                            (src/eq.h:379-380)
//           t = A ss, <t, s>, <t, t>               (src/eq.h:381-383)
//
// The sweeps are written on the off-diagonal part: with R x = A x - a_c x
// the first sweep from zero is w1 = v / a_c, and x + (v - A x) / a_c is
// w1 - R x / a_c, so neither the right-hand side nor the centre value is
// needed again.
//
// A block owns tiles of the (j, k) plane and marches through their i-planes.
// The box of a tile (ROWS rows of W cells, three cells of halo around the
// tile) is held by the block's threads, each M cells of one column k in
// consecutive rows: a thread carries its cells through all four phases and
// through i in registers, and only the k +- 1 neighbours and the row above and
// below its own go through shared memory.  Step L of the march takes plane L
// from the ring of TMA stages and computes
//   phase 1: v, w1             on plane L       (needs the inputs only)
//   phase 2: w2 = w1 - R w1/a  on plane L - 1   (w1 of planes L-2, L-1, L)
//   phase 3: w3 = w1 - R w2/a  on plane L - 2
//   phase 4: A w3, the sums    on plane L - 3
// A phase's i + 1 operand is the value the thread has just computed for that
// cell, and its in-plane neighbours were stored in the step before, so one
// barrier per step is enough and the four phases of the M cells are
// independent up to that one value: their latencies overlap.
//
// What bounds it: latency.  On 256 x 128 x 128 the four warps of a scheduler
// (register-limited: 128 a thread) issue in half of the cycles, the FP64 pipe
// is a quarter busy and DRAM half.  Measured slower: patches of 2 x 2 cells
// with 16-byte accesses and 12 warps (P 262, S 217 us on 512 x 256 x 128
// against 263 and 200), and the march unrolled by three so that no register is
// moved (329 and 197; spills).  Inputs brought by each thread's own cp.async
// instead of TMA cost 9 % of an iteration.
//
// Cells outside the interior come out as 0 in every phase, the value of the
// vectors' guide cells: those are never written, TMA fills with zeros outside
// the stored grid, and such a cell's coefficients are set to 0 and its
// diagonal is not.
#pragma once

#include "poisson.cuh"
#include "poisson_math.cuh"

namespace dalm {
namespace {

enum HalfKind { HALF_P = 0, HALF_S = 1 };

constexpr int HH = 3;           // halo: two stencil sweeps and A w3
constexpr int HALF_MAXP = 122;  // planes of one march: longer ranges are split

// W: cells per row of the box (from four cells below the tile, so that a tile
// that starts on an even cell starts its TMA box on a 16-byte boundary); M
// rows per thread.
template <int W_, int ROWS_, int M_>
struct HalfGeo {
    static constexpr int W = W_, ROWS = ROWS_, M = M_;
    static constexpr int NT = W * (ROWS / M);              // threads with cells
    static constexpr int THREADS = (NT + 31) / 32 * 32;
    static constexpr int CELLS = W * ROWS;
    static constexpr int BK = W - 8, BJ = ROWS - 2 * HH;   // largest tile
    static constexpr int BOX = CELLS * 8;                  // bytes of a TMA box
    static constexpr int STAGE = (BOX + 127) / 128 * 128;  // ... in the ring
    static constexpr int NS_P = 3, NS_S = 4;               // planes in flight
    static constexpr int RING = (NS_P * 3 > NS_S * 2 ? NS_P * 3 : NS_S * 2) * STAGE;
    static constexpr int PLANE = CELLS + 2 * W;            // a guard row on both sides
    static constexpr int COEF = 3 * (HALF_MAXP + 2 * HH);
    static constexpr int SMEM = RING + (6 * PLANE + COEF) * 8;
    static_assert(ROWS % M == 0 && SMEM <= 226 * 1024, "block shape");
};
// Tiles of up to 64 x 15 cells, and of 32 x 18 for grids at most 32 cells high;
// 16 and 15 warps: a seventeenth warp would leave a thread 96 registers
// instead of 128.
using HalfWide = HalfGeo<WIDE_BOX_K, WIDE_BOX_J, 3>;
using HalfNarrow = HalfGeo<NARROW_BOX_K, NARROW_BOX_J, 2>;

// The interior cut into ntj x ntk tiles (balanced, at most BJ x BK) of ni
// planes each.  Work unit u = tile * ni + plane: a block takes a contiguous
// range of units, so any number of blocks is loaded evenly.
struct HalfPlan {
    Box box;
    int ntj, ntk, ni;
    long long units;
    __host__ __device__ static HalfPlan make(const Box &b, int bj, int bk) {
        HalfPlan p;
        p.box = b;
        p.ni = b.hi[0] - b.lo[0];
        p.ntj = (b.hi[1] - b.lo[1] + bj - 1) / bj;
        p.ntk = (b.hi[2] - b.lo[2] + bk - 1) / bk;
        p.units = (long long)p.ntj * p.ntk * p.ni;
        return p;
    }
    // a tile's cells; k0 at an even distance from the interior's first cell
    __host__ __device__ void tile_range(int tj, int tk, int &j0, int &j1, int &k0, int &k1) const {
        const int nj = box.hi[1] - box.lo[1], nk = box.hi[2] - box.lo[2], hk = (nk + 1) / 2;
        j0 = box.lo[1] + (int)((long long)tj * nj / ntj);
        j1 = box.lo[1] + (int)((long long)(tj + 1) * nj / ntj);
        k0 = box.lo[2] + 2 * (int)((long long)tk * hk / ntk);
        k1 = box.lo[2] + 2 * (int)((long long)(tk + 1) * hk / ntk);
        if (k1 > box.hi[2]) k1 = box.hi[2];
    }
};

struct HalfArgs {  // beside the inputs' TMA maps, P: r, old p, old q;  S: r, q
    const double *r0;    // P
    double *v, *w, *av;  // P: new p, pp, new q;  S: s, ss, t
};

// The barriers of the ring of TMA stages, initialised once per kernel, and a
// bit per stage: the parity of its next completion.
struct HalfRing {
    unsigned long long *bar;  // [4], shared
    unsigned parity = 0;
    __device__ explicit HalfRing(unsigned long long *b) : bar(b) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < 4; s++) mbar_init(&bar[s], 1);
            fence_barrier_init();
        }
        __syncthreads();
    }
    __device__ __forceinline__ bool wait(int s) {
        const bool ok = mbar_wait(&bar[s], (parity >> s) & 1u);
        parity ^= 1u << s;
        return ok;
    }
};

// The units [u0, u1) of one half; acc: this thread's part of the sums (P:
// <r0, q>; S: <t, s>, <t, t>).  c1, c2: P beta, omega; S alpha.  Every thread
// of the block calls it; false (in every thread) when a TMA wait ran out.
template <int KIND, typename G>
__device__ __forceinline__ bool half_march(const Grid &g, const PoissonCoef &C, const HalfPlan &H,
                                           const CUtensorMap *mr, const CUtensorMap *mp,
                                           const CUtensorMap *mq, const HalfArgs &A, double c1,
                                           double c2, bool first, long long u0, long long u1,
                                           unsigned char *smem, HalfRing &R, double (&acc)[2]) {
    constexpr int W = G::W, M = G::M, NT = G::NT;
    constexpr int NIN = KIND == HALF_P ? 3 : 2, NS = KIND == HALF_P ? G::NS_P : G::NS_S;
    double *wp = (double *)(smem + G::RING) + W;  // P1, P2, P3: two planes each, past the guard row
    double *cf = (double *)(smem + G::RING) + 6 * G::PLANE;
    const int tid = threadIdx.x, c = tid % W, rq = tid / W;
    const bool act = tid < NT;  // the last warp's rest only keeps the barriers
    const int e = act ? rq * M * W + c : 0;
    const Box &bx = H.box;
    const double inv_md = C.inv_max_diag;
    const int sx = (int)g.sx, sy = (int)g.sy;

    for (long long u = u0; u < u1;) {
        const int tile = (int)(u / H.ni), first_plane = (int)(u - (long long)tile * H.ni);
        const int np = (int)min((long long)min(H.ni - first_plane, HALF_MAXP), u1 - u);
        u += np;
        const int tj = tile / H.ntk, tk = tile - tj * H.ntk;
        int j0, j1, k0, k1;
        H.tile_range(tj, tk, j0, j1, k0, k1);
        const int ib = bx.lo[0] + first_plane - HH, nload = np + 2 * HH;

        // this thread's column and cells
        const int k = k0 - 4 + c, jr = j0 - HH + rq * M;
        const bool kin = act && k >= bx.lo[2] && k < bx.hi[2];
        const double at = kin ? C.at[k] : 0.0, ab = kin ? C.ab[k] : 0.0;
        double an[M], as[M], cs[M];
        bool own[M], any = false;
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int j = jr + m;
            const bool ok = kin && j >= bx.lo[1] && j < bx.hi[1];
            an[m] = ok ? C.an[j] : 0.0;
            as[m] = ok ? C.as[j] : 0.0;
            // the diagonal's column part; any non-zero value outside
            cs[m] = ok ? C.an_u[j] + C.as_u[j] + C.at_u[k] + C.ab_u[k] : 1.0;
            own[m] = ok && j >= j0 && j < j1 && k >= k0 && k < k1;
            any = any || own[m];
        }
        // per-plane coefficients of planes ib .. ib + nload - 1
        for (int q = tid; q < nload; q += G::THREADS) {
            const int i = ib + q;
            const bool ok = i >= bx.lo[0] && i < bx.hi[0];
            cf[3 * q] = ok ? C.ae[i] : 0.0;
            cf[3 * q + 1] = ok ? C.aw[i] : 0.0;
            cf[3 * q + 2] = ok ? C.xpart[i] : 0.0;
        }
        auto issue = [&](int L) {  // thread 0
            const int s = L % NS;
            unsigned char *st = smem + (size_t)s * NIN * G::STAGE;
            const int x = k0 - 4 + (int)g.off, y = j0 - HH, z = ib + L;
            mbar_expect_tx(&R.bar[s], NIN * G::BOX);
            tma_load_3d(st, mr, x, y, z, &R.bar[s]);
            if (KIND == HALF_P) tma_load_3d(st + G::STAGE, mp, x, y, z, &R.bar[s]);
            tma_load_3d(st + (NIN - 1) * G::STAGE, mq, x, y, z, &R.bar[s]);
        };
        __syncthreads();  // cf; the previous march's reads are done
        int issued = 0;
        if (tid == 0) {
            fence_proxy_async();  // the ring was read through the generic proxy
            for (; issued < NS && issued < nload; issued++) issue(issued);
        }

        double w1a[M], w1b[M], w1c[M];  // w1 on planes L-1, L-2, L-3
        double ra[M], rb[M];            // 1/a_c on planes L-1, L-2
        double w2a[M], w2b[M];          // w2 on planes L-2, L-3
        double w3a[M], w3b[M];          // w3 on planes L-3, L-4
        double r0n[M];
#pragma unroll
        for (int m = 0; m < M; m++)
            w1a[m] = w1b[m] = w1c[m] = ra[m] = rb[m] = w2a[m] = w2b[m] = w3a[m] = w3b[m] = r0n[m] = 0.0;

        // R x without the i neighbours: plane values x of this thread's rows,
        // their k neighbours and the rows above and below in P
        auto in_plane = [&](const double *P, const double (&x)[M], double (&o)[M]) {
            double s = P[e - W];
#pragma unroll
            for (int m = 0; m < M; m++) {
                const double n = m < M - 1 ? x[m < M - 1 ? m + 1 : 0] : P[e + M * W];
                double v = an[m] * n;
                v = __fma_rn(as[m], s, v);
                v = __fma_rn(at, P[e + m * W + 1], v);
                o[m] = __fma_rn(ab, P[e + m * W - 1], v);
                s = x[m];
            }
        };
        // a thread whose wait ran out stops computing and waiting, but keeps the
        // block's barriers to the end of the march
        bool fail = false;
        int waited = 0;                              // loads this thread has seen complete
        int o = ib * sx + jr * sy + k + (int)g.off;  // first cell's offset on plane L
        int s = 0;                                   // s = L % NS
        for (int L = 0; L < nload; L++, o += sx, s = s + 1 < NS ? s + 1 : 0) {
            double *P1w = wp + (0 + (L & 1)) * G::PLANE, *P1 = wp + (0 + (~L & 1)) * G::PLANE;
            double *P2w = wp + (2 + (~L & 1)) * G::PLANE, *P2 = wp + (2 + (L & 1)) * G::PLANE;
            double *P3w = wp + (4 + (L & 1)) * G::PLANE, *P3 = wp + (4 + (~L & 1)) * G::PLANE;
            const double *cL = cf + 3 * L;
            if (!fail) fail = !R.wait(s);
            if (!fail) waited++;
            if (act && !fail) {
                double w1[M], w2[M], w3[M], rc[M], r0c[M];
                const double *st = (const double *)(smem + (size_t)s * NIN * G::STAGE) + e;
                if (KIND == HALF_P) {
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        r0c[m] = r0n[m];
                        if (L >= 2 * HH - 1 && L + 1 < nload && own[m]) r0n[m] = A.r0[o - 2 * sx + m * sy];
                    }
                }
                // phase 1, plane L
                const bool out = L >= HH && L < HH + np;
#pragma unroll
                for (int m = 0; m < M; m++) {
                    const double rv = st[m * W], qv = st[(NIN - 1) * (G::STAGE / 8) + m * W];
                    double v;
                    if (KIND == HALF_P) {
                        const double pv = st[G::STAGE / 8 + m * W];
                        v = first ? rv : __fma_rn(c1, __fma_rn(-c2, qv, pv), rv);
                    } else {
                        v = __fma_rn(-c1, qv, rv);
                    }
                    rc[m] = fast_rcp((cL[2] - cs[m]) * inv_md);
                    w1[m] = v * rc[m];
                    if (out && own[m]) A.v[o + m * sy] = v;
                }
                // phase 2, plane L - 1
                if (L >= 2) {
                    const double ae = cL[-3], aw = cL[-2];
                    double p[M];
                    in_plane(P1, w1a, p);
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        p[m] = __fma_rn(aw, w1b[m], p[m]);
                        p[m] = __fma_rn(ae, w1[m], p[m]);
                        w2[m] = __fma_rn(-p[m], ra[m], w1a[m]);
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < M; m++) w2[m] = 0.0;
                }
                // phase 3, plane L - 2
                if (L >= 4) {
                    const double ae = cL[-6], aw = cL[-5];
                    const bool put = L >= HH + 2 && L < HH + 2 + np;
                    double p[M];
                    in_plane(P2, w2a, p);
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        p[m] = __fma_rn(aw, w2b[m], p[m]);
                        p[m] = __fma_rn(ae, w2[m], p[m]);
                        w3[m] = __fma_rn(-p[m], rb[m], w1b[m]);
                        if (put && own[m]) A.w[o - 2 * sx + m * sy] = w3[m];
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < M; m++) w3[m] = 0.0;
                }
                // phase 4, plane L - 3
                if (L >= 2 * HH && any) {
                    const double ae = cL[-9], aw = cL[-8], xp = cL[-7];
                    double p[M];
                    in_plane(P3, w3a, p);
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        const double ac = (xp - cs[m]) * inv_md;
                        p[m] = __fma_rn(ac, w3a[m], p[m]);
                        p[m] = __fma_rn(aw, w3b[m], p[m]);
                        p[m] = __fma_rn(ae, w3[m], p[m]);
                        if (own[m]) {
                            A.av[o - HH * sx + m * sy] = p[m];
                            if (KIND == HALF_P) {
                                acc[0] = __fma_rn(r0c[m], p[m], acc[0]);
                            } else {
                                acc[0] = __fma_rn(p[m], w1c[m] * ac, acc[0]);  // w1 a_c = s
                                acc[1] = __fma_rn(p[m], p[m], acc[1]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < M; m++) {
                    P1w[e + m * W] = w1[m];
                    P2w[e + m * W] = w2[m];
                    P3w[e + m * W] = w3[m];
                    if (KIND == HALF_S) w1c[m] = w1b[m];
                    w1b[m] = w1a[m];
                    w1a[m] = w1[m];
                    rb[m] = ra[m];
                    ra[m] = rc[m];
                    w2b[m] = w2a[m];
                    w2a[m] = w2[m];
                    w3b[m] = w3a[m];
                    w3a[m] = w3[m];
                }
            }
            __syncthreads();
            if (tid == 0 && !fail && issued < nload) {
                fence_proxy_async();  // the stage just read is free
                issue(issued++);
            }
        }
        if (__syncthreads_or(fail)) {
            if (tid == 0)  // drain what is still in flight
                for (int q = waited + 1; q < issued; q++) R.wait(q % NS);
            return false;
        }
    }
    return true;
}

}  // namespace
}  // namespace dalm
