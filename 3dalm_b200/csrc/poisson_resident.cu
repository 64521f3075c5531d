// Whole FP64 pressure solves as one cooperative kernel.
//
// One launch per sweep makes a solve wait for launches and last waves: a
// red-black SOR iteration of 128 x 64 x 64 cells moves 21 MB, all of it in L2,
// and took 26 us in three launches.  Here the solve stays on the device for the
// whole loop: one block per SM (or fewer), a barrier over the blocks between
// dependent sweeps, and every block computing the Krylov scalars for itself
// from the blocks' partial sums in block order, so that the result does not
// depend on scheduling.
//
//   SOR      two barriers per iteration.  The residual that decides the stop
//            is not a pass of its own: at the cells of the colour relaxed
//            last it is (1 - w) times what the relaxation has just computed,
//            and at the other colour it is what the next iteration's first
//            half-sweep computes before it relaxes.  That half-sweep's values
//            are kept apart, so it can be dropped when the solve stops.
//   Jacobi   one barrier per iteration, the same way.
//   BiCGStab nine barriers per iteration with the Jacobi(3) preconditioner
//            and the vectors in registers, a barrier per half-sweep with the
//            SOR preconditioner.
//
// What bounds them on grids that leave registers or L2 unfilled: the barriers
// (1.24 us each) and the latency of the loads after them.  us per iteration,
// launched / here: SOR 24x12x12 13.2 / 2.9, 128x64x64 26.4 / 7.3, 384x192x100
// 139 / 87, 4000x80x80 409 / 305; Jacobi 72x20x100 17.7 / 4.6, 384x192x100
// 93 / 50, 4000x80x80 285 / 169; BiCGStab with
// the step around it, 40x20x20 44 / 25, 100x40x33 74 / 29, 131x75x53 93 / 58.
//
// Cell values are computed with the launched kernels' operations in their
// order (poisson_math.cuh), or on the off-diagonal part where the cells are in
// registers; sums differ in their order.
//
// A block whose barrier does not complete within BARRIER_POLLS polls marks the
// solve's state and leaves; the others leave at their next barrier.  A straggler may
// still find a barrier complete that another block gave up, so the mark is
// never written over (finish), and the host reports DALM_ERR_DEVICE_WAIT
// whatever else the state says.
#include "poisson.cuh"
#include "poisson_math.cuh"

namespace dalm {

namespace {

constexpr int RT = 512;                       // threads of the sweep kernels
constexpr unsigned BARRIER_POLLS = 1u << 21;  // about a second

// The grid's barrier and sums.  One thread of a block adds 1 to a counter
// (release) and polls it (acquire) until every block has: 2441 cycles over 148
// blocks, the stores before it included.  (A fence on either side of a relaxed
// addition and poll: 3196; a flag per block that every block reads: 5999.)
// Partial sums go through two sets of slots in turn, so a block may store the
// next ones while another still reads the last; every block adds them in block
// order.
struct GridSync {
    unsigned *count;  // [0] arrivals, [1] failed; zeroed before the launch
    double2 *part;    // [2][gridDim.x]
    unsigned goal = 0;
    int set = 0;
    __device__ GridSync(unsigned *c, double *p) : count(c), part((double2 *)p) {}
    static __device__ __forceinline__ unsigned load(const unsigned *p) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        return v;
    }
    // one thread, after a block barrier: true once every block has arrived
    __device__ __forceinline__ bool arrive_wait() {
        goal += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        for (unsigned n = 0; (int)(load(count) - goal) < 0;) {
            if (++n >= BARRIER_POLLS || ((n & 255u) == 0 && load(count + 1))) {
                atomicExch(count + 1, 1u);
                return false;
            }
        }
        return true;
    }
    // false in every thread when the wait ran out here or anywhere
    __device__ __forceinline__ bool sync() {
        __syncthreads();
        if (gridDim.x == 1) return true;
        return !__syncthreads_or(threadIdx.x == 0 && !arrive_wait());
    }
    // A barrier with the grid's sums of a and (N = 2) b: fin(a, b) runs in
    // thread 0 of every block before the block goes on.
    template <int N, typename F>
    __device__ __forceinline__ bool reduce(double a, double b, F fin) {
        __shared__ double red[2][32];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        a = warp_reduce(a, false);
        if (N == 2) b = warp_reduce(b, false);
        if (lane == 0) {
            red[0][warp] = a;
            if (N == 2) red[1][warp] = b;
        }
        __syncthreads();
        bool bad = false;
        if (warp == 0) {
            const bool in = lane < (int)(blockDim.x >> 5);
            a = warp_reduce(in ? red[0][lane] : 0.0, false);
            b = N == 2 ? warp_reduce(in ? red[1][lane] : 0.0, false) : 0.0;
            if (gridDim.x > 1) {
                double2 *slot = part + set * gridDim.x;
                if (lane == 0) {
                    slot[blockIdx.x] = make_double2(a, b);
                    bad = !arrive_wait();
                }
                bad = __shfl_sync(0xffffffffu, bad, 0);
                double2 v[5];  // up to 160 blocks' loads together
                a = b = 0.0;
                for (unsigned q0 = 0; q0 < gridDim.x; q0 += 160) {
#pragma unroll
                    for (int m = 0; m < 5; m++) {
                        const unsigned q = q0 + 32 * m + lane;
                        v[m] = q < gridDim.x ? __ldcg(slot + q) : make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int m = 0; m < 5; m++) {
                        a += v[m].x;
                        b += v[m].y;
                    }
                }
                a = warp_reduce(a, false);
                if (N == 2) b = warp_reduce(b, false);
                set ^= 1;
            }
            if (lane == 0 && !bad) fin(a, b);
        }
        return !__syncthreads_or(bad);
    }
};

// n / d for n d < 2^32, d >= 2, by multiplication with m = ceil(2^32 / d):
// m d - 2^32 < d, so the quotient's error n (m d - 2^32) / (d 2^32) is less
// than 1 / d
struct Divisor {
    unsigned d, m;
    static Divisor make(unsigned d) { return Divisor{d, (unsigned)(((1ull << 32) + d - 1) / d)}; }
    __device__ __forceinline__ unsigned div(unsigned n) const { return __umulhi(n, m); }
};

// The interior's cells in rows along k: all of them, or one colour
// ((i + j + k) % 2, stored indices) with half as many slots per row.
struct Cells {
    Box box;
    Divisor nj, nk, hk;
    unsigned all, half;
    static Cells make(const Box &b) {
        Cells s;
        s.box = b;
        const unsigned ni = b.hi[0] - b.lo[0], nj = b.hi[1] - b.lo[1], nk = b.hi[2] - b.lo[2];
        s.nj = Divisor::make(nj);
        s.nk = Divisor::make(nk);
        s.hk = Divisor::make((nk + 1) / 2);
        s.all = ni * nj * nk;
        s.half = ni * nj * ((nk + 1) / 2);
        return s;
    }
};

// per-axis coefficients in shared memory, indexed by stored cell
struct AxisCoef {
    const double *ae, *aw, *xp, *an, *as, *js, *at, *ab, *tu, *bu;
    double inv_md;
    static size_t bytes(const Grid &g) { return sizeof(double) * (3 * (size_t)g.nx + 3 * (size_t)g.ny + 4 * (size_t)g.nz); }
    __device__ void stage(const Grid &g, const PoissonCoef &C, double *s) {
        double *d[10];
        const int n[3] = {g.nx, g.ny, g.nz};
        for (int q = 0; q < 10; q++) {
            d[q] = s;
            s += n[q < 3 ? 0 : q < 6 ? 1 : 2];
        }
        for (int i = threadIdx.x; i < g.nx; i += blockDim.x)
            d[0][i] = C.ae[i], d[1][i] = C.aw[i], d[2][i] = C.xpart[i];
        for (int j = threadIdx.x; j < g.ny; j += blockDim.x)
            d[3][j] = C.an[j], d[4][j] = C.as[j], d[5][j] = C.an_u[j] + C.as_u[j];
        for (int k = threadIdx.x; k < g.nz; k += blockDim.x)
            d[6][k] = C.at[k], d[7][k] = C.ab[k], d[8][k] = C.at_u[k], d[9][k] = C.ab_u[k];
        ae = d[0]; aw = d[1]; xp = d[2]; an = d[3]; as = d[4]; js = d[5];
        at = d[6]; ab = d[7]; tu = d[8]; bu = d[9];
        inv_md = C.inv_max_diag;
        __syncthreads();
    }
    __device__ __forceinline__ double diag(int i, int j, int k) const {
        return (xp[i] - ((js[j] + tu[k]) + bu[k])) * inv_md;
    }
};

struct Cell {
    int i, j, k, c;
    bool ok;
};
struct Star {  // a cell and its six neighbours
    double c, e, w, n, s, t, b;
};

struct Domain {
    Cells S;
    int sx, sy, off;
    AxisCoef K;
    // slot n of all cells (color < 0) or of one colour
    __device__ __forceinline__ Cell cell(unsigned n, int color) const {
        Cell q;
        const Divisor &d = color < 0 ? S.nk : S.hk;
        const unsigned row = d.div(n), l = n - row * d.d, i = S.nj.div(row);
        q.i = S.box.lo[0] + (int)i;
        q.j = S.box.lo[1] + (int)(row - i * S.nj.d);
        q.k = S.box.lo[2] + (int)l;
        if (color >= 0) q.k += (int)l + ((q.i + q.j + S.box.lo[2] + color) & 1);
        q.ok = n < (color < 0 ? S.all : S.half) && q.k < S.box.hi[2];
        q.c = q.ok ? q.i * sx + q.j * sy + q.k + off : 0;
        if (!q.ok) q.i = S.box.lo[0], q.j = S.box.lo[1], q.k = S.box.lo[2];
        return q;
    }
    // own: the array of the cell itself, nb: of its neighbours
    __device__ __forceinline__ Star load(const Cell &q, const double *own, const double *nb) const {
        Star v{0, 0, 0, 0, 0, 0, 0};
        if (q.ok) {
            v.c = own[q.c];
            v.e = nb[q.c + sx];
            v.w = nb[q.c - sx];
            v.n = nb[q.c + sy];
            v.s = nb[q.c - sy];
            v.t = nb[q.c + 1];
            v.b = nb[q.c - 1];
        }
        return v;
    }
    // A x (apply_a<false>'s operations)
    __device__ __forceinline__ double apply(const Cell &q, double ac, const Star &v) const {
        double o = ac * v.c;
        o = __fma_rn(K.ae[q.i], v.e, o);
        o = __fma_rn(K.aw[q.i], v.w, o);
        o = __fma_rn(K.an[q.j], v.n, o);
        o = __fma_rn(K.as[q.j], v.s, o);
        o = __fma_rn(K.at[q.k], v.t, o);
        return __fma_rn(K.ab[q.k], v.b, o);
    }
};

// Runs body(cells, count U) over the slots of this thread, U at a time, so
// that the loads of U cells are in flight together.
template <int U, typename F>
__device__ __forceinline__ void for_cells(const Domain &D, int color, F body) {
    const unsigned stride = gridDim.x * blockDim.x, total = color < 0 ? D.S.all : D.S.half;
    for (unsigned n = blockIdx.x * blockDim.x + threadIdx.x; n < total; n += U * stride) {
        Cell q[U];
#pragma unroll
        for (int u = 0; u < U; u++) q[u] = D.cell(n + u * stride < total ? n + u * stride : total, color);
        body(q);
    }
}

__device__ __forceinline__ void finish(const KrylovState &S, KrylovState *st, bool failed) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (failed) {
        st->wait_error = 1;
    } else if (blockIdx.x == 0) {  // what a solve changes, but for the mark
        st->rho = S.rho, st->rho_old = S.rho_old, st->alpha = S.alpha, st->omega = S.omega, st->beta = S.beta;
        st->err = S.err, st->it = S.it, st->done = S.done, st->breakdown = S.breakdown;
    }
}

// ---- red-black SOR and Jacobi ------------------------------------------------

// Up to `budget` iterations of SOR (src/eq.h:291-306) from x; tmp holds the
// red cells of the other time level.
__global__ void __launch_bounds__(RT, 1)
k_resident_sor(Grid g, PoissonCoef C, Cells cells, double *x, double *tmp, const double *b, double w,
               long long budget, double *part, unsigned *sync, KrylovState *st) {
    constexpr int U = 4;
    extern __shared__ double resident_smem[];
    __shared__ KrylovState S;
    Domain D{cells, (int)g.sx, (int)g.sy, (int)g.off, {}};
    D.K.stage(g, C, resident_smem);
    if (threadIdx.x == 0) S = *st;
    __syncthreads();
    if (S.done) return;
    GridSync grid(sync, part);
    double *cur = x, *nxt = tmp;  // red cells
    double black = 0.0;           // this thread's squared residuals at the black cells
    bool ok = true;
    for (long long n = 0;; n++) {
        // red: the residual of the last iterate, and the next iteration's values
        double acc = black;
        for_cells<U>(D, 0, [&](const Cell (&q)[U]) {
            Star v[U];
            double rhs[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = D.load(q[u], cur, x);
                rhs[u] = q[u].ok ? b[q[u].c] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double ac = D.K.diag(q[u].i, q[u].j, q[u].k);
                const double res = rhs[u] - D.apply(q[u], ac, v[u]);
                acc = __fma_rn(res, res, acc);
                if (q[u].ok) nxt[q[u].c] = __fma_rn(w, res * fast_rcp(ac), v[u].c);
            }
        });
        ok = grid.reduce<1>(acc, 0.0, [&](double r2, double) { if (n > 0) finish_iteration(&S, r2); });
        if (!ok || S.done || n == budget) break;
        // black: neighbours are the new red cells
        black = 0.0;
        for_cells<U>(D, 1, [&](const Cell (&q)[U]) {
            Star v[U];
            double rhs[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = D.load(q[u], x, nxt);
                rhs[u] = q[u].ok ? b[q[u].c] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double ac = D.K.diag(q[u].i, q[u].j, q[u].k);
                const double res = rhs[u] - D.apply(q[u], ac, v[u]);
                const double left = (1.0 - w) * res;
                black = __fma_rn(left, left, black);
                if (q[u].ok) x[q[u].c] = __fma_rn(w, res * fast_rcp(ac), v[u].c);
            }
        });
        if (!(ok = grid.sync())) break;
        double *o = cur;
        cur = nxt;
        nxt = o;
    }
    if (ok && cur != x)
        for_cells<U>(D, 0, [&](const Cell (&q)[U]) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (q[u].ok) x[q[u].c] = cur[q[u].c];
        });
    finish(S, st, !ok);
}

// The same with the iterate in registers, for grids of up to SOR_UI x 2 cells
// per thread: a thread owns the cell pairs (k, k + 1) of SOR_UI consecutive
// planes of one (j, k), one red and one black cell each, their right-hand
// sides and reciprocal diagonals.  Neighbours along i and the other cell of
// the pair come from registers; the rest goes through the two colours'
// packed arrays ([ni + 2][nj + 2][hk + 2], zero outside the interior), so
// every access is a row of consecutive values.
constexpr int SOR_UI = 4;

struct Packed {
    int ni, nj, hk, sj, si;  // interior planes, rows, pairs per row; strides
    Divisor dhk, dnj;
    unsigned columns, threads;
    __host__ __device__ int at(int i, int j, int l) const { return (i + 1) * si + (j + 1) * sj + l + 1; }
    __host__ __device__ int total() const { return (ni + 2) * si; }
    static Packed make(const Box &b) {
        Packed p;
        p.ni = b.hi[0] - b.lo[0];
        p.nj = b.hi[1] - b.lo[1];
        p.hk = (b.hi[2] - b.lo[2] + 1) / 2;
        p.sj = p.hk + 2;
        p.si = p.sj * (p.nj + 2);
        p.dhk = Divisor::make((unsigned)p.hk);
        p.dnj = Divisor::make((unsigned)p.nj);
        p.columns = (unsigned)(p.nj * p.hk);
        p.threads = p.columns * (unsigned)((p.ni + SOR_UI - 1) / SOR_UI);
        return p;
    }
};

template <bool ONE>  // ONE: a single block, the packed arrays in its shared memory
__global__ void __launch_bounds__(RT, 1)
k_resident_sor_regs(Grid g, PoissonCoef C, Box box, Packed Q, double *x, double *red, double *blk,
                    const double *b, double w, long long budget, double *part, unsigned *sync,
                    KrylovState *st) {
    constexpr int U = SOR_UI;
    extern __shared__ double resident_smem[];
    __shared__ KrylovState S;
    if (threadIdx.x == 0) S = *st;
    __syncthreads();
    if (S.done) return;
    GridSync grid(sync, part);
    if (ONE) {
        red = resident_smem + 3 * (Q.ni + U);
        blk = red + Q.total();
    }
    // coefficients along i of the interior, 0 past its end
    double *ci = resident_smem;
    for (int n = threadIdx.x; n < Q.ni + U; n += RT) {
        const int i = box.lo[0] + n;
        ci[3 * n] = n < Q.ni ? C.ae[i] : 0.0;
        ci[3 * n + 1] = n < Q.ni ? C.aw[i] : 0.0;
        ci[3 * n + 2] = n < Q.ni ? C.xpart[i] : 0.0;
    }
    // zero both packed arrays: their guard cells are read (with coefficient 0)
    for (int n = blockIdx.x * RT + threadIdx.x; n < Q.total(); n += gridDim.x * RT) red[n] = blk[n] = 0.0;
    bool ok = grid.sync();

    const unsigned id = blockIdx.x * RT + threadIdx.x;
    const bool act = id < Q.threads;
    const unsigned row = Q.dhk.div(act ? id : 0);
    const int l = (int)((act ? id : 0) - row * Q.dhk.d);
    const unsigned chunk = Q.dnj.div(row);
    const int jj = (int)(row - chunk * Q.dnj.d), ii = (int)chunk * U;
    const int nu = act ? min(U, Q.ni - ii) : 0;
    const int j = box.lo[1] + jj, i0 = box.lo[0] + ii, ka = box.lo[2] + 2 * l;
    const bool two = ka + 1 < box.hi[2];  // the pair's second cell exists
    const int p0 = (i0 + j + box.lo[2]) & 1;  // 1: the red cell of plane i0 is the pair's second
    const double an = C.an[j], as = C.as[j], js = C.an_u[j] + C.as_u[j];
    // the pair's cells: coefficient of the other cell of the pair (in), of the
    // neighbour outside the pair (out), and the diagonal's column part
    const double in0 = two ? C.at[ka] : 0.0, out0 = C.ab[ka], cs0 = (js + C.at_u[ka]) + C.ab_u[ka];
    const double in1 = two ? C.ab[ka + 1] : 0.0, out1 = two ? C.at[ka + 1] : 0.0;
    const double cs1 = two ? (js + C.at_u[ka + 1]) + C.ab_u[ka + 1] : cs0;
    // A: the red cell of even planes (and black of odd ones), B: the other
    const double inA = p0 ? in1 : in0, outA = p0 ? out1 : out0, csA = p0 ? cs1 : cs0;
    const double inB = p0 ? in0 : in1, outB = p0 ? out0 : out1, csB = p0 ? cs0 : cs1;
    const int dA = p0 ? 1 : -1;  // the pair that holds A's outer neighbour
    const bool okA = !p0 || two, okB = p0 || two;
    const double md = C.inv_max_diag;
    const int at0 = Q.at(ii, jj, l);
    const int c0 = (int)g.at(i0, j, ka);
    double r[U], k[U], br[U], bk[U], rr[U], rk[U], nr[U];  // red, black; b; 1/a_c; new red
    const double *cu = ci + 3 * (act ? ii : 0);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const bool v = u < nu;
        const int c = c0 + (v ? u : 0) * (int)g.sx;
        const int s = (p0 ^ u) & 1;  // the red cell's place in the pair
        const bool okr = v && (u & 1 ? okB : okA), okk = v && (u & 1 ? okA : okB);
        r[u] = okr ? x[c + s] : 0.0;
        br[u] = okr ? b[c + s] : 0.0;
        k[u] = okk ? x[c + 1 - s] : 0.0;
        bk[u] = okk ? b[c + 1 - s] : 0.0;
        rr[u] = okr ? fast_rcp((cu[3 * u + 2] - (u & 1 ? csB : csA)) * md) : 0.0;
        rk[u] = okk ? fast_rcp((cu[3 * u + 2] - (u & 1 ? csA : csB)) * md) : 0.0;
        nr[u] = 0.0;
        if (v) blk[at0 + u * Q.si] = k[u];
    }
    // red cells first need the neighbours' black cells
    ok = ok && grid.sync();

    // b - A x without the centre term at every cell of one colour: `o` the
    // other colour's values (registers own, packed nb)
    auto gather = [&](const double (&own)[U], const double *nb, bool first_color, const double (&rhs)[U],
                      double (&t)[U]) {
        double n[U], s[U], q[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool isA = ((u & 1) == 0) == first_color;
            const int a = at0 + u * Q.si;
            n[u] = u < nu ? nb[a + Q.sj] : 0.0;
            s[u] = u < nu ? nb[a - Q.sj] : 0.0;
            q[u] = u < nu ? nb[a + (isA ? dA : -dA)] : 0.0;
        }
        double w0 = nu > 0 ? nb[at0 - Q.si] : 0.0, e1 = nu > 0 ? nb[at0 + nu * Q.si] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool isA = ((u & 1) == 0) == first_color;
            const double e = u + 1 < nu ? own[u + 1 < U ? u + 1 : u] : e1;
            double v = __fma_rn(-cu[3 * u], e, rhs[u]);
            v = __fma_rn(-cu[3 * u + 1], u > 0 ? own[u > 0 ? u - 1 : 0] : w0, v);
            v = __fma_rn(-an, n[u], v);
            v = __fma_rn(-as, s[u], v);
            v = __fma_rn(isA ? -inA : -inB, own[u], v);
            t[u] = __fma_rn(isA ? -outA : -outB, q[u], v);
        }
    };
    double black = 0.0;
    for (long long n = 0; ok; n++) {
        double acc = black, t[U];
        gather(k, blk, true, br, t);
#pragma unroll
        for (int u = 0; u < U; u++) {
            // t = b - R x; the relaxed cell and its residual before
            const double d = __fma_rn(t[u], rr[u], -r[u]);  // (b - A x) / a_c
            nr[u] = __fma_rn(w, d, r[u]);
            const double ac = (cu[3 * u + 2] - (u & 1 ? csB : csA)) * md;
            const double res = rr[u] != 0.0 ? __fma_rn(-ac, r[u], t[u]) : 0.0;
            acc = __fma_rn(res, res, acc);
            if (u < nu) red[at0 + u * Q.si] = nr[u];
        }
        ok = grid.reduce<1>(acc, 0.0, [&](double r2, double) { if (n > 0) finish_iteration(&S, r2); });
        if (!ok || S.done || n == budget) break;
        black = 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) r[u] = nr[u];
        gather(r, red, false, bk, t);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double d = __fma_rn(t[u], rk[u], -k[u]);
            const double ac = (cu[3 * u + 2] - (u & 1 ? csA : csB)) * md;
            const double left = rk[u] != 0.0 ? (1.0 - w) * __fma_rn(-ac, k[u], t[u]) : 0.0;
            k[u] = __fma_rn(w, d, k[u]);
            black = __fma_rn(left, left, black);
            if (u < nu) blk[at0 + u * Q.si] = k[u];
        }
        ok = grid.sync();
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (!ok || u >= nu) continue;
        const int c = c0 + u * (int)g.sx, s = (p0 ^ u) & 1;
        if (u & 1 ? okB : okA) x[c + s] = r[u];
        if (u & 1 ? okA : okB) x[c + 1 - s] = k[u];
    }
    finish(S, st, !ok);
}

// Up to `budget` Jacobi iterations from x; tmp holds the other iterate.
__global__ void __launch_bounds__(RT, 1)
k_resident_jacobi(Grid g, PoissonCoef C, Cells cells, double *x, double *tmp, const double *b,
                  long long budget, double *part, unsigned *sync, KrylovState *st) {
    constexpr int U = 4;
    extern __shared__ double resident_smem[];
    __shared__ KrylovState S;
    Domain D{cells, (int)g.sx, (int)g.sy, (int)g.off, {}};
    D.K.stage(g, C, resident_smem);
    if (threadIdx.x == 0) S = *st;
    __syncthreads();
    if (S.done) return;
    GridSync grid(sync, part);
    double *cur = x, *nxt = tmp;
    bool ok = true;
    for (long long n = 0;; n++) {
        double acc = 0.0;
        for_cells<U>(D, -1, [&](const Cell (&q)[U]) {
            Star v[U];
            double rhs[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = D.load(q[u], cur, cur);
                rhs[u] = q[u].ok ? b[q[u].c] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double ac = D.K.diag(q[u].i, q[u].j, q[u].k);
                const double res = rhs[u] - D.apply(q[u], ac, v[u]);
                acc = __fma_rn(res, res, acc);
                if (q[u].ok) nxt[q[u].c] = v[u].c + res * fast_rcp(ac);
            }
        });
        ok = grid.reduce<1>(acc, 0.0, [&](double r2, double) { if (n > 0) finish_iteration(&S, r2); });
        if (!ok || S.done || n == budget) break;
        double *o = cur;
        cur = nxt;
        nxt = o;
    }
    if (ok && cur != x)
        for_cells<U>(D, -1, [&](const Cell (&q)[U]) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (q[u].ok) x[q[u].c] = cur[q[u].c];
        });
    finish(S, st, !ok);
}

// ---- BiCGStab ------------------------------------------------------------------

// x += alpha pp + omega ss; r = s - omega t (k_bicg_xr's operations) on this
// thread's cells; its parts of <r0, r>, <r, r>
__device__ __forceinline__ void update_xr(const Domain &D, const PoissonBufs &B, double alpha,
                                          double omega, double (&acc)[2]) {
    constexpr int U = 2;
    for_cells<U>(D, -1, [&](const Cell (&q)[U]) {
        double x[U], pp[U], ss[U], s[U], t[U], r0[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = q[u].c;
            x[u] = q[u].ok ? B.x[c] : 0.0;
            pp[u] = q[u].ok ? B.pp[c] : 0.0;
            ss[u] = q[u].ok ? B.ss[c] : 0.0;
            s[u] = q[u].ok ? B.s[c] : 0.0;
            t[u] = q[u].ok ? B.t[c] : 0.0;
            r0[u] = q[u].ok ? B.r0[c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double r = __fma_rn(-omega, t[u], s[u]);
            if (q[u].ok) {
                B.x[q[u].c] = __fma_rn(omega, ss[u], __fma_rn(alpha, pp[u], x[u]));
                B.r[q[u].c] = r;
            }
            acc[0] += r0[u] * r;
            acc[1] += r * r;
        }
    });
}

// The interior's columns for k_resident_bicg: a thread owns U consecutive
// planes of one (j, k), k fastest.
struct Columns {
    Box box;
    Divisor nj, nk;
    unsigned threads;
    static Columns make(const Box &b, int U) {
        Columns c;
        c.box = b;
        c.nj = Divisor::make((unsigned)(b.hi[1] - b.lo[1]));
        c.nk = Divisor::make((unsigned)(b.hi[2] - b.lo[2]));
        c.threads = c.nj.d * c.nk.d * (unsigned)((b.hi[0] - b.lo[0] + U - 1) / U);
        return c;
    }
};

// Up to `budget` iterations with the Jacobi(3) preconditioner from the state
// in B (r, p, q, x), which it leaves there for another launch.  A thread keeps
// its cells' r, p, q and the solve's running values in registers (MEM: p and q
// in memory); what its neighbours need of it goes through memory: w1, w2 and
// the preconditioned vector of either half, six vectors an iteration, each
// followed by a barrier, and three sums.  Sweeps are written on the
// off-diagonal part as in poisson_half.cuh.
template <int U, bool MEM>
__global__ void __launch_bounds__(RT, 1)
k_resident_bicg(Grid g, PoissonCoef C, Columns Q, PoissonBufs B, long long budget, double *part,
                unsigned *sync, KrylovState *st) {
    extern __shared__ double resident_smem[];
    __shared__ KrylovState S;
    if (threadIdx.x == 0) S = *st;
    __syncthreads();
    if (S.done) return;
    GridSync grid(sync, part);
    const Box &bx = Q.box;
    const int ni = bx.hi[0] - bx.lo[0];
    double *ci = resident_smem;  // coefficients along i, 0 past the interior
    for (int n = threadIdx.x; n < ni + U; n += RT) {
        const int i = bx.lo[0] + n;
        ci[3 * n] = n < ni ? C.ae[i] : 0.0;
        ci[3 * n + 1] = n < ni ? C.aw[i] : 0.0;
        ci[3 * n + 2] = n < ni ? C.xpart[i] : 0.0;
    }
    __syncthreads();
    const unsigned id = blockIdx.x * RT + threadIdx.x;
    const bool act = id < Q.threads;
    const unsigned row = Q.nk.div(act ? id : 0), chunk = Q.nj.div(row);
    const int k = bx.lo[2] + (int)((act ? id : 0) - row * Q.nk.d);
    const int j = bx.lo[1] + (int)(row - chunk * Q.nj.d), ii = (int)chunk * U;
    const int nu = act ? min(U, ni - ii) : 0, lane = threadIdx.x & 31;
    const double an = C.an[j], as = C.as[j], at = C.at[k], ab = C.ab[k];
    const double cs = C.an_u[j] + C.as_u[j] + C.at_u[k] + C.ab_u[k], md = C.inv_max_diag;
    const double *cu = ci + 3 * ii;
    const int sx = (int)g.sx, sy = (int)g.sy;
    const int c0 = (int)g.at(bx.lo[0] + ii, j, k);

    auto load = [&](const double *f, double (&v)[U]) {
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = u < nu ? f[c0 + u * sx] : 0.0;
    };
    auto store = [&](double *f, const double (&v)[U]) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (u < nu) f[c0 + u * sx] = v[u];
    };
    // off-diagonal part of A x at the thread's cells: x in registers and in f
    auto off = [&](const double (&x)[U], const double *f, double (&o)[U]) {
        double n[U], s[U], t[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double *c = f + c0 + u * sx;
            n[u] = u < nu ? c[sy] : 0.0;
            s[u] = u < nu ? c[-sy] : 0.0;
            t[u] = lane == 31 && u < nu ? c[1] : 0.0;
            b[u] = lane == 0 && u < nu ? c[-1] : 0.0;
        }
        const double w = nu > 0 ? f[c0 - sx] : 0.0, e = nu > 0 ? f[c0 + nu * sx] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            // the other lanes' k neighbours are in the next lanes (at a row's
            // end the coefficient is 0)
            const double up = __shfl_down_sync(0xffffffffu, x[u], 1), dn = __shfl_up_sync(0xffffffffu, x[u], 1);
            double v = cu[3 * u] * (u + 1 < nu ? x[u + 1 < U ? u + 1 : u] : e);
            v = __fma_rn(cu[3 * u + 1], u > 0 ? x[u > 0 ? u - 1 : 0] : w, v);
            v = __fma_rn(at, lane == 31 ? t[u] : up, v);
            v = __fma_rn(ab, lane == 0 ? b[u] : dn, v);
            v = __fma_rn(an, n[u], v);
            o[u] = __fma_rn(as, s[u], v);
        }
    };
    auto diag = [&](int u) { return (cu[3 * u + 2] - cs) * md; };
    // z = M^-1 v into f3 (and z), av = A z; false when a barrier ran out
    auto precondition = [&](const double (&v)[U], double *f3, double (&z)[U], double (&av)[U]) {
        double w1[U], o[U];
#pragma unroll
        for (int u = 0; u < U; u++) w1[u] = v[u] * fast_rcp(diag(u));
        store(B.tp, w1);
        if (!grid.sync()) return false;
        off(w1, B.tp, o);
#pragma unroll
        for (int u = 0; u < U; u++) z[u] = __fma_rn(-o[u], fast_rcp(diag(u)), w1[u]);
        store(B.ts, z);
        if (!grid.sync()) return false;
        off(z, B.ts, o);
#pragma unroll
        for (int u = 0; u < U; u++) z[u] = __fma_rn(-o[u], fast_rcp(diag(u)), w1[u]);
        store(f3, z);
        if (!grid.sync()) return false;
        off(z, f3, o);
#pragma unroll
        for (int u = 0; u < U; u++) av[u] = __fma_rn(diag(u), z[u], o[u]);
        return true;
    };
    double r[U], p[MEM ? 1 : U], q[MEM ? 1 : U];
    load(B.r, r);
    if constexpr (!MEM) {
        load(B.pk, p);
        load(B.q, q);
    }
    bool ok = true;
    for (long long n = 0; n < budget && !S.done && ok; n++) {
        const bool first = S.it == 0;
        const double beta = S.beta, old_omega = S.omega;
        double v[U], z[U], av[U];
        double a0 = 0.0, a1 = 0.0;
        if constexpr (MEM) {
            double m[U];
            load(B.pk, v);
            load(B.q, m);
#pragma unroll
            for (int u = 0; u < U; u++)
                v[u] = first ? r[u] : __fma_rn(beta, __fma_rn(-old_omega, m[u], v[u]), r[u]);
            store(B.pk, v);
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = first ? r[u] : __fma_rn(beta, __fma_rn(-old_omega, q[u], p[u]), r[u]);
                p[u] = v[u];
            }
        }
        if (!(ok = precondition(v, B.pp, z, av))) break;
        load(B.r0, z);
#pragma unroll
        for (int u = 0; u < U; u++) a0 = __fma_rn(z[u], av[u], a0);
        if constexpr (MEM) {
            store(B.q, av);
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) q[u] = av[u];
        }
        if (!(ok = grid.reduce<1>(a0, 0.0, [&](double a, double) { fin_q(&S, a); }))) break;
        const double alpha = S.alpha;
#pragma unroll
        for (int u = 0; u < U; u++) r[u] = __fma_rn(-alpha, av[u], r[u]);  // s
        if (!(ok = precondition(r, B.ss, z, av))) break;
        a0 = a1 = 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (u >= nu) av[u] = 0.0;
            a0 = __fma_rn(av[u], r[u], a0);
            a1 = __fma_rn(av[u], av[u], a1);
        }
        if (!(ok = grid.reduce<2>(a0, a1, [&](double a, double b) { fin_t(&S, a, b); }))) break;
        const double omega = S.omega;
        a0 = a1 = 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (u < nu) {
                const int c = c0 + u * sx;
                B.x[c] = __fma_rn(omega, z[u], __fma_rn(alpha, B.pp[c], B.x[c]));
                r[u] = __fma_rn(-omega, av[u], r[u]);
                a0 = __fma_rn(B.r0[c], r[u], a0);
                a1 = __fma_rn(r[u], r[u], a1);
            }
        ok = grid.reduce<2>(a0, a1, [&](double a, double b) { fin_xr(&S, a, b); });
    }
    if (ok) {
        store(B.r, r);
        if constexpr (!MEM) {
            store(B.pk, p);
            store(B.q, q);
        }
    }
    finish(S, st, !ok);
}

// One colour's relaxation of A z = rhs in place; `zero`: z's own cells are
// still the zero guess.
__device__ __forceinline__ void relax_color(const Domain &D, double *z, const double *rhs, double w,
                                            int color, bool zero) {
    constexpr int U = 4;
    for_cells<U>(D, color, [&](const Cell (&q)[U]) {
        Star v[U];
        double f[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            v[u] = D.load(q[u], z, z);
            if (zero) v[u].c = 0.0;
            f[u] = q[u].ok ? rhs[q[u].c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double ac = D.K.diag(q[u].i, q[u].j, q[u].k);
            const double rel = (f[u] - D.apply(q[u], ac, v[u])) * fast_rcp(ac);
            if (q[u].ok) z[q[u].c] = __fma_rn(w, rel, v[u].c);
        }
    });
}

// Up to `budget` iterations with the SOR preconditioner (src/eq.h:404-473):
// from a zero guess the first red half-sweep is w v / a_c, fused with the
// update of v.
__global__ void __launch_bounds__(RT, 1)
k_resident_bicg_sor(Grid g, PoissonCoef C, Cells cells, PoissonBufs B, int sweeps, double w,
                    long long budget, double *part, unsigned *sync, KrylovState *st) {
    constexpr int U = 4;
    extern __shared__ double resident_smem[];
    __shared__ KrylovState S;
    Domain D{cells, (int)g.sx, (int)g.sy, (int)g.off, {}};
    D.K.stage(g, C, resident_smem);
    if (threadIdx.x == 0) S = *st;
    __syncthreads();
    if (S.done) return;
    GridSync grid(sync, part);
    bool ok = true;
    // v = update(c), z = M^-1 v, av = A z; v's sums with f: <f, av> or <av, v>, <av, av>
    auto half = [&](auto update, double *vv, double *z, double *av, const double *f, auto fin) {
        for_cells<U>(D, -1, [&](const Cell (&q)[U]) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = q[u].ok ? update(q[u].c) : 0.0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double ac = D.K.diag(q[u].i, q[u].j, q[u].k);
                if (!q[u].ok) continue;
                vv[q[u].c] = v[u];
                if (((q[u].i + q[u].j + q[u].k) & 1) == 0) z[q[u].c] = w * (v[u] * fast_rcp(ac));
            }
        });
        if (!grid.sync()) return false;
        for (int n = 0; n < sweeps; n++)
            for (int color = 0; color < 2; color++) {
                if (n == 0 && color == 0) continue;
                relax_color(D, z, vv, w, color, n == 0);
                if (!grid.sync()) return false;
            }
        double sum[2] = {0.0, 0.0};
        for_cells<U>(D, -1, [&](const Cell (&q)[U]) {
            Star s[U];
            double o[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                s[u] = D.load(q[u], z, z);
                o[u] = q[u].ok ? f[q[u].c] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double a = D.apply(q[u], D.K.diag(q[u].i, q[u].j, q[u].k), s[u]);
                if (q[u].ok) {
                    av[q[u].c] = a;
                    sum[0] += o[u] * a;
                    sum[1] += a * a;
                }
            }
        });
        return grid.reduce<2>(sum[0], sum[1], fin);
    };
    for (long long n = 0; n < budget && !S.done; n++) {
        const bool first = S.it == 0;
        const double beta = S.beta, old_omega = S.omega;
        ok = half([&](int c) { return first ? B.r[c] : __fma_rn(beta, __fma_rn(-old_omega, B.q[c], B.pk[c]), B.r[c]); },
                  B.pk, B.pp, B.q, B.r0, [&](double a, double) { fin_q(&S, a); });
        if (!ok) break;
        const double alpha = S.alpha;
        ok = half([&](int c) { return __fma_rn(-alpha, B.q[c], B.r[c]); }, B.s, B.ss, B.t, B.s,
                  [&](double a, double b) { fin_t(&S, a, b); });
        if (!ok) break;
        double v[2] = {0.0, 0.0};
        update_xr(D, B, S.alpha, S.omega, v);
        ok = grid.reduce<2>(v[0], v[1], [&](double a, double b) { fin_xr(&S, a, b); });
        if (!ok) break;
    }
    finish(S, st, !ok);
}

// Dynamic shared memory of the kernels at most: the axis tables of
// resident_available, the packed colours of one block, or three coefficients
// per plane.
constexpr size_t AXIS_SMEM = 200 * 1024, PACKED_SMEM = 150 * 1024, RESIDENT_SMEM = 208 * 1024;

// false when the device does not hold the blocks together after all (it can
// have fewer multiprocessors to give than it reports): nothing was launched
template <typename K, typename... Args>
bool cooperative(const LaunchCtx &L, K kernel, int blocks, int threads, size_t smem, Args... args) {
    void *ptrs[] = {(void *)&args...};
    L.pre(KK_RESIDENT);
    const cudaError_t e =
        cudaLaunchCooperativeKernel((const void *)kernel, dim3(blocks), dim3(threads), ptrs, smem, L.s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return false;
    }
    DALM_CUDA(e);
    L.post(KK_RESIDENT);
    return true;
}

template <int U, bool MEM>
bool resident_bicg(const LaunchCtx &L, const Grid &g, const PoissonCoef &C, const PoissonBufs &B,
                   const PoissonConfig &cfg, long long budget, double *part, unsigned *sync,
                   KrylovState *st) {
    const Columns Q = Columns::make(cfg.seg.box, U);
    return cooperative(L, k_resident_bicg<U, MEM>, (int)((Q.threads + RT - 1) / RT), RT,
                       3 * sizeof(double) * (size_t)(g.ni() + U), g, C, Q, B, budget, part, sync, st);
}

}  // namespace

bool resident_available(const PoissonConfig &cfg, const Grid &g) {
    if (cfg.reference_sums) return false;
    if (cfg.method == PM_BICG && !(cfg.pc == PC_JACOBI ? cfg.pc_sweeps == 3 : cfg.pc_sweeps >= 1))
        return false;
    const unsigned long long cells = (unsigned long long)g.ni() * g.nj() * g.nk();
    if (cfg.method == PM_BICG && cfg.pc == PC_JACOBI &&
        Columns::make(cfg.seg.box, 8).threads > (unsigned)cfg.sm_count * RT)
        return false;
    // Divisor's range, and the axis tables' shared memory
    return g.nj() >= 2 && g.nk() >= 3 && cells * (unsigned long long)(g.nj() + g.nk()) < (1ull << 32) &&
           AxisCoef::bytes(g) <= AXIS_SMEM;
}

void prepare_resident(const PoissonConfig &cfg) {
    if (cfg.method == PM_SOR) {
        allow_shared(k_resident_sor_regs<true>, RESIDENT_SMEM);
        allow_shared(k_resident_sor_regs<false>, RESIDENT_SMEM);
        allow_shared(k_resident_sor, RESIDENT_SMEM);
    } else if (cfg.method == PM_JACOBI) {
        allow_shared(k_resident_jacobi, RESIDENT_SMEM);
    } else if (cfg.pc == PC_SOR) {
        allow_shared(k_resident_bicg_sor, RESIDENT_SMEM);
    } else {
        allow_shared(k_resident_bicg<1, false>, RESIDENT_SMEM);
        allow_shared(k_resident_bicg<2, false>, RESIDENT_SMEM);
        allow_shared(k_resident_bicg<4, false>, RESIDENT_SMEM);
        allow_shared(k_resident_bicg<8, true>, RESIDENT_SMEM);
    }
}

bool launch_resident_solve(const LaunchCtx &L, const Grid &g, const PoissonCoef &C,
                           const PoissonBufs &B, const PoissonConfig &cfg, long long budget,
                           double *part, unsigned *sync, KrylovState *st) {
    const Cells cells = Cells::make(cfg.seg.box);
    const unsigned threads = (unsigned)cfg.sm_count * RT;
    DALM_CUDA(cudaMemsetAsync(sync, 0, 2 * sizeof(unsigned), L.s));
    // a count that no number of arrivals completes
    if (cfg.stall_waits) DALM_CUDA(cudaMemsetAsync(sync, 0xc0, sizeof(unsigned), L.s));
    if (cfg.method == PM_BICG && cfg.pc == PC_JACOBI) {
        // the fewest planes per thread that fit the grid on the device
        auto fits = [&](int planes) { return Columns::make(cfg.seg.box, planes).threads <= threads; };
        if (fits(1)) return resident_bicg<1, false>(L, g, C, B, cfg, budget, part, sync, st);
        if (fits(2)) return resident_bicg<2, false>(L, g, C, B, cfg, budget, part, sync, st);
        if (fits(4)) return resident_bicg<4, false>(L, g, C, B, cfg, budget, part, sync, st);
        return resident_bicg<8, true>(L, g, C, B, cfg, budget, part, sync, st);
    }
    // a grid of up to 8192 cells in one block, which needs no grid barrier;
    // else two cells of a colour per thread, at most a block per SM
    const unsigned want = (cells.half + 2 * RT - 1) / (2 * RT);
    const int blocks = cells.half <= 8 * RT ? 1 : (int)(want < (unsigned)cfg.sm_count ? want : cfg.sm_count);
    const size_t smem = AxisCoef::bytes(g);
    if (cfg.method == PM_SOR) {
        const Packed Q = Packed::make(cfg.seg.box);
        const size_t axis = 3 * sizeof(double) * (size_t)(Q.ni + SOR_UI), packed = 2 * sizeof(double) * (size_t)Q.total();
        if (Q.threads <= RT && packed <= PACKED_SMEM)
            return cooperative(L, k_resident_sor_regs<true>, 1, RT, axis + packed, g, C, cfg.seg.box, Q, B.x, B.tp,
                               B.ts, B.b, cfg.relax, budget, part, sync, st);
        if (Q.threads <= threads)
            return cooperative(L, k_resident_sor_regs<false>, (int)((Q.threads + RT - 1) / RT), RT, axis, g, C,
                               cfg.seg.box, Q, B.x, B.tp, B.ts, B.b, cfg.relax, budget, part, sync, st);
        return cooperative(L, k_resident_sor, blocks, RT, smem, g, C, cells, B.x, B.tp, B.b, cfg.relax, budget,
                           part, sync, st);
    }
    if (cfg.method == PM_JACOBI)
        return cooperative(L, k_resident_jacobi, blocks, RT, smem, g, C, cells, B.x, B.tp, B.b, budget, part,
                           sync, st);
    return cooperative(L, k_resident_bicg_sor, blocks, RT, smem, g, C, cells, B, cfg.pc_sweeps, cfg.pc_relax,
                       budget, part, sync, st);
}

}  // namespace dalm
