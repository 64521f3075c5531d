// FP64 stencil kernels of one time step.
//
// Compiled with --fmad=false: every expression keeps the reference's
// operation order and rounding (no contraction), so these stages agree with
// the reference bit for bit; the only libm call is cbrt in the eddy
// viscosity.
#include <algorithm>
#include <type_traits>

#include "flow.cuh"

namespace dalm {

namespace {

__device__ __forceinline__ double sgn(double v) { return (double)((v > 0.) - (v < 0.)); }

// The smooth van Albada limiter (DALM_LIMITER_VAN_ALBADA, an extension: the
// reference has only the limiter above): the face value of a cell with
// backward / forward differences a, b is  f +- (s/4)[(1 - k s) a + (1 + k s) b]
// with the switch s = (2ab + eps)/(a^2 + b^2 + eps) (van Albada, van Leer &
// Roberts 1982, in the kappa-MUSCL form), eps = 1e-12; differentiable
// everywhere, unlike the b=4 limiter.
__device__ __forceinline__ double va_switch(double a, double b) {
    const double eps = 1e-12;
    return (2. * a * b + eps) / (a * a + b * b + eps);
}

// The b = (3 - kappa) / (1 - kappa) limiter term s_a max(0, min(|a|, s_a bb b))
// (src/cfd.h:37-54) from a and t = bb b: the smaller of the two if they have
// the same sign, else 0.  EX: also where one of them is NaN, which the
// reference's minimum ignores.
template <bool EX>
__device__ __forceinline__ double limited(double a, double t) {
    if (EX) {
        const double s = sgn(a);
        return s * fmax(0., fmin(fabs(a), s * t));
    }
    const double m = fabs(t) < fabs(a) ? t : a;
    return (__double2hiint(a) ^ __double2hiint(t)) >= 0 ? m : 0.0;
}

// kappa = 1/3 MUSCL states on both sides of the face between cells c and
// p = c + 1 from the differences d2 = fc - fm, d3 = fp - fc, d4 = fpp - fp,
// and the upwind flux (src/cfd.h:37-60).  The reference forms a face's states
// once for each of the two cells; they are the same operations on the same
// values, so computing the face once gives both cells' bits.
template <int LIM, bool EX>
__device__ __forceinline__ double face_flux(double fc, double fp, double d2, double d3, double d4,
                                            double J) {
    const double kap = 1. / 3.;
    const double bb = (3. - kap) / (1. - kap);
    double l, r;
    if (LIM == 1) {
        const double sp = va_switch(d4, d3), sc = va_switch(d3, d2);
        r = fp - (sp / 4.) * ((1. - kap * sp) * d4 + (1. + kap * sp) * d3);
        l = fc + (sc / 4.) * ((1. - kap * sc) * d2 + (1. + kap * sc) * d3);
    } else {
        const double t2 = bb * d2, t3 = bb * d3, t4 = bb * d4;
        const double g6 = limited<EX>(d4, t3), g5 = limited<EX>(d3, t4);
        const double g4 = limited<EX>(d3, t2), g3 = limited<EX>(d2, t3);
        r = fp - 0.25 * ((1. - kap) * g6 + (1. + kap) * g5);
        l = fc + 0.25 * ((1. - kap) * g3 + (1. + kap) * g4);
    }
    return 0.5 * (J * (r + l) - fabs(J) * (r - l));
}

__device__ __forceinline__ double sq(double v) { return v * v; }

// Loop over the cells of a Segments box: each block takes (32 k) x (8 j)
// column segments and marches along i, so the per-cell index arithmetic is
// done once per segment instead of per cell.  The body sees i, j, k;
// `continue` skips to the next cell.
#define TILE_LOOP(S)                                                      \
    for (int u_ = blockIdx.x; u_ < (S).count; u_ += gridDim.x) {          \
        int i0_, i1_, j, k;                                               \
        if (!(S).column(u_, i0_, i1_, j, k)) continue;                    \
        for (int i = i0_; i < i1_; i++) {
#define TILE_END \
        }        \
    }

// Smagorinsky viscosity at (i,j,k) from the velocity (src/cfd.h:786-825).
// The filter factor (Cs cbrt(dx dy dz))^2 comes precomputed per cell.
__device__ __forceinline__ double smagorinsky(const StepParams &P, Vec3<const double> U, int i,
                                              int j, int k) {
    const Grid &g = P.g;
    long long c = g.at(i, j, k);
    long long e = g.at(i + 1, j, k), w = g.at(i - 1, j, k), n = g.at(i, j + 1, k),
              s = g.at(i, j - 1, k), t = c + 1, b = c - 1;
    double dxew = P.m.x[i + 1] - P.m.x[i - 1];
    double dyns = P.m.y[j + 1] - P.m.y[j - 1];
    double dztb = P.m.z[k + 1] - P.m.z[k - 1];
    double dudx = (U.c[0][e] - U.c[0][w]) / dxew;
    double dudy = (U.c[0][n] - U.c[0][s]) / dyns;
    double dudz = (U.c[0][t] - U.c[0][b]) / dztb;
    double dvdx = (U.c[1][e] - U.c[1][w]) / dxew;
    double dvdy = (U.c[1][n] - U.c[1][s]) / dyns;
    double dvdz = (U.c[1][t] - U.c[1][b]) / dztb;
    double dwdx = (U.c[2][e] - U.c[2][w]) / dxew;
    double dwdy = (U.c[2][n] - U.c[2][s]) / dyns;
    double dwdz = (U.c[2][t] - U.c[2][b]) / dztb;
    double s1 = 2 * sq(dudx), s2 = 2 * sq(dvdy), s3 = 2 * sq(dwdz);
    double s4 = sq(dudy + dvdx), s5 = sq(dudz + dwdx), s6 = sq(dvdz + dwdy);
    double shear = sqrt(s1 + s2 + s3 + s4 + s5 + s6);
    return P.filter2[c] * shear;
}

// ---------------------------------------------------------------- predictor
//
// cpy_array(Uold, U) + calc_intermediate_U (src/solver.h:1042-1053,
// src/cfd.h:176-322).  The copy is a buffer swap on the host; this kernel
// writes the interior of the new buffer and the guide cells at the ends of
// its k rows, k_copy_guides the other guide cells.  nut is the Smagorinsky
// viscosity of Uold, which is exactly the array the reference computed at
// the end of the previous step (calc_nut after apply_Ubc,
// src/solver.h:1157-1164), so it is evaluated inline.
//
// A block marches a column segment along i.  Each thread keeps its column's
// five i-neighbours in a register ring, and the current plane with a two-cell
// halo in j and k is staged in shared memory (double-buffered, one barrier
// per plane, the next plane's loads in flight meanwhile).  The x face of a
// cell is the next plane's west face and is carried; the y and z faces are
// computed by both cells, which share half of their limiter terms.
//
// Quotients by spacings are div_near's while every value that the block has
// loaded lies in its range, which a thread tests for the values it loads
// (a branch in every quotient: 1.75 ms on 512 x 256 x 128, this 1.23); else
// divisions.
//
// Bound by FP64 issue and latency (its bytes would take 0.25 ms on
// 512 x 256 x 128; the FP64 pipe is 47 % busy).  There: 1.23 ms, against
// 3.40 ms with 36 divisions a cell, six limiter terms per face pair through
// fmin / fmax, and every neighbour loaded through 64-bit indices.
constexpr int PR = TJ + 4, PCOL = TK + 4;  // plane with halo: 12 x 36
template <int LIM>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_predict(StepParams P, Segments T, Vec3<const double> V, Vec3<double> Un, Vec3<const double> JU,
          Vec3<const double> F) {
    __shared__ double plane[2][3][PR][PCOL];
    const Grid &g = P.g;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int sx = (int)g.sx, sy = (int)g.sy;
    int i0, i1, j, k;
    const bool valid = T.column(blockIdx.x, i0, i1, j, k);
    const bool inmem = j < g.ny && k < g.nz;
    const int j0 = j - row, k0 = k - lane;
    const int c0 = inmem ? (int)g.at(i0, j, k) : 0;
    // this thread's halo cell of a plane: warps 0-3 the rows j0-2, j0-1,
    // j0+8, j0+9, warp 4 the columns k0-2, k0-1, k0+32, k0+33 of the 8 rows
    int hrow = -1, hcol = 0, hc = 0;
    if (row < 4) {
        const int r = row < 2 ? row : row + TJ, jj = j0 - 2 + r;
        if (jj >= 0 && jj < g.ny && k < g.nz) hrow = r, hcol = lane + 2, hc = (int)g.at(i0, jj, k);
    } else if (row == 4) {
        const int q = lane >> 3, rr = lane & 7, col = q < 2 ? q : q + TK;
        const int kk = k0 - 2 + col, jj = j0 + rr;
        if (kk >= 0 && kk < g.nz && jj < g.ny) hrow = rr + 2, hcol = col, hc = (int)g.at(i0, jj, kk);
    }
    double ring[3][5];
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
        for (int d = 0; d < 5; d++) ring[m][d] = inmem ? V.c[m][c0 + (d - 2) * sx] : 0.0;
    // the column's y and z spacings and their reciprocals, in shared memory:
    // in registers they would be spilled
    enum { D = 0, UP, DN, CC, RD, RUP, RDN, RCC, NAX };
    __shared__ double ya[NAX][TJ], za[NAX][TK];
    auto axis = [&](int a, const double *x, const double *dd, int n, double *o, int stride) {
        o[D * stride] = dd[n];
        o[UP * stride] = x[n + 1] - x[n];
        o[DN * stride] = x[n] - x[n - 1];
        o[CC * stride] = x[n + 1] - x[n - 1];
        o[RD * stride] = P.invd[a][n];
        o[RUP * stride] = P.inv[a][n].x;
        o[RDN * stride] = P.inv[a][n - 1].x;
        o[RCC * stride] = P.inv[a][n].y;
    };
    if (lane == 0 && j < T.box.hi[1]) axis(1, P.m.y, P.m.dy, j, &ya[0][row], TJ);
    if (row == 0 && k < T.box.hi[2]) axis(2, P.m.z, P.m.dz, k, &za[0][lane], TK);
#pragma unroll
    for (int m = 0; m < 3; m++) {
        plane[0][m][row + 2][lane + 2] = ring[m][2];
        if (hrow >= 0) plane[0][m][hrow][hcol] = V.c[m][hc];
    }
    const double rre = 1 / P.re;
    // far: a value that the block has loaded is neither 0 nor within 2^-760 to
    // 2^200.  Without one, differences of values are 0 or at least 2^-812, and
    // differences of their quotients by spacings within 2^-100 to 2^100 at
    // least 2^-965: div_near's range.
    bool far = false;
#pragma unroll
    for (int m = 0; m < 3; m++) {
#pragma unroll
        for (int d = 0; d < 5; d++) far |= is_far<-760, 200>(ring[m][d]);
        if (hrow >= 0) far |= is_far<-760, 200>(plane[0][m][hrow][hcol]);
    }
    far = __syncthreads_or(far);
    double fW[3] = {0, 0, 0};
    if (valid) {
        const double JUW = JU.c[0][c0 - sx];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const double d2 = ring[m][1] - ring[m][0], d3 = ring[m][2] - ring[m][1], d4 = ring[m][3] - ring[m][2];
            fW[m] = far ? face_flux<LIM, true>(ring[m][1], ring[m][2], d2, d3, d4, JUW)
                        : face_flux<LIM, false>(ring[m][1], ring[m][2], d2, d3, d4, JUW);
        }
    }
    for (int i = i0; i < i1; i++) {
        const int b = (i - i0) & 1, c = c0 + (i - i0) * sx;
        const bool more = i + 1 < i1;
        double nxt[3];
        if (more) {
#pragma unroll
            for (int m = 0; m < 3; m++) {
                nxt[m] = inmem ? V.c[m][c + 3 * sx] : 0.0;
                if (hrow >= 0)
                    cp_async8((unsigned)__cvta_generic_to_shared(&plane[b ^ 1][m][hrow][hcol]),
                              V.c[m] + hc + (i + 1 - i0) * sx, true);
            }
            cp_async_commit();
        }
        auto cell = [&](auto exact) {
            constexpr bool EX = decltype(exact)::value;
            auto quot = [](double a, double d, double y) { return EX ? a / d : div_near(a, d, y); };
            const double JE = JU.c[0][c], JN = JU.c[1][c], JS = JU.c[1][c - sy], JT = JU.c[2][c],
                         JB = JU.c[2][c - 1], filter = P.filter2[c];
            const double dx = P.m.dx[i], idx = P.invd[0][i];
            const double xe = P.m.x[i + 1], xi = P.m.x[i], xw = P.m.x[i - 1];
            const double2 ix = P.inv[0][i];
            const double ixW = P.inv[0][i - 1].x;
            // Smagorinsky viscosity (src/cfd.h:786-825)
            double visc;
            {
                double G[3][3];
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    const double(*t)[PCOL] = plane[b][m];
                    G[m][0] = quot(ring[m][3] - ring[m][1], xe - xw, ix.y);
                    G[m][1] = quot(t[row + 3][lane + 2] - t[row + 1][lane + 2], ya[CC][row], ya[RCC][row]);
                    G[m][2] = quot(t[row + 2][lane + 3] - t[row + 2][lane + 1], za[CC][lane], za[RCC][lane]);
                }
                const double s1 = 2 * sq(G[0][0]), s2 = 2 * sq(G[1][1]), s3 = 2 * sq(G[2][2]);
                const double s4 = sq(G[0][1] + G[1][0]), s5 = sq(G[0][2] + G[2][0]),
                             s6 = sq(G[1][2] + G[2][1]);
                const double shear = sqrt(s1 + s2 + s3 + s4 + s5 + s6);
                visc = rre + filter * shear;
            }
            const double dy = ya[D][row], dz = za[D][lane];
            const double J = dx * dy * dz, iJ = 1 / J;
            const bool has_f = P.fbox.contains(i, j, k);
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const double(*t)[PCOL] = plane[b][m];
                const double fc = ring[m][2];
                const double e1 = ring[m][3] - fc, w1 = fc - ring[m][1];
                const double yn = t[row + 3][lane + 2], ys = t[row + 1][lane + 2];
                const double zt = t[row + 2][lane + 3], zb = t[row + 2][lane + 1];
                const double n1 = yn - fc, n2 = t[row + 4][lane + 2] - yn, s1 = fc - ys,
                             s2 = ys - t[row][lane + 2];
                const double t1 = zt - fc, t2 = t[row + 2][lane + 4] - zt, b1 = fc - zb,
                             b2 = zb - t[row + 2][lane];
                const double fE = face_flux<LIM, EX>(fc, ring[m][3], w1, e1, ring[m][4] - ring[m][3], JE);
                const double fN = face_flux<LIM, EX>(fc, yn, s1, n1, n2, JN);
                const double fS = face_flux<LIM, EX>(ys, fc, s2, s1, n1, JS);
                const double fT = face_flux<LIM, EX>(fc, zt, b1, t1, t2, JT);
                const double fB = face_flux<LIM, EX>(zb, fc, b2, b1, t1, JB);
                const double conv = div_by(fE - fW[m] + fN - fS + fT - fB, J, iJ);
                fW[m] = fE;
                const double diff =
                    visc * (quot(quot(e1, xe - xi, ix.x) - quot(w1, xi - xw, ixW), dx, idx) +
                            quot(quot(n1, ya[UP][row], ya[RUP][row]) -
                                       quot(s1, ya[DN][row], ya[RDN][row]), dy, ya[RD][row]) +
                            quot(quot(t1, za[UP][lane], za[RUP][lane]) -
                                       quot(b1, za[DN][lane], za[RDN][lane]), dz, za[RD][lane]));
                const double fm = has_f ? F.c[m][c] : 0.0;
                Un.c[m][c] = fc + P.dt * (-conv + diff + fm);
            }
        };
        if (valid) {
            if (far) cell(std::true_type{});
            else cell(std::false_type{});
            // the guide cells at the ends of this k row (U* = U^n there)
            if (k == g.gc || k == g.nz - g.gc - 1) {
                const int d = k == g.gc ? -1 : 1;
                for (int q = 1; q <= g.gc; q++)
#pragma unroll
                    for (int m = 0; m < 3; m++) Un.c[m][c + q * d] = V.c[m][c + q * d];
            }
        }
        if (more) {
#pragma unroll
            for (int m = 0; m < 3; m++) {
                plane[b ^ 1][m][row + 2][lane + 2] = ring[m][3];
                ring[m][0] = ring[m][1];
                ring[m][1] = ring[m][2];
                ring[m][2] = ring[m][3];
                ring[m][3] = ring[m][4];
                ring[m][4] = nxt[m];
            }
            cp_async_wait<0>();
#pragma unroll
            for (int m = 0; m < 3; m++) {
                far |= is_far<-760, 200>(nxt[m]);
                if (hrow >= 0) far |= is_far<-760, 200>(plane[b ^ 1][m][hrow][hcol]);
            }
        }
        far = __syncthreads_or(far);
    }
}

// U* = U^n on the guide cells of the rows (i, j) outside the interior: one
// warp per row, 2 gc planes of ny rows, then 2 gc strips of nx - 2 gc rows.
__global__ void __launch_bounds__(256) k_copy_guides(Grid g, Vec3<const double> V, Vec3<double> Un) {
    const int gc = g.gc, ni = g.nx - 2 * gc, lane = threadIdx.x & 31;
    const unsigned a = 2u * gc * g.ny, rows = a + 2u * gc * ni, nw = gridDim.x * (blockDim.x >> 5);
    for (unsigned r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += nw) {
        int i, j;
        if (r < a) {
            const int p = (int)(r / g.ny);
            i = p < gc ? p : g.nx - 2 * gc + p;
            j = (int)(r - (unsigned)p * g.ny);
        } else {
            const unsigned q = r - a;
            const int p = (int)(q / ni);
            j = p < gc ? p : g.ny - 2 * gc + p;
            i = gc + (int)(q - (unsigned)p * ni);
        }
        const long long c0 = g.at(i, j, 0);
        for (int k = lane; k < g.nz; k += 32)
#pragma unroll
            for (int m = 0; m < 3; m++) Un.c[m][c0 + k] = V.c[m][c0 + k];
    }
}

// ------------------------------------------- face fluxes, their BCs, RHS

// interpolate_JU face values (src/cfd.h:395-420) with apply_JUbc overrides
// (src/bc.h:235-302, inflow profile extension) for the faces the override
// touches.  Faces are identified by their lower cell (i,j,k).
__device__ __forceinline__ double face_x(const StepParams &P, Vec3<const double> U, int i, int j,
                                         int k) {
    const Grid &g = P.g;
    double yz = P.m.dy[j] * P.m.dz[k];
    if (i == g.gc - 1 && j >= g.gc && j < g.ny - g.gc && k >= g.gc && k < g.nz - g.gc) {
        double u = P.prof ? P.prof[((long long)j * g.nz + k) * 3] : P.uin[0];
        return yz * u;
    }
    return 0.5 * (U.c[0][g.at(i, j, k)] * yz + U.c[0][g.at(i + 1, j, k)] * yz);
}
__device__ __forceinline__ double face_y(const StepParams &P, Vec3<const double> U, int i, int j,
                                         int k) {
    const Grid &g = P.g;
    if ((j == g.gc - 1 || j == g.ny - g.gc - 1) && i >= g.gc && i < g.nx - g.gc && k >= g.gc &&
        k < g.nz - g.gc)
        return 0;
    double xz = P.m.dx[i] * P.m.dz[k];
    return 0.5 * (U.c[1][g.at(i, j, k)] * xz + U.c[1][g.at(i, j + 1, k)] * xz);
}
__device__ __forceinline__ double face_z(const StepParams &P, Vec3<const double> U, int i, int j,
                                         int k) {
    const Grid &g = P.g;
    if ((k == g.gc - 1 || k == g.nz - g.gc - 1) && i >= g.gc && i < g.nx - g.gc && j >= g.gc &&
        j < g.ny - g.gc)
        return 0;
    double xy = P.m.dx[i] * P.m.dy[j];
    return 0.5 * (U.c[2][g.at(i, j, k)] * xy + U.c[2][g.at(i, j, k + 1)] * xy);
}

// interpolate_JU + apply_JUbc + calc_poisson_rhs (src/solver.h:1055-1077).
// Covers faces i,j,k in [gc-1, N-gc).  Blocks [0, T.count) march the
// interior's column segments along i, carrying the west face and the centre
// velocity; the RHS's south and bottom faces are recomputed (same
// arithmetic, same bits).  512 x 256 x 128: 0.21 ms, 4.4 TB/s (0.40 ms over
// the face box, every face from scratch).
template <bool RHS>
__global__ void __launch_bounds__(TILE_THREADS)
k_flux_rhs(StepParams P, Segments T, Vec3<const double> U, Vec3<double> JU, double *b) {
    const Grid &g = P.g;
    if ((int)blockIdx.x >= T.count) {
        const long long step = (long long)(gridDim.x - T.count) * blockDim.x;
        for (long long n = (long long)(blockIdx.x - T.count) * blockDim.x + threadIdx.x;
             n < face_shell_cells(g); n += step) {
            int i, j, k;
            face_shell_cell(g, n, i, j, k);
            const long long c = g.at(i, j, k);
            JU.c[0][c] = face_x(P, U, i, j, k);
            JU.c[1][c] = face_y(P, U, i, j, k);
            JU.c[2][c] = face_z(P, U, i, j, k);
        }
        return;
    }
    int i0, i1, j, k;
    if (!T.column(blockIdx.x, i0, i1, j, k)) return;
    const int sx = (int)g.sx, sy = (int)g.sy;
    int c = (int)g.at(i0, j, k);
    const double dy = P.m.dy[j], dz = P.m.dz[k], yz = dy * dz;
    const bool wall_n = j == g.ny - g.gc - 1, wall_s = j == g.gc;
    const bool wall_t = k == g.nz - g.gc - 1, wall_b = k == g.gc;
    const double scale = P.dt * P.max_diag, iscale = 1 / scale;
    double u = U.c[0][c];
    double fw = RHS ? face_x(P, U, i0 - 1, j, k) : 0.0;
#pragma unroll 2
    for (int i = i0; i < i1; i++, c += sx) {
        const double ue = U.c[0][c + sx], v = U.c[1][c], vn = U.c[1][c + sy], w = U.c[2][c],
                     wt = U.c[2][c + 1];
        const double vs = RHS ? U.c[1][c - sy] : 0.0, wb = RHS ? U.c[2][c - 1] : 0.0;
        const double dx = P.m.dx[i], xz = dx * dz, xy = dx * dy;
        const double fe = 0.5 * (u * yz + ue * yz);
        const double fn = wall_n ? 0.0 : 0.5 * (v * xz + vn * xz);
        const double ft = wall_t ? 0.0 : 0.5 * (w * xy + wt * xy);
        JU.c[0][c] = fe;
        JU.c[1][c] = fn;
        JU.c[2][c] = ft;
        if (RHS) {
            const double fs = wall_s ? 0.0 : 0.5 * (vs * xz + v * xz);
            const double fb = wall_b ? 0.0 : 0.5 * (wb * xy + w * xy);
            const double J = dx * dy * dz;
            const double divergence = (fe - fw + fn - fs + ft - fb) / J;
            b[c] = div_by(divergence, scale, iscale);
        }
        fw = fe;
        u = ue;
    }
}

// ------------------------------------------------------------- projection

// apply_pbc (src/bc.h:304-411): one thread per guide cell of the six faces.
__global__ void k_pressure_bc(StepParams P, double *p) {
    const Grid &g = P.g;
    int GC = g.gc;
    long long nyz = (long long)g.nj() * g.nk(), nxz = (long long)g.ni() * g.nk(),
              nxy = (long long)g.ni() * g.nj();
    long long tot = 2 * (nyz + nxz + nxy);
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < tot;
         n += (long long)gridDim.x * blockDim.x) {
        long long r = n;
        if (r < 2 * nyz) {
            int side = (int)(r / nyz);
            long long q = r % nyz;
            int j = GC + (int)(q / g.nk()), k = GC + (int)(q % g.nk());
            if (side == 0) {
                p[g.at(GC - 1, j, k)] = p[g.at(GC, j, k)];
            } else {
                int ii = g.nx - GC - 1, io = g.nx - GC;
                double hi = 0.5 * P.m.dx[ii], ho = 0.5 * P.m.dx[io], pbc = 0;
                p[g.at(io, j, k)] = pbc - (p[g.at(ii, j, k)] - pbc) * (ho / hi);
            }
            continue;
        }
        r -= 2 * nyz;
        if (r < 2 * nxz) {
            int side = (int)(r / nxz);
            long long q = r % nxz;
            int i = GC + (int)(q / g.nk()), k = GC + (int)(q % g.nk());
            if (side == 0) p[g.at(i, GC - 1, k)] = p[g.at(i, GC, k)];
            else p[g.at(i, g.ny - GC, k)] = p[g.at(i, g.ny - GC - 1, k)];
            continue;
        }
        r -= 2 * nxz;
        int side = (int)(r / nxy);
        long long q = r % nxy;
        int i = GC + (int)(q / g.nj()), j = GC + (int)(q % g.nj());
        if (side == 0) p[g.at(i, j, GC - 1)] = p[g.at(i, j, GC)];
        else p[g.at(i, j, g.nz - GC)] = p[g.at(i, j, g.nz - GC - 1)];
    }
}

// Projected face flux with the apply_JUbc override: project_p's compact
// correction (src/cfd.h:716-740) then the BC (src/bc.h:235-302).
__device__ __forceinline__ double proj_face(const StepParams &P, Vec3<double> JU, const double *p,
                                            int axis, int i, int j, int k) {
    const Grid &g = P.g;
    long long c = g.at(i, j, k);
    if (axis == 0) {
        if (i == g.gc - 1 && j >= g.gc && j < g.ny - g.gc && k >= g.gc && k < g.nz - g.gc) {
            double u = P.prof ? P.prof[((long long)j * g.nz + k) * 3] : P.uin[0];
            return (P.m.dy[j] * P.m.dz[k]) * u;
        }
        double yz = P.m.dy[j] * P.m.dz[k];
        double dpdx = (p[g.at(i + 1, j, k)] - p[c]) / (P.m.x[i + 1] - P.m.x[i]);
        return JU.c[0][c] - P.dt * yz * dpdx;
    } else if (axis == 1) {
        if ((j == g.gc - 1 || j == g.ny - g.gc - 1) && i >= g.gc && i < g.nx - g.gc &&
            k >= g.gc && k < g.nz - g.gc)
            return 0;
        double xz = P.m.dx[i] * P.m.dz[k];
        double dpdy = (p[g.at(i, j + 1, k)] - p[c]) / (P.m.y[j + 1] - P.m.y[j]);
        return JU.c[1][c] - P.dt * xz * dpdy;
    } else {
        if ((k == g.gc - 1 || k == g.nz - g.gc - 1) && i >= g.gc && i < g.nx - g.gc &&
            j >= g.gc && j < g.ny - g.gc)
            return 0;
        double xy = P.m.dx[i] * P.m.dy[j];
        double dpdz = (p[g.at(i, j, k + 1)] - p[c]) / (P.m.z[k + 1] - P.m.z[k]);
        return JU.c[2][c] - P.dt * xy * dpdz;
    }
}

// project_p (src/cfd.h:601-783) + set_solid_U + the apply_JUbc that follows it
// + calc_divergence norm + calc_max_cfl (src/solver.h:1122-1186).  The
// velocity BCs (apply_Ubc) run in k_velocity_bc after this kernel; they touch
// guide cells only, so the interior velocity used for the CFL here is final.
// A thread owns the three faces of its lower cell; the divergence of an
// interior cell also needs its west face, carried along the march, and its
// south and bottom faces, which it recomputes from the pre-projection flux.
// 512 x 256 x 128: 0.52 ms, 3.4 TB/s (0.95 ms over the face box, with eleven
// divisions a cell and the west face recomputed).
// Because other threads overwrite those faces in the same launch, the
// projected flux goes to a second buffer (JUout) and the host swaps the two.
// Blocks from T.count on take the faces below the interior.
__global__ void __launch_bounds__(TILE_THREADS, 3)
k_project(StepParams P, Segments T, Vec3<double> U, Vec3<double> JUin, Vec3<double> JUout,
          const double *p, Partials<2> part, DiagState *diag) {
    const Grid &g = P.g;
    double div2 = 0, cfl = 0;
    int i0, i1, j, k;
    if ((int)blockIdx.x >= T.count) {
        const long long step = (long long)(gridDim.x - T.count) * blockDim.x;
        for (long long n = (long long)(blockIdx.x - T.count) * blockDim.x + threadIdx.x;
             n < face_shell_cells(g); n += step) {
            face_shell_cell(g, n, i0, j, k);
            const long long c = g.at(i0, j, k);
#pragma unroll
            for (int a = 0; a < 3; a++) JUout.c[a][c] = proj_face(P, JUin, p, a, i0, j, k);
        }
    } else if (T.column(blockIdx.x, i0, i1, j, k)) {
        const int sx = (int)g.sx, sy = (int)g.sy;
        int c = (int)g.at(i0, j, k);
        const double dt = P.dt, dy = P.m.dy[j], dz = P.m.dz[k], yz = dy * dz;
        const bool wall_n = j == g.ny - g.gc - 1, wall_s = j == g.gc;
        const bool wall_t = k == g.nz - g.gc - 1, wall_b = k == g.gc;
        const double yN = P.m.y[j + 1] - P.m.y[j], yS = P.m.y[j] - P.m.y[j - 1],
                     yC = P.m.y[j + 1] - P.m.y[j - 1];
        const double zT = P.m.z[k + 1] - P.m.z[k], zB = P.m.z[k] - P.m.z[k - 1],
                     zC = P.m.z[k + 1] - P.m.z[k - 1];
        const double2 iy = P.inv[1][j], iz = P.inv[2][k];
        const double iyS = P.inv[1][j - 1].x, izB = P.inv[2][k - 1].x;
        const double idy = P.invd[1][j], idz = P.invd[2][k];
        double pw = p[c - sx], pc = p[c];
        double fw = proj_face(P, JUin, p, 0, i0 - 1, j, k);
        for (int i = i0; i < i1; i++, c += sx) {
            const double pe = p[c + sx], pn = p[c + sy], ps = p[c - sy], pt = p[c + 1], pb = p[c - 1];
            const double ju = JUin.c[0][c], jv = JUin.c[1][c], jvs = JUin.c[1][c - sy],
                         jw = JUin.c[2][c], jwb = JUin.c[2][c - 1];
            double u = U.c[0][c], v = U.c[1][c], w = U.c[2][c];
            const double dx = P.m.dx[i], xz = dx * dz, xy = dx * dy;
            const double2 ix = P.inv[0][i];
            double q[8] = {pe - pc, pn - pc, pt - pc, pc - ps, pc - pb, dt * (pe - pw), dt * (pn - ps), dt * (pt - pb)};
            const double by[8] = {P.m.x[i + 1] - P.m.x[i], yN, zT, yS, zB, P.m.x[i + 1] - P.m.x[i - 1], yC, zC};
            const double rb[8] = {ix.x, iy.x, iz.x, iyS, izB, ix.y, iy.y, iz.y};
            divs_by(q, by, rb);
            const double fe = ju - dt * yz * q[0];
            const double fn = wall_n ? 0.0 : jv - dt * xz * q[1];
            const double ft = wall_t ? 0.0 : jw - dt * xy * q[2];
            JUout.c[0][c] = fe;
            JUout.c[1][c] = fn;
            JUout.c[2][c] = ft;
            u = u - q[5];
            v = v - q[6];
            w = w - q[7];
            if (P.solid) {  // set_solid_U (src/cfd.h:1143-1160)
                const double sf = P.solid[c];
                u = (1. - sf) * u;
                v = (1. - sf) * v;
                w = (1. - sf) * w;
            }
            U.c[0][c] = u;
            U.c[1][c] = v;
            U.c[2][c] = w;
            const double fs = wall_s ? 0.0 : jvs - dt * xz * q[3];
            const double fb = wall_b ? 0.0 : jwb - dt * xy * q[4];
            const double J = dx * dy * dz;
            const double d = (fe - fw + fn - fs + ft - fb) / J;
            div2 += d * d;
            double co[3] = {fabs(u) * dt, fabs(v) * dt, fabs(w) * dt};
            divs_by(co, {dx, dy, dz}, {P.invd[0][i], idy, idz});
            const double local = co[0] + co[1] + co[2];
            cfl = local > cfl ? local : cfl;
            fw = fe;
            pw = pc;
            pc = pe;
        }
    }
    if (P.reference_sums) return;  // k_seq_diag sums in the reference's order
    double v[2] = {div2, cfl};
    if (grid_reduce<2>(v, 2u, part) && threadIdx.x == 0) {
        diag->div2 = v[0];
        diag->max_cfl = v[1];
        diag->avg_div = sqrt(v[0]) / sqrt(diag->ncell);
    }
}

// divergence of cell c from the face fluxes (src/cfd.h:1093-1105) and the
// cell CFL number (src/cfd.h:1126-1130)
template <typename T>
__device__ __forceinline__ double cell_div(const StepParams &P, Vec3<const T> JU, int i, int j,
                                           int k) {
    const Grid &g = P.g;
    long long c = g.at(i, j, k);
    double J = P.m.dx[i] * P.m.dy[j] * P.m.dz[k];
    return ((double)JU.c[0][c] - (double)JU.c[0][g.at(i - 1, j, k)] + (double)JU.c[1][c] -
            (double)JU.c[1][g.at(i, j - 1, k)] + (double)JU.c[2][c] - (double)JU.c[2][c - 1]) / J;
}
template <typename T>
__device__ __forceinline__ double cell_cfl(const StepParams &P, Vec3<const T> U, int i, int j,
                                           int k) {
    long long c = P.g.at(i, j, k);
    return fabs((double)U.c[0][c]) * P.dt / P.m.dx[i] + fabs((double)U.c[1][c]) * P.dt / P.m.dy[j] +
           fabs((double)U.c[2][c]) * P.dt / P.m.dz[k];
}

// Diagnostics alone (after set_state): sum div^2 and max CFL.
template <typename T>
__global__ void __launch_bounds__(TILE_THREADS)
k_diag(StepParams P, Segments S, Vec3<const T> U, Vec3<const T> JU, Partials<2> part,
       DiagState *diag) {
    double div2 = 0, cfl = 0;
    TILE_LOOP(S)
        double d = cell_div(P, JU, i, j, k);
        div2 += d * d;
        double local = cell_cfl(P, U, i, j, k);
        cfl = local > cfl ? local : cfl;
    TILE_END
    double v[2] = {div2, cfl};
    if (grid_reduce<2>(v, 2u, part) && threadIdx.x == 0) {
        diag->div2 = v[0];
        diag->max_cfl = v[1];
        diag->avg_div = sqrt(v[0]) / sqrt(diag->ncell);
    }
}

// The same diagnostics summed in the reference's serial order by one warp:
// calc_l2_norm(div) (src/mv.h:33-55) and calc_max_cfl (src/cfd.h:1109-1141).
__global__ void k_seq_diag(StepParams P, Vec3<const double> U, Vec3<const double> JU,
                           DiagState *diag) {
    const Grid &g = P.g;
    double tot[2];
    warp_serial_sums<2>(
        g,
        [&](long long c, double (&t)[2]) {
            long long r = c - g.off;
            int i = (int)(r / g.sx), j = (int)((r % g.sx) / g.sy), k = (int)(r % g.sy);
            double d = cell_div(P, JU, i, j, k);
            t[0] = d * d;
            t[1] = 0;
        },
        tot);
    // max is exact in any order
    double cfl = 0;
    int lane = threadIdx.x & 31;
    for (int i = g.gc; i < g.nx - g.gc; i++)
        for (int j = g.gc; j < g.ny - g.gc; j++)
            for (int k = g.gc + lane; k < g.nz - g.gc; k += 32) {
                double local = cell_cfl(P, U, i, j, k);
                cfl = local > cfl ? local : cfl;
            }
    for (int o = 16; o > 0; o >>= 1) {
        double other = __shfl_down_sync(0xffffffffu, cfl, o);
        cfl = other > cfl ? other : cfl;
    }
    if (lane == 0) {
        diag->div2 = tot[0];
        diag->max_cfl = cfl;
        diag->avg_div = sqrt(tot[0]) / sqrt(diag->ncell);
    }
}

// Three-point Lagrange extrapolation (src/util.h:201-212).
__device__ __forceinline__ double quad_poly(double x0, double x1, double x2, double f0, double f1,
                                            double f2, double x3) {
    double l0 = ((x3 - x1) * (x3 - x2)) / ((x0 - x1) * (x0 - x2));
    double l1 = ((x3 - x0) * (x3 - x2)) / ((x1 - x0) * (x1 - x2));
    double l2 = ((x3 - x0) * (x3 - x1)) / ((x2 - x0) * (x2 - x1));
    return f0 * l0 + f1 * l1 + f2 * l2;
}

// apply_Ubc (src/bc.h:5-233): inflow (uniform Uin or profile), convective
// outflow on Uold, slip y-/y+/z+, no-slip z-.  One thread per face column;
// each writes the gc guide cells of its column.  Reads only interior cells
// of U and the old guide values, so the faces are independent.
// T is the storage type of U (double; float for the FP32 stencil fields of
// the mixed form): the arithmetic is FP64 either way.
template <typename T>
__global__ void k_velocity_bc(StepParams P, Vec3<T> U, Vec3<const T> V) {
    const Grid &g = P.g;
    int GC = g.gc;
    long long nyz = (long long)g.nj() * g.nk(), nxz = (long long)g.ni() * g.nk(),
              nxy = (long long)g.ni() * g.nj();
    long long tot = 2 * (nyz + nxz + nxy);
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < tot;
         n += (long long)gridDim.x * blockDim.x) {
        long long r = n;
        if (r < 2 * nyz) {
            int side = (int)(r / nyz);
            long long q = r % nyz;
            int j = GC + (int)(q / g.nk()), k = GC + (int)(q % g.nk());
            if (side == 0) {
                for (int i = 0; i < GC; i++) {
                    long long id = g.at(i, j, k);
                    for (int m = 0; m < 3; m++)
                        U.c[m][id] = (T)(P.prof ? P.prof[((long long)j * g.nz + k) * 3 + m] : P.uin[m]);
                }
            } else {
                for (int i = g.nx - GC; i < g.nx; i++) {
                    long long i0 = g.at(i, j, k), i1 = g.at(i - 1, j, k), i2 = g.at(i - 2, j, k);
                    double uout = (double)U.c[0][i0];
                    double nv[3];
                    for (int m = 0; m < 3; m++) {
                        double f0 = (double)V.c[m][i0], f1 = (double)V.c[m][i1], f2 = (double)V.c[m][i2];
                        double grad = (3 * f0 - 4 * f1 + f2) / 2;
                        nv[m] = f0 - uout * P.dt * grad / P.m.dx[i];
                    }
                    for (int m = 0; m < 3; m++) U.c[m][i0] = (T)nv[m];
                }
            }
            continue;
        }
        r -= 2 * nyz;
        if (r < 2 * nxz) {
            int side = (int)(r / nxz);
            long long q = r % nxz;
            int i = GC + (int)(q / g.nk()), k = GC + (int)(q % g.nk());
            int j0 = side ? g.ny - GC - 2 : GC + 1, j1 = side ? g.ny - GC - 1 : GC;
            int j3 = side ? g.ny - GC : GC - 1, j4 = side ? g.ny - GC + 1 : GC - 2;
            long long a0 = g.at(i, j0, k), a1 = g.at(i, j1, k), a3 = g.at(i, j3, k),
                      a4 = g.at(i, j4, k);
            double y0 = P.m.y[j0], y1 = P.m.y[j1];
            double y2 = side ? P.m.y[j1] + 0.5 * P.m.dy[j1] : P.m.y[j1] - 0.5 * P.m.dy[j1];
            double y3 = P.m.y[j3], y4 = P.m.y[j4];
            double ubc[3] = {(double)U.c[0][a1], 0, (double)U.c[2][a1]};
            for (int m = 0; m < 3; m++) {
                double f0 = (double)U.c[m][a0], f1 = (double)U.c[m][a1], f2 = ubc[m];
                U.c[m][a3] = (T)quad_poly(y0, y1, y2, f0, f1, f2, y3);
                U.c[m][a4] = (T)quad_poly(y0, y1, y2, f0, f1, f2, y4);
            }
            continue;
        }
        r -= 2 * nxz;
        int side = (int)(r / nxy);
        long long q = r % nxy;
        int i = GC + (int)(q / g.nj()), j = GC + (int)(q % g.nj());
        int k0 = side ? g.nz - GC - 2 : GC + 1, k1 = side ? g.nz - GC - 1 : GC;
        int k3 = side ? g.nz - GC : GC - 1, k4 = side ? g.nz - GC + 1 : GC - 2;
        long long a0 = g.at(i, j, k0), a1 = g.at(i, j, k1), a3 = g.at(i, j, k3),
                  a4 = g.at(i, j, k4);
        double z0 = P.m.z[k0], z1 = P.m.z[k1];
        double z2 = side ? P.m.z[k1] + 0.5 * P.m.dz[k1] : P.m.z[k1] - 0.5 * P.m.dz[k1];
        double z3 = P.m.z[k3], z4 = P.m.z[k4];
        double ubc[3] = {0, 0, 0};
        // z+ slip; z- no slip, or slip upstream of a retracted floor's start
        // (src/bc.h:140-160)
        if (side || (P.retracted && P.m.x[i] < P.floor_start)) {
            ubc[0] = (double)U.c[0][a1];
            ubc[1] = (double)U.c[1][a1];
        }
        for (int m = 0; m < 3; m++) {
            double f0 = (double)U.c[m][a0], f1 = (double)U.c[m][a1], f2 = ubc[m];
            U.c[m][a3] = (T)quad_poly(z0, z1, z2, f0, f1, f2, z3);
            U.c[m][a4] = (T)quad_poly(z0, z1, z2, f0, f1, f2, z4);
        }
    }
}

__global__ void __launch_bounds__(TILE_THREADS)
k_nut_field(StepParams P, Segments T, Vec3<const double> U, double *nut) {
    TILE_LOOP(T)
        nut[P.g.at(i, j, k)] = smagorinsky(P, U, i, j, k);
    TILE_END
}

__global__ void __launch_bounds__(TILE_THREADS)
k_div_field(StepParams P, Segments T, Vec3<const double> JU, double *div) {
    const Grid &g = P.g;
    TILE_LOOP(T)
        long long c = g.at(i, j, k);
        double J = P.m.dx[i] * P.m.dy[j] * P.m.dz[k];
        div[c] = (JU.c[0][c] - JU.c[0][g.at(i - 1, j, k)] + JU.c[1][c] -
                  JU.c[1][g.at(i, j - 1, k)] + JU.c[2][c] - JU.c[2][c - 1]) / J;
    TILE_END
}

// Q-criterion on the interior (calc_q_at_cell, src/cfd.h:949-975): central
// differences over x[i+1] - x[i-1] etc., same operation order.
__global__ void __launch_bounds__(TILE_THREADS)
k_q_field(StepParams P, Segments T, Vec3<const double> U, double *q) {
    const Grid &g = P.g;
    TILE_LOOP(T)
        const long long c = g.at(i, j, k);
        const long long ce = g.at(i + 1, j, k), cw = g.at(i - 1, j, k);
        const long long cn = g.at(i, j + 1, k), cs = g.at(i, j - 1, k);
        const long long ct = c + 1, cb = c - 1;
        const double dxew = P.m.x[i + 1] - P.m.x[i - 1];
        const double dyns = P.m.y[j + 1] - P.m.y[j - 1];
        const double dztb = P.m.z[k + 1] - P.m.z[k - 1];
        const double dudx = (U.c[0][ce] - U.c[0][cw]) / dxew;
        const double dudy = (U.c[0][cn] - U.c[0][cs]) / dyns;
        const double dudz = (U.c[0][ct] - U.c[0][cb]) / dztb;
        const double dvdx = (U.c[1][ce] - U.c[1][cw]) / dxew;
        const double dvdy = (U.c[1][cn] - U.c[1][cs]) / dyns;
        const double dvdz = (U.c[1][ct] - U.c[1][cb]) / dztb;
        const double dwdx = (U.c[2][ce] - U.c[2][cw]) / dxew;
        const double dwdy = (U.c[2][cn] - U.c[2][cs]) / dyns;
        const double dwdz = (U.c[2][ct] - U.c[2][cb]) / dztb;
        q[c] = -0.5 * (dudx * dudx + dvdy * dvdy + dwdz * dwdz +
                       2 * (dudy * dvdx + dudz * dwdx + dvdz * dwdy));
    TILE_END
}

// Running time average over every stored cell (calc_ax_plus_by,
// src/mv.h:322-335 as used at src/solver.h:1198-1203).
template <typename T>
__global__ void k_tavg(Grid g, Vec3<double> A, Vec3<const T> U, double w) {
    long long tot = (long long)g.nx * g.ny * g.nz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < tot;
         n += (long long)gridDim.x * blockDim.x) {
        int k = (int)(n % g.nz);
        long long r = n / g.nz;
        int j = (int)(r % g.ny), i = (int)(r / g.ny);
        long long c = g.at(i, j, k);
        for (int m = 0; m < 3; m++) A.c[m][c] = (1. - w) * A.c[m][c] + w * (double)U.c[m][c];
    }
}

__global__ void k_to_device(Grid g, const double *ref, int nc, double *d0, double *d1, double *d2) {
    long long tot = (long long)g.nx * g.ny * g.nz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < tot;
         n += (long long)gridDim.x * blockDim.x) {
        int k = (int)(n % g.nz);
        long long r = n / g.nz;
        int j = (int)(r % g.ny), i = (int)(r / g.ny);
        long long c = g.at(i, j, k);
        if (nc == 1) {
            d0[c] = ref[n];
        } else {
            d0[c] = ref[3 * n];
            d1[c] = ref[3 * n + 1];
            d2[c] = ref[3 * n + 2];
        }
    }
}

__global__ void k_to_ref(Grid g, const double *s0, const double *s1, const double *s2, int nc,
                         double *ref) {
    long long tot = (long long)g.nx * g.ny * g.nz;
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < tot;
         n += (long long)gridDim.x * blockDim.x) {
        int k = (int)(n % g.nz);
        long long r = n / g.nz;
        int j = (int)(r % g.ny), i = (int)(r / g.ny);
        long long c = g.at(i, j, k);
        if (nc == 1) {
            ref[n] = s0[c];
        } else {
            ref[3 * n] = s0[c];
            ref[3 * n + 1] = s1[c];
            ref[3 * n + 2] = s2[c];
        }
    }
}

__global__ void k_fill(double *p, long long n, double v) {
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n;
         x += (long long)gridDim.x * blockDim.x)
        p[x] = v;
}

Box interior_box(const Grid &g) {
    return Box{{g.gc, g.gc, g.gc}, {g.nx - g.gc, g.ny - g.gc, g.nz - g.gc}};
}

int plane_blocks(const Grid &g) {
    long long tot = 2 * ((long long)g.nj() * g.nk() + (long long)g.ni() * g.nk() +
                         (long long)g.ni() * g.nj());
    long long b = (tot + 255) / 256;
    return (int)(b < 4096 ? (b > 0 ? b : 1) : 4096);
}

template <typename T>
__global__ void k_gather_points(Vec3<const T> U, const long long *idx, int n, double *out) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    for (int m = 0; m < 3; m++) out[3 * t + m] = (double)U.c[m][idx[t]];
}

// element-wise precision conversions over whole allocations (same layout)
__global__ void k_widen(const float *src, double *dst, long long n) {
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n;
         x += (long long)gridDim.x * blockDim.x)
        dst[x] = (double)src[x];
}
__global__ void k_narrow(const double *src, float *dst, long long n) {
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < n;
         x += (long long)gridDim.x * blockDim.x)
        dst[x] = (float)src[x];
}

}  // namespace

void launch_predict(const LaunchCtx &L, const StepParams &P, Vec3<const double> uold,
                    Vec3<double> unew, Vec3<const double> ju, Vec3<const double> f) {
    const Grid &g = P.g;
    const Segments T = Segments::make(interior_box(g), L.blocks);
    L.pre(KK_PREDICT);
    if (P.limiter == 1)
        k_predict<1><<<T.count, TILE_THREADS, 0, L.s>>>(P, T, uold, unew, ju, f);
    else
        k_predict<0><<<T.count, TILE_THREADS, 0, L.s>>>(P, T, uold, unew, ju, f);
    L.post(KK_PREDICT);
    const long long outer = 2LL * g.gc * g.ny + 2LL * g.gc * (g.nx - 2 * g.gc);
    L.pre(KK_LAYOUT);
    k_copy_guides<<<(int)std::min<long long>((outer + 7) / 8, L.blocks), 256, 0, L.s>>>(g, uold, unew);
    L.post(KK_LAYOUT);
}

void launch_flux_rhs(const LaunchCtx &L, const StepParams &P, Vec3<const double> u,
                     Vec3<double> ju, double *b) {
    const Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_FLUX_RHS);
    k_flux_rhs<true><<<T.count + shell_blocks(P.g, T), TILE_THREADS, 0, L.s>>>(P, T, u, ju, b);
    L.post(KK_FLUX_RHS);
}

void launch_flux_only(const LaunchCtx &L, const StepParams &P, Vec3<const double> u,
                      Vec3<double> ju) {
    const Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_FLUX_RHS);
    k_flux_rhs<false><<<T.count + shell_blocks(P.g, T), TILE_THREADS, 0, L.s>>>(P, T, u, ju, nullptr);
    L.post(KK_FLUX_RHS);
}

void launch_pressure_bc(const LaunchCtx &L, const StepParams &P, double *p) {
    L.pre(KK_PBC);
    k_pressure_bc<<<plane_blocks(P.g), 256, 0, L.s>>>(P, p);
    L.post(KK_PBC);
}

void launch_project(const LaunchCtx &L, const StepParams &P, Vec3<double> u,
                    Vec3<double> ju_in, Vec3<double> ju_out, const double *p, Partials<2> part,
                    DiagState *diag) {
    const Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_PROJECT);
    k_project<<<T.count + shell_blocks(P.g, T), TILE_THREADS, 0, L.s>>>(P, T, u, ju_in, ju_out, p, part,
                                                                      diag);
    L.post(KK_PROJECT);
    if (P.reference_sums) {
        L.pre(KK_DIAG);
        k_seq_diag<<<1, 32, 0, L.s>>>(P, {{u.c[0], u.c[1], u.c[2]}},
                                      {{ju_out.c[0], ju_out.c[1], ju_out.c[2]}}, diag);
        L.post(KK_DIAG);
    }
}

template <typename T>
void launch_velocity_bc(const LaunchCtx &L, const StepParams &P, Vec3<T> u, Vec3<const T> uold) {
    L.pre(KK_UBC);
    k_velocity_bc<T><<<plane_blocks(P.g), 256, 0, L.s>>>(P, u, uold);
    L.post(KK_UBC);
}
template void launch_velocity_bc<double>(const LaunchCtx &, const StepParams &, Vec3<double>,
                                         Vec3<const double>);
template void launch_velocity_bc<float>(const LaunchCtx &, const StepParams &, Vec3<float>,
                                        Vec3<const float>);

void launch_diag(const LaunchCtx &L, const StepParams &P, Vec3<const double> u,
                 Vec3<const double> ju, Partials<2> part, DiagState *diag) {
    Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_DIAG);
    if (P.reference_sums)
        k_seq_diag<<<1, 32, 0, L.s>>>(P, u, ju, diag);
    else
        k_diag<double><<<L.blocks, TILE_THREADS, 0, L.s>>>(P, T, u, ju, part, diag);
    L.post(KK_DIAG);
}

void launch_diag(const LaunchCtx &L, const StepParams &P, Vec3<const float> u,
                 Vec3<const float> ju, Partials<2> part, DiagState *diag) {
    Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_DIAG);
    k_diag<float><<<L.blocks, TILE_THREADS, 0, L.s>>>(P, T, u, ju, part, diag);
    L.post(KK_DIAG);
}

void launch_nut_field(const LaunchCtx &L, const StepParams &P, Vec3<const double> u, double *nut) {
    Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_LAYOUT);
    k_nut_field<<<L.blocks, TILE_THREADS, 0, L.s>>>(P, T, u, nut);
    L.post(KK_LAYOUT);
}

void launch_div_field(const LaunchCtx &L, const StepParams &P, Vec3<const double> ju, double *div) {
    Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_LAYOUT);
    k_div_field<<<L.blocks, TILE_THREADS, 0, L.s>>>(P, T, ju, div);
    L.post(KK_LAYOUT);
}

void launch_q_field(const LaunchCtx &L, const StepParams &P, Vec3<const double> u, double *q) {
    Segments T = Segments::make(interior_box(P.g), L.blocks);
    L.pre(KK_LAYOUT);
    k_q_field<<<L.blocks, TILE_THREADS, 0, L.s>>>(P, T, u, q);
    L.post(KK_LAYOUT);
}

template <typename T>
void launch_tavg(const LaunchCtx &L, const Grid &g, Vec3<double> tavg, Vec3<const T> u, double w) {
    L.pre(KK_TAVG);
    k_tavg<T><<<L.blocks, 256, 0, L.s>>>(g, tavg, u, w);
    L.post(KK_TAVG);
}
template void launch_tavg<double>(const LaunchCtx &, const Grid &, Vec3<double>,
                                  Vec3<const double>, double);
template void launch_tavg<float>(const LaunchCtx &, const Grid &, Vec3<double>, Vec3<const float>,
                                 double);

void launch_to_device_layout(const LaunchCtx &L, const Grid &g, const double *ref, int ncomp,
                             double *const *dst) {
    L.pre(KK_LAYOUT);
    k_to_device<<<L.blocks, 256, 0, L.s>>>(g, ref, ncomp, dst[0], ncomp == 3 ? dst[1] : nullptr,
                                           ncomp == 3 ? dst[2] : nullptr);
    L.post(KK_LAYOUT);
}

void launch_to_ref_layout(const LaunchCtx &L, const Grid &g, double *const *src, int ncomp,
                          double *ref) {
    L.pre(KK_LAYOUT);
    k_to_ref<<<L.blocks, 256, 0, L.s>>>(g, src[0], ncomp == 3 ? src[1] : nullptr,
                                        ncomp == 3 ? src[2] : nullptr, ncomp, ref);
    L.post(KK_LAYOUT);
}

template <typename T>
void launch_gather_points(const LaunchCtx &L, Vec3<const T> u, const long long *idx, int n,
                          double *out) {
    if (n <= 0) return;
    L.pre(KK_LAYOUT);
    k_gather_points<T><<<(n + 127) / 128, 128, 0, L.s>>>(u, idx, n, out);
    L.post(KK_LAYOUT);
}
template void launch_gather_points<double>(const LaunchCtx &, Vec3<const double>,
                                           const long long *, int, double *);
template void launch_gather_points<float>(const LaunchCtx &, Vec3<const float>, const long long *,
                                          int, double *);

void launch_widen(const LaunchCtx &L, const float *src, double *dst, long long n) {
    L.pre(KK_LAYOUT);
    k_widen<<<L.blocks, 256, 0, L.s>>>(src, dst, n);
    L.post(KK_LAYOUT);
}
void launch_narrow(const LaunchCtx &L, const double *src, float *dst, long long n) {
    L.pre(KK_LAYOUT);
    k_narrow<<<L.blocks, 256, 0, L.s>>>(src, dst, n);
    L.post(KK_LAYOUT);
}

void launch_fill(const LaunchCtx &L, double *p, long long n, double v) {
    L.pre(KK_LAYOUT);
    k_fill<<<L.blocks, 256, 0, L.s>>>(p, n, v);
    L.post(KK_LAYOUT);
}

}  // namespace dalm
