// One warp's exact solve of a z-column by the partition method, and the
// lanes' row segments: shared by the launched half-sweeps (multigrid.cu) and
// the cluster V-cycle (multigrid_cluster.cu).  The method is described at
// k_mg_smooth.
#pragma once

#include "multigrid.cuh"

namespace dalm {
namespace {

// Steps 2 and 3 of the line solve for the lane's rows d[] (right-hand
// sides in, solution out in x[]): the row coefficients from the column's
// constants, the lane's Thomas sweeps and the cyclic reduction over lanes.
template <int R>
__device__ __forceinline__ void line_solve(float az, float sxy, const float *w2, const float *cf2,
                                           int nk, int lane, const float (&d)[R], float (&x)[R]) {
    const unsigned full = 0xffffffffu;
    float a[R], b[R], c[R];
#pragma unroll
    for (int s = 0; s < R; s++) {
        const int k = R * lane + s;
        if (k < nk) {
            const float lo = az * cf2[k], hi = az * cf2[k + 1];
            a[s] = -lo;
            b[s] = w2[k] * sxy + lo + hi;
            c[s] = -hi;
        } else {
            a[s] = 0.f;
            b[s] = 1.f;
            c[s] = 0.f;
        }
    }
    // 2. rows s < R - 1: x_s = D_s - A_s y_{l-1} - C_s y_l (in e, fa, g)
    float e[R], fa[R], g[R];
    float ra = a[R - 1], rb = b[R - 1], rc = c[R - 1], rd = d[R - 1];
    if (R > 1) {
#pragma unroll
        for (int s = 0; s < R - 1; s++) {
            const float den = s == 0 ? b[0] : b[s] - a[s] * g[s > 0 ? s - 1 : 0];
            const float q = __fdividef(1.f, den);
            e[s] = (s == 0 ? d[0] : d[s] - a[s] * e[s > 0 ? s - 1 : 0]) * q;
            fa[s] = (s == 0 ? a[0] : -a[s] * fa[s > 0 ? s - 1 : 0]) * q;
            g[s] = c[s] * q;
        }
#pragma unroll
        for (int s = R - 3; s >= 0; s--) {
            e[s] -= g[s] * e[s + 1];
            fa[s] -= g[s] * fa[s + 1];
            g[s] = -g[s] * g[s + 1];
        }
        // 3. the last row, with x of the next lane's first row
        float An = __shfl_down_sync(full, fa[0], 1), Cn = __shfl_down_sync(full, g[0], 1);
        float Dn = __shfl_down_sync(full, e[0], 1);
        if (lane == 31) An = Cn = Dn = 0.f;
        const float al = a[R - 1], cl = c[R - 1];
        ra = -al * fa[R - 2];
        rb = b[R - 1] - al * g[R - 2] - cl * An;
        rc = -cl * Cn;
        rd = d[R - 1] - al * e[R - 2] - cl * Dn;
    }
#pragma unroll
    for (int delta = 1; delta < 32; delta <<= 1) {
        float am = __shfl_up_sync(full, ra, delta), bm = __shfl_up_sync(full, rb, delta);
        float cm = __shfl_up_sync(full, rc, delta), dm = __shfl_up_sync(full, rd, delta);
        float ap = __shfl_down_sync(full, ra, delta), bp = __shfl_down_sync(full, rb, delta);
        float cp = __shfl_down_sync(full, rc, delta), dp = __shfl_down_sync(full, rd, delta);
        if (lane < delta) am = 0.f, bm = 1.f, cm = 0.f, dm = 0.f;  // identity rows
        if (lane + delta >= 32) ap = 0.f, bp = 1.f, cp = 0.f, dp = 0.f;
        // approximate quotients (2 ulp): the preconditioner needs no
        // correctly rounded division
        const float alpha = -__fdividef(ra, bm), gamma = -__fdividef(rc, bp);
        rb += alpha * cm + gamma * ap;
        rd += alpha * dm + gamma * dp;
        ra = alpha * am;
        rc = gamma * cp;
    }
    const float y = __fdividef(rd, rb);
    float ym = __shfl_up_sync(full, y, 1);
    if (lane == 0) ym = 0.f;
#pragma unroll
    for (int s = 0; s < R; s++)
        x[s] = s == R - 1 ? y : e[s < R - 1 ? s : 0] - fa[s < R - 1 ? s : 0] * ym -
                                    g[s < R - 1 ? s : 0] * y;
}

// The same with every matrix-only quantity read from the level's factor
// table (MgLevel::ltab, mglf_* layout; T points at this lane's entry of
// the column's class): two shuffles and two FMAs per reduction step.
template <int R>
__device__ __forceinline__ void line_solve_table(const float *T, int lane, const float (&d)[R],
                                                 float (&x)[R]) {
    const unsigned full = 0xffffffffu;
    float e[R];
    float rd = d[R - 1];
    if (R > 1) {
#pragma unroll
        for (int s = 0; s < R - 1; s++)
            e[s] = (s == 0 ? d[0] : d[s] - T[32 * mglf_a(s)] * e[s > 0 ? s - 1 : 0]) *
                   T[32 * mglf_q(s)];
#pragma unroll
        for (int s = R - 3; s >= 0; s--) e[s] -= T[32 * mglf_g(s)] * e[s + 1];
        float Dn = __shfl_down_sync(full, e[0], 1);
        if (lane == 31) Dn = 0.f;
        rd = d[R - 1] - T[32 * mglf_al(R)] * e[R - 2] - T[32 * mglf_cl(R)] * Dn;
    }
#pragma unroll
    for (int t = 0; t < 5; t++) {
        const int delta = 1 << t;
        float dm = __shfl_up_sync(full, rd, delta), dp = __shfl_down_sync(full, rd, delta);
        if (lane < delta) dm = 0.f;
        if (lane + delta >= 32) dp = 0.f;
        rd += T[32 * mglf_alpha(R, t)] * dm + T[32 * mglf_gamma(R, t)] * dp;
    }
    const float y = rd * T[32 * mglf_invrb(R)];
    float ym = __shfl_up_sync(full, y, 1);
    if (lane == 0) ym = 0.f;
#pragma unroll
    for (int s = 0; s < R; s++)
        x[s] = s == R - 1 ? y
                          : e[s < R - 1 ? s : 0] - T[32 * mglf_xa(s < R - 1 ? s : 0)] * ym -
                                T[32 * mglf_xc(s < R - 1 ? s : 0)] * y;
}

// a x + b y and the expressions of a cell built from it.  The fused products
// are spelled out: the launched kernels and the cluster kernel then give the
// same bits, whatever the compiler would fuse in either.
__device__ __forceinline__ float mg_pair(float a, float x, float b, float y) {
    return __fmaf_rn(a, x, __fmul_rn(b, y));
}
// a column's right-hand side at one cell: f + the x and y neighbours' terms
__device__ __forceinline__ float mg_line_rhs(float f, float w2, float wi, float wj, float xe, float xw, float yn,
                                             float ys, float e, float w, float n, float s) {
    return __fmaf_rn(w2, mg_pair(wj, mg_pair(xe, e, xw, w), wi, mg_pair(yn, n, ys, s)), f);
}
// the x and y part of a column's diagonal, over w2
__device__ __forceinline__ float mg_line_sxy(float wi, float wj, float xe, float xw, float yn, float ys) {
    return mg_pair(wj, xe + xw, wi, yn + ys);
}
// (K x) at one cell, az = w0 w1
__device__ __forceinline__ float mg_cell_apply(float w2, float w0, float w1, float az, float sxy, float xe, float xw,
                                               float yn, float ys, float zt, float zb, float c, float e, float w,
                                               float n, float s, float t, float b) {
    const float diag = mg_pair(w2, sxy, az, zt + zb);
    const float nb = mg_pair(w2, mg_pair(w1, mg_pair(xe, e, xw, w), w0, mg_pair(yn, n, ys, s)), az,
                             mg_pair(zt, t, zb, b));
    return __fmaf_rn(diag, c, -nb);
}

// A class's entry of the factor table in registers, for a warp that solves
// several columns of the class, or one column several times: load() and
// solve() do line_solve_table's operations.
template <int R>
struct LineFactors {
    static constexpr int H = R > 1 ? R - 1 : 1;
    float q[H], a[H], g[H], xa[H], xc[H];  // rows 0 .. R - 2
    float al, cl, alpha[5], gamma[5], last;

    __device__ __forceinline__ void load(const float *T) {
#pragma unroll
        for (int s = 0; s < R - 1; s++) {
            q[s] = T[32 * mglf_q(s)];
            a[s] = T[32 * mglf_a(s)];
            g[s] = T[32 * mglf_g(s)];
            xa[s] = T[32 * mglf_xa(s)];
            xc[s] = T[32 * mglf_xc(s)];
        }
        if (R > 1) {
            al = T[32 * mglf_al(R)];
            cl = T[32 * mglf_cl(R)];
        }
#pragma unroll
        for (int t = 0; t < 5; t++) {
            alpha[t] = T[32 * mglf_alpha(R, t)];
            gamma[t] = T[32 * mglf_gamma(R, t)];
        }
        last = T[32 * mglf_invrb(R)];
    }
    __device__ __forceinline__ void solve(int lane, const float (&d)[R], float (&x)[R]) const {
        const unsigned full = 0xffffffffu;
        float e[R];
        float rd = d[R - 1];
        if (R > 1) {
#pragma unroll
            for (int s = 0; s < R - 1; s++) e[s] = (s == 0 ? d[0] : d[s] - a[s] * e[s > 0 ? s - 1 : 0]) * q[s];
#pragma unroll
            for (int s = R - 3; s >= 0; s--) e[s] -= g[s] * e[s + 1];
            float Dn = __shfl_down_sync(full, e[0], 1);
            if (lane == 31) Dn = 0.f;
            rd = d[R - 1] - al * e[R - 2] - cl * Dn;
        }
#pragma unroll
        for (int t = 0; t < 5; t++) {
            const int delta = 1 << t;
            float dm = __shfl_up_sync(full, rd, delta), dp = __shfl_down_sync(full, rd, delta);
            if (lane < delta) dm = 0.f;
            if (lane + delta >= 32) dp = 0.f;
            rd += alpha[t] * dm + gamma[t] * dp;
        }
        const float y = rd * last;
        float ym = __shfl_up_sync(full, y, 1);
        if (lane == 0) ym = 0.f;
#pragma unroll
        for (int s = 0; s < R; s++)
            x[s] = s == R - 1 ? y : e[s < R - 1 ? s : 0] - xa[s < R - 1 ? s : 0] * ym - xc[s < R - 1 ? s : 0] * y;
    }
};

// R consecutive floats at p (VEC path: p is 4R-byte aligned)
template <int R>
__device__ __forceinline__ void load_seg(const float *p, float (&v)[R]) {
    if constexpr (R == 8) {
        const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else if constexpr (R == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    } else if constexpr (R == 2) {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        v[0] = a.x, v[1] = a.y;
    } else {
#pragma unroll
        for (int s = 0; s < R; s++) v[s] = p[s];
    }
}

template <int R>
__device__ __forceinline__ void store_seg(float *p, const float (&v)[R]) {
    if constexpr (R == 8) {
        reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else if constexpr (R == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 2) {
        *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
    } else {
#pragma unroll
        for (int s = 0; s < R; s++) p[s] = v[s];
    }
}

}  // namespace
}  // namespace dalm
