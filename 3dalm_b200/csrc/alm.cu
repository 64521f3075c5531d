// Actuator-line kernels (FP64), compiled with --fmad=false so the blade-point
// arithmetic keeps the reference's rounding; only the libm calls (sin, cos,
// atan, exp) may differ from the host's by an ulp.
#include <algorithm>

#include "alm_point.cuh"

namespace dalm {

namespace {

// dynamic shared memory of either kernel at most
constexpr size_t ALM_SMEM = 200 * 1024;

__device__ __forceinline__ double sq(double v) { return v * v; }

// update_ap_position + calc_ap_force (src/alm.h:233-370) and the turbine's
// torque and thrust in blade-point order (src/alm.h:384-398): one block per
// turbine, a thread per blade point; the arithmetic is almpt's
// (alm_point.cuh), shared with the host path of the reference-order mode.
// T: storage type of the velocity field (double, or float for the mixed
// form's FP32 stencil fields); the point model is FP64 either way.
//
// A point's chain is some 25 dependent reads of the mesh and polar angles by
// bisection; staged: they are first copied to shared memory, where a read
// takes a tenth of the time (`staged` false: they do not fit).  40x20x20
// to 512x256x128: 15-23 us with the sums, against 17-25 and 7-10 in two launches.
template <typename T>
__global__ void __launch_bounds__(512)
k_alm_points(StepParams P, AlmDev A, double t, Vec3<const T> U, bool staged) {
    extern __shared__ double alm_smem[];
    const double *x = P.m.x, *y = P.m.y, *z = P.m.z, *atk = A.atk;
    double *sum = alm_smem;  // [2][ap_per_wt]
    if (staged) {
        double *d = alm_smem + 2 * A.ap_per_wt;
        auto stage = [&](const double *&src, int n) {
            for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = src[i];
            src = d;
            d += n;
        };
        stage(x, P.g.nx);
        stage(y, P.g.ny);
        stage(z, P.g.nz);
        stage(atk, A.atk_count);
        __syncthreads();
    }
    const int w = blockIdx.x;
    const TurbineDev &wt = A.wt[w];
    for (int n = threadIdx.x; n < A.ap_per_wt; n += blockDim.x) {
        const int a = w * A.ap_per_wt + n, bid = n / A.ap_per_blade;
        almpt::Pose q;
        almpt::point_pose(wt, A.r[a], bid, A.blades, t, q);
        long long id[8];
        double frac[3], f[3] = {0, 0, 0}, torque = 0, thrust = 0;
        if (almpt::point_cell(P.g, x, y, z, q.xyz, id, frac)) {
            double Uap[3];
            for (int m = 0; m < 3; m++) {
                const T *v = U.c[m];
                double c8[8];
                for (int n8 = 0; n8 < 8; n8++) c8[n8] = (double)v[id[n8]];
                Uap[m] = almpt::trilinear(c8, frac);
            }
            almpt::point_force(wt, q, Uap, A.twist[a], A.chord[a], A.dr[a], atk, A.atk_count,
                               A.cd + (long long)a * A.atk_count, A.cl + (long long)a * A.atk_count,
                               f, torque, thrust);
        }
        for (int m = 0; m < 3; m++) {
            A.pt_xyz[a * 3 + m] = q.xyz[m];
            A.pt_f[a * 3 + m] = f[m];
        }
        A.pt_torque[a] = torque;
        A.pt_thrust[a] = thrust;
        if (staged) {
            sum[n] = torque;
            sum[A.ap_per_wt + n] = thrust;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double *tq = staged ? sum : A.pt_torque + w * A.ap_per_wt;
        const double *th = staged ? sum + A.ap_per_wt : A.pt_thrust + w * A.ap_per_wt;
        double torque = 0, thrust = 0;
        for (int n = 0; n < A.ap_per_wt; n++) {
            torque += tq[n];
            thrust += th[n];
        }
        A.wt_torque[w] = torque;
        A.wt_thrust[w] = thrust;
    }
}

// distribute_ap_force (src/alm.h:416-448), support-confined: a block owns
// 32 k x 8 j cells of PP planes; it gathers, in blade-point order, the points
// whose truncated support reaches them, then every cell sums those points in
// that order (the reference's order with the negligible far terms left out).
//
// The Gaussian is a product of one factor per axis, so a point's factors are
// evaluated once per plane, row and column of the block (for PG points at a
// time, in shared memory) instead of once per cell: an FP64 exponential is some
// forty dependent instructions.  Three rotors of 512 x 256 x 128: 45 -> 27 us,
// one of 131 x 75 x 53: 39 -> 20 us.  Two planes a block: with eight there are
// too few blocks (61 us on the latter).
constexpr int PP = 2, PG = 32;
template <typename FT>
__global__ void __launch_bounds__(TILE_THREADS)
k_alm_project(StepParams P, AlmDev A, Box box, int ntk, int ntj, Vec3<FT> F) {
    extern __shared__ int list[];
    __shared__ int warp_count[TILE_THREADS / 32];
    __shared__ double e[PG][PP + TJ + TK], d2[PG][PP + TJ + TK], pf[PG][3];
    const Grid &g = P.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tk = blockIdx.x % ntk, tj = (blockIdx.x / ntk) % ntj, ti = blockIdx.x / (ntk * ntj);
    const int k0 = box.lo[2] + tk * TK, j0 = box.lo[1] + tj * TJ, i0 = box.lo[0] + ti * PP;
    const int k1 = min(k0 + TK, box.hi[2]), j1 = min(j0 + TJ, box.hi[1]), i1 = min(i0 + PP, box.hi[0]);
    // the block's bounding box (cell-centre arrays are increasing)
    const double lo[3] = {P.m.x[i0], P.m.y[j0], P.m.z[k0]};
    const double hi[3] = {P.m.x[i1 - 1], P.m.y[j1 - 1], P.m.z[k1 - 1]};
    int total = 0;
    for (int base = 0; base < A.ap_count; base += TILE_THREADS) {
        const int a = base + threadIdx.x;
        bool near = false;
        if (a < A.ap_count) {
            double r2 = 0;
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const double p = A.pt_xyz[a * 3 + m];
                r2 += sq(p < lo[m] ? lo[m] - p : (p > hi[m] ? p - hi[m] : 0.0));
            }
            near = r2 <= A.cutoff2;
        }
        const unsigned mask = __ballot_sync(0xffffffffu, near);
        if (lane == 0) warp_count[warp] = __popc(mask);
        __syncthreads();
        int before = total;
        for (int w = 0; w < TILE_THREADS / 32; w++) {
            if (w < warp) before += warp_count[w];
            total += warp_count[w];
        }
        if (near) list[before + __popc(mask & ((1u << lane) - 1u))] = a;
        __syncthreads();
    }
    const int j = j0 + warp, k = k0 + lane;
    double f[PP][3];
#pragma unroll
    for (int u = 0; u < PP; u++) f[u][0] = f[u][1] = f[u][2] = 0;
    for (int base = 0; base < total; base += PG) {
        const int np = min(PG, total - base);
        for (int q = threadIdx.x; q < np * (PP + TJ + TK); q += TILE_THREADS) {
            const int p = q / (PP + TJ + TK), s = q - p * (PP + TJ + TK), a = list[base + p];
            const int axis = s < PP ? 0 : s < PP + TJ ? 1 : 2;
            const int n = axis == 0 ? min(i0 + s, i1 - 1)
                                    : axis == 1 ? min(j0 + s - PP, j1 - 1) : min(k0 + s - PP - TJ, k1 - 1);
            const double c = axis == 0 ? P.m.x[n] : axis == 1 ? P.m.y[n] : P.m.z[n];
            const double r2 = sq(c - A.pt_xyz[a * 3 + axis]);
            d2[p][s] = r2;
            e[p][s] = exp(-r2 / A.pw2);
        }
        for (int q = threadIdx.x; q < 3 * np; q += TILE_THREADS) pf[q / 3][q % 3] = A.pt_f[list[base + q / 3] * 3 + q % 3];
        __syncthreads();
        for (int p = 0; p < np; p++) {
            const double dy = d2[p][PP + warp], dz = d2[p][PP + TJ + lane];
            const double eyz = A.e_coef * (e[p][PP + warp] * e[p][PP + TJ + lane]);
            const double f0 = pf[p][0], f1 = pf[p][1], f2 = pf[p][2];
#pragma unroll
            for (int u = 0; u < PP; u++) {
                if (d2[p][u] + dy + dz <= A.cutoff2) {
                    const double wght = e[p][u] * eyz;
                    f[u][0] += wght * f0;
                    f[u][1] += wght * f1;
                    f[u][2] += wght * f2;
                }
            }
        }
        __syncthreads();
    }
    if (j >= j1 || k >= k1) return;
#pragma unroll
    for (int u = 0; u < PP; u++)
        if (i0 + u < i1) {
            const long long c = g.at(i0 + u, j, k);
            F.c[0][c] = (FT)f[u][0];
            F.c[1][c] = (FT)f[u][1];
            F.c[2][c] = (FT)f[u][2];
        }
}

}  // namespace

template <typename T>
void prepare_alm() {
    allow_shared(k_alm_points<T>, ALM_SMEM);
    allow_shared(k_alm_project<T>, ALM_SMEM);
}
template void prepare_alm<double>();
template void prepare_alm<float>();

template <typename T>
void launch_alm_points(const LaunchCtx &L, const StepParams &P, const AlmDev &A, double t,
                       Vec3<const T> u) {
    if (A.ap_count <= 0) return;
    // the sums' terms, the mesh and the polar angles in shared memory
    const size_t bytes = sizeof(double) * (2 * (size_t)A.ap_per_wt + P.g.nx + P.g.ny + P.g.nz + A.atk_count);
    const bool staged = bytes <= ALM_SMEM;
    const size_t smem = staged ? bytes : 0;
    const int threads = std::min(512, std::max(128, (A.ap_per_wt + 31) / 32 * 32));
    L.pre(KK_ALM_POINTS);
    k_alm_points<T><<<A.wt_count, threads, smem, L.s>>>(P, A, t, u, staged);
    L.post(KK_ALM_POINTS);
}
template void launch_alm_points<double>(const LaunchCtx &, const StepParams &, const AlmDev &,
                                        double, Vec3<const double>);
template void launch_alm_points<float>(const LaunchCtx &, const StepParams &, const AlmDev &,
                                       double, Vec3<const float>);

template <typename FT>
void launch_alm_project(const LaunchCtx &L, const StepParams &P, const AlmDev &A,
                        const Box &box, Vec3<FT> f) {
    if (A.ap_count <= 0 || box.empty()) return;
    const int ntk = (box.hi[2] - box.lo[2] + TK - 1) / TK, ntj = (box.hi[1] - box.lo[1] + TJ - 1) / TJ;
    const int nti = (box.hi[0] - box.lo[0] + PP - 1) / PP;
    // the list of points, beside 22 KB of static tables
    const size_t smem = sizeof(int) * (size_t)A.ap_count;
    L.pre(KK_ALM_PROJECT);
    k_alm_project<FT><<<ntk * ntj * nti, TILE_THREADS, smem, L.s>>>(P, A, box, ntk, ntj, f);
    L.post(KK_ALM_PROJECT);
}
template void launch_alm_project<double>(const LaunchCtx &, const StepParams &, const AlmDev &,
                                         const Box &, Vec3<double>);
template void launch_alm_project<float>(const LaunchCtx &, const StepParams &, const AlmDev &,
                                        const Box &, Vec3<float>);

}  // namespace dalm
