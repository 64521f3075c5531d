// The coarse part of the multigrid V-cycle (all levels from one on, or the
// whole cycle of a small grid) as one kernel on one thread-block cluster.
//
// A coarse half-sweep has a few hundred columns and no bandwidth to speak of:
// as a launch of its own it costs 2.6 to 4 us, nearly all of it launch, first
// loads and last store, and a V-cycle has fifty to seventy of them.  Here x and
// f of every level live in the cluster's distributed shared memory, the planes
// of a level dealt out over the blocks; a half-sweep reads its neighbours'
// columns from shared memory (its own or a neighbour block's) and ends at a
// cluster barrier.  Only the first level's f comes from global memory and only
// its x goes back.
//
// What bounds it: the chain of a half-sweep, neighbour loads, line solve, store
// and barrier.  A block's warps take at most one column each per half-sweep, so
// levels with more columns than the cluster has warps stay launches over the
// whole device (with four columns a warp on the first level the kernel was
// slower than the launches it replaced).  64x32x40: 50 us for the 34 phases of
// four levels, against about 2.7 us for each of the launches.
//
// Operations are mg_vcycle's in the folded form of DeviceCycle (multigrid.cu):
// the restriction leaves out the colour smoothed last, and a prolongation is
// added to the neighbours by the half-sweep after it.
#include <algorithm>
#include <type_traits>

#include "multigrid.cuh"
#include "multigrid_line.cuh"
#include "poisson.cuh"

namespace dalm {

namespace {

constexpr int CW = MG_CLUSTER_WARPS, CT = 32 * CW;

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the same shared-memory address in block `rank` of the cluster
__device__ __forceinline__ const float *in_block(const float *p, unsigned rank) {
    const float *r;
    asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return r;
}

// A level as a block sees it.
struct Lv {
    const MgClusterLevel *c;
    float *x, *f;             // this block's planes
    const float **planes;     // every plane of x, in the block that owns it
    int to_f;                 // from a column of x to the same column of f
    const float *w0, *cf0, *w1, *cf1, *w2, *cf2, *tab;
    const int *cls0, *cls1;
};

template <int C>
using Colour = std::integral_constant<int, C>;

struct Cycle {
    unsigned rank, blocks;
    float *sm;
    const MgClusterLevel *lv;  // in shared memory
    int lane, warp;

    // planes [first(r), first(r + 1)) of a level belong to block r
    __device__ __forceinline__ int first(int ni, unsigned r) const {
        return (int)((r * (unsigned)ni + blocks - 1) / blocks);
    }
    __device__ __forceinline__ Lv level(int l) const {
        const MgClusterLevel &c = lv[l];
        const int *cls = reinterpret_cast<const int *>(sm) + c.cls;
        return Lv{&c, sm + c.x, sm + c.f, reinterpret_cast<const float **>(sm + c.planes), c.f - c.x,
                  sm + c.w0, sm + c.cf0, sm + c.w1, sm + c.cf1, sm + c.w2, sm + c.cf2, sm + c.tab,
                  cls, cls + c.n[0]};
    }
    // the addresses of every level's planes
    __device__ __forceinline__ void map_planes(int levels) const {
        for (int l = 0; l < levels; l++) {
            const MgClusterLevel &c = lv[l];
            const float **planes = reinterpret_cast<const float **>(sm + c.planes);
            for (int i = threadIdx.x; i < c.n[0]; i += CT) {
                const unsigned o = (unsigned)i * blocks / (unsigned)c.n[0];
                const float *p = sm + c.x + (i - first(c.n[0], o)) * c.n[1] * c.S;
                planes[i] = o == rank ? p : in_block(p, o);
            }
        }
    }

    // The zebra half-sweeps of one visit to a level, every column of a colour
    // solved exactly: colour 0 then 1 nu times before the coarse correction
    // (from zero), 1 then 0 after it (the first of them adds the coarse level's
    // correction to the neighbours it reads).  A warp has at most one column
    // of either colour; what the visit needs of a column beside its
    // neighbours - right-hand side, coefficients, the factors of its line -
    // stays in registers.
    template <int R>
    __device__ __forceinline__ void visit(int l, int nu, bool post) const {
        const Lv L = level(l);
        const MgClusterLevel &c = *L.c;
        const int i0 = first(c.n[0], rank), np = first(c.n[0], rank + 1) - i0;
        const int n0 = c.n[0], n1 = c.n[1], S = c.S, njh = (n1 + 1) / 2;
        const int ip = warp / njh, h = warp - ip * njh, i = i0 + ip;
        const bool in = ip < np;  // uniform in the warp, as everything but the lane
        LineFactors<R> F[2];
        float f[2][R], w2[R], wj[2], yn[2], ys[2];
        int at[2];
        bool has[2];
        const float wi = in ? L.w0[i] : 0.f, xe = in ? L.cf0[i + 1] : 0.f, xw = in ? L.cf0[i] : 0.f;
        load_seg<R>(L.w2 + R * lane, w2);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int j = 2 * h + ((i + q) & 1);
            has[q] = in && j < n1;
            at[q] = (ip * n1 + j) * S + R * lane;
            if (!has[q]) continue;
            wj[q] = L.w1[j], yn[q] = L.cf1[j + 1], ys[q] = L.cf1[j];
            load_seg<R>(L.f + at[q], f[q]);
            if (c.tab >= 0)
                F[q].load(L.tab + (L.cls0[i] * c.lky + L.cls1[j]) * mglf_count(R) * 32 + lane);
            else
                F[q].factor(wi * wj[q], wj[q] * (xe + xw) + wi * (yn[q] + ys[q]), L.w2, L.cf2, c.n[2], lane);
        }
        const float *east = in && i + 1 < n0 ? L.planes[i + 1] : nullptr;
        const float *west = in && i > 0 ? L.planes[i - 1] : nullptr;
        auto half = [&](auto colour, bool zero, bool pending) {
            constexpr int q = decltype(colour)::value;  // constant: the arrays stay in registers
            if (has[q]) {
                const int j = 2 * h + ((i + q) & 1);
                float d[R], x[R];
#pragma unroll
                for (int t = 0; t < R; t++) d[t] = f[q][t];
                if (!zero) {
                    float e[R], w[R], n[R], s[R];
                    auto nb = [&](const float *p, int ii, int jj, float (&v)[R]) {
                        if (!p) {
#pragma unroll
                            for (int t = 0; t < R; t++) v[t] = 0.f;
                            return;
                        }
                        load_seg<R>(p, v);
                        if (pending) {
                            const Lv C = level(l + 1);
                            const float *xc = C.planes[ii / C.c->fac[0]] + jj / C.c->fac[1] * C.c->S;
                            const int shift = C.c->fac[2] == 2 ? 1 : 0;
#pragma unroll
                            for (int t = 0; t < R; t++)
                                if (R * lane + t < c.n[2]) v[t] += xc[(R * lane + t) >> shift];
                        }
                    };
                    nb(east ? east + j * S + R * lane : nullptr, i + 1, j, e);
                    nb(west ? west + j * S + R * lane : nullptr, i - 1, j, w);
                    nb(j + 1 < n1 ? L.x + at[q] + S : nullptr, i, j + 1, n);
                    nb(j > 0 ? L.x + at[q] - S : nullptr, i, j - 1, s);
#pragma unroll
                    for (int t = 0; t < R; t++)
                        d[t] = d[t] + w2[t] * (wj[q] * (xe * e[t] + xw * w[t]) + wi * (yn[q] * n[t] + ys[q] * s[t]));
                }
                F[q].solve(lane, d, x);
                store_seg<R>(L.x + at[q], x);
            }
            cluster_sync();
        };
        for (int s = 0; s < nu; s++) {
            if (post) {
                half(Colour<1>{}, false, s == 0);
                half(Colour<0>{}, false, false);
            } else {
                half(Colour<0>{}, s == 0, false);
                half(Colour<1>{}, false, false);
            }
        }
    }
    template <int RMAX>
    __device__ __forceinline__ void smooth(int l, int nu, bool post) const {
        const int R = lv[l].S / 32;
        if (R == 1) visit<1>(l, nu, post);
        if (RMAX >= 2 && R == 2) visit<2>(l, nu, post);
        if (RMAX >= 3 && R == 3) visit<3>(l, nu, post);
        if (RMAX >= 4 && R == 4) visit<4>(l, nu, post);
    }

    // f of level l + 1: the sums of the children's residuals f - K x, the
    // children of colour `skip` (whose residual is zero) left out
    __device__ __forceinline__ void restrict_to(int l, int skip) const {
        const Lv F = level(l), C = level(l + 1);
        const MgClusterLevel &f = *F.c, &c = *C.c;
        const int I0 = first(c.n[0], rank), np = first(c.n[0], rank + 1) - I0, f2 = c.fac[2];
        for (int q = warp; q < np * c.n[1]; q += CW) {
            const int ip = q / c.n[1], I = I0 + ip, J = q - ip * c.n[1];
            float *out = C.f + (ip * c.n[1] + J) * c.S;
            for (int K = lane; K < c.n[2]; K += 32) {
                float sum = 0.f;
                for (int a = 0; a < c.fac[0]; a++)
                    for (int b = 0; b < c.fac[1]; b++) {
                        const int i = I * c.fac[0] + a, j = J * c.fac[1] + b;
                        if (((i + j) & 1) == skip) continue;
                        const float *x = F.planes[i] + j * f.S, *rhs = x + F.to_f;
                        const float *xe = i + 1 < f.n[0] ? F.planes[i + 1] + j * f.S : nullptr;
                        const float *xw = i > 0 ? F.planes[i - 1] + j * f.S : nullptr;
                        const float *xn = j + 1 < f.n[1] ? x + f.S : nullptr, *xs = j > 0 ? x - f.S : nullptr;
                        const float w0 = F.w0[i], w1 = F.w1[j], az = w0 * w1;
                        const float ce = F.cf0[i + 1], cw = F.cf0[i], cn = F.cf1[j + 1], cs = F.cf1[j];
                        const float sxy = w1 * (ce + cw) + w0 * (cn + cs);
                        for (int t = 0; t < f2; t++) {
                            const int k = K * f2 + t;
                            const float w2 = F.w2[k], zt = F.cf2[k + 1], zb = F.cf2[k];
                            const float diag = w2 * sxy + az * (zt + zb);
                            const float nb =
                                w2 * (w1 * (ce * (xe ? xe[k] : 0.f) + cw * (xw ? xw[k] : 0.f)) +
                                      w0 * (cn * (xn ? xn[k] : 0.f) + cs * (xs ? xs[k] : 0.f))) +
                                az * (zt * (k + 1 < f.n[2] ? x[k + 1] : 0.f) + zb * (k > 0 ? x[k - 1] : 0.f));
                            sum += rhs[k] - (diag * x[k] - nb);
                        }
                    }
                out[K] = sum;
            }
        }
        cluster_sync();
    }

    // x = K^-1 f on the coarsest level: a warp per row of the dense inverse
    __device__ __forceinline__ void coarse(int l, const float *kinv, int n) const {
        const Lv L = level(l);
        const MgClusterLevel &c = *L.c;
        const int i0 = first(c.n[0], rank), np = first(c.n[0], rank + 1) - i0;
        float *all = sm + c.gather;  // the level's f in cell order
        for (int r = threadIdx.x; r < n; r += CT) {
            const int k = r % c.n[2], row = r / c.n[2], j = row % c.n[1], i = row / c.n[1];
            all[r] = L.planes[i][j * c.S + L.to_f + k];
        }
        __syncthreads();
        const int plane = c.n[1] * c.n[2];
        for (int q = warp; q < np * plane; q += CW) {
            const float *row = kinv + (size_t)(i0 * plane + q) * n;
            float s = 0.f;
            for (int r = lane; r < n; r += 32) s += row[r] * all[r];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0) L.x[q / c.n[2] * c.S + q % c.n[2]] = s;
        }
        cluster_sync();
    }
};

// RMAX: rows per lane of the first level's columns (32 RMAX cells at most)
template <int RMAX>
__global__ void __launch_bounds__(CT, 1)
k_mg_cluster(MgCluster M, const float *f, float *x, const KrylovState *st) {
    pdl_wait();
    if (st->done) return;  // the same in every block
    extern __shared__ __align__(16) float cluster_smem[];
    float *sm = cluster_smem;
    // the level table, its coefficients and factor tables; x and f zeroed (the
    // lanes' rows past a column's end stay zero)
    for (int n = threadIdx.x; n < M.words; n += CT) sm[n] = M.image[n];
    for (int n = M.words + threadIdx.x; n < M.total; n += CT) sm[n] = 0.f;
    __syncthreads();
    Cycle y;
    y.rank = cluster_rank();
    y.blocks = M.blocks;
    y.sm = sm;
    y.lv = reinterpret_cast<const MgClusterLevel *>(sm);
    y.lane = threadIdx.x & 31;
    y.warp = threadIdx.x >> 5;
    y.map_planes(M.levels);
    const MgClusterLevel &c = y.lv[0];
    const int i0 = y.first(c.n[0], y.rank), np = y.first(c.n[0], y.rank + 1) - i0;
    for (int q = y.warp; q < np * c.n[1]; q += CW) {
        const int ip = q / c.n[1], j = q - ip * c.n[1];
        const float *src = f + M.top.at(i0 + ip, j, 0);
        for (int k = y.lane; k < c.n[2]; k += 32) sm[c.f + q * c.S + k] = src[k];
    }
    cluster_sync();
    const int last = M.levels - 1;
    for (int l = 0; l < last; l++) {
        y.smooth<RMAX>(l, mg_nu(M.first + l), false);
        y.restrict_to(l, 1);
    }
    y.coarse(last, M.kinv, M.ncoarse);
    for (int l = last - 1; l >= 0; l--) y.smooth<RMAX>(l, mg_nu(M.first + l), true);
    for (int q = y.warp; q < np * c.n[1]; q += CW) {
        const int ip = q / c.n[1], j = q - ip * c.n[1];
        float *dst = x + M.top.at(i0 + ip, j, 0);
        for (int k = y.lane; k < c.n[2]; k += 32) dst[k] = sm[c.x + q * c.S + k];
    }
    // (every block's shared memory was last read before the last barrier)
}

cudaLaunchConfig_t config(const MgCluster &M, cudaLaunchAttribute *attr, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)M.blocks);
    cfg.blockDim = dim3(CT);
    cfg.dynamicSmemBytes = (size_t)M.total * 4;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)M.blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

// the kernel for this cycle, with its shared memory and cluster size allowed
auto kernel_of(const MgCluster &M) {
    const int R = (M.top.n[2] + 31) / 32;
    auto k = R == 1 ? k_mg_cluster<1> : R == 2 ? k_mg_cluster<2> : R == 3 ? k_mg_cluster<3> : k_mg_cluster<4>;
    DALM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, M.total * 4));
    DALM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return k;
}

}  // namespace

bool mg_cluster_fits(const MgCluster &M) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = config(M, attr, 0);
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel_of(M), &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n >= 1;
}

void launch_mg_cluster(const LaunchCtx &L, const MgCluster &M, const float *f, float *x, const KrylovState *st) {
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = config(M, attr, L.s);
    L.pre(KK_MG_COARSE);
    DALM_CUDA(cudaLaunchKernelEx(&cfg, kernel_of(M), M, f, x, st));
    L.post(KK_MG_COARSE);
}

}  // namespace dalm
