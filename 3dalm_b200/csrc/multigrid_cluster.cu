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
// and barrier, at about ten cycles an instruction.  A block's warps take at
// most one column each per half-sweep, so levels with more columns than the
// cluster has warps stay launches over the whole device (with four columns a
// warp on the first level the kernel was slower than the launches it replaced).
// So what a visit can do once is done once, before its half-sweeps: the finer
// levels' line factors come from their tables, addresses and coefficients stay
// in registers, and what lies past the grid is a column of zeros instead of a
// branch.  64x32x40 0.94 ms a step, 160x96x72 2.80 (0.98 and 2.89 with generic
// addresses and a spilled state).  Factors formed once per visit or once per
// handle on the other levels too took 0.90 and 2.70, but other roundings than
// the launched kernels' elimination, and where the stop leaves the pressure
// loose (128 cells along z at a small time step) those show as 1e-4 of it.
// Small levels whole in one block, with block barriers for cluster barriers,
// gained nothing.
//
// Operations are mg_vcycle's in the folded form of DeviceCycle (multigrid.cu),
// and give the launched kernels' bits: the restriction leaves out the colour
// smoothed last, and a prolongation is added to the neighbours by the
// half-sweep after it.
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
__device__ __forceinline__ void copy_async(float *shared, const float *global) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(shared)),
                 "l"(global)
                 : "memory");
}
// the address of a word of shared memory in block `rank` of the cluster
__device__ __forceinline__ unsigned in_block(const float *p, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
// loads and a store at such an address.  Volatile: they keep their place
// between the cluster barriers.
__device__ __forceinline__ float load_word(unsigned a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void store_word(unsigned a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
template <int R>
__device__ __forceinline__ void load_rows(unsigned a, float (&v)[R]) {
    if constexpr (R == 4)
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                     : "r"(a));
    else if constexpr (R == 2)
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a));
    else
#pragma unroll
        for (int t = 0; t < R; t++) v[t] = load_word(a + 4 * t);
}

// A level as a block sees it.
struct Lv {
    const MgClusterLevel *c;
    float *x, *f;             // this block's planes
    const unsigned *planes;   // every plane of x, in the block that owns it
    int to_f;                 // bytes from a column of x to the same column of f
    const float *w0, *cf0, *w1, *cf1, *w2, *cf2;
    const int *cls0, *cls1;
};

template <int C>
using Colour = std::integral_constant<int, C>;

struct Cycle {
    unsigned rank, blocks;
    float *sm;
    const MgClusterLevel *lv;  // in shared memory
    const float *tables;       // line factors, in global memory
    float *zeros;              // a column of zeros: what lies past the grid
    unsigned zeros_at;
    int lane, warp;

    // planes [first(r), first(r + 1)) of a level belong to block r
    __device__ __forceinline__ int first(const MgClusterLevel &c, unsigned r) const {
        return (int)((r * (unsigned)c.n[0] + blocks - 1) / blocks);
    }
    __device__ __forceinline__ Lv level(int l) const {
        const MgClusterLevel &c = lv[l];
        const int *cls = reinterpret_cast<const int *>(sm) + c.cls;
        return Lv{&c, sm + c.x, sm + c.f, reinterpret_cast<const unsigned *>(sm + c.planes), 4 * (c.f - c.x),
                  sm + c.w0, sm + c.cf0, sm + c.w1, sm + c.cf1, sm + c.w2, sm + c.cf2,
                  cls, cls + c.n[0]};
    }
    // the addresses of every level's planes
    __device__ __forceinline__ void map_planes(int levels) const {
        for (int l = 0; l < levels; l++) {
            const MgClusterLevel &c = lv[l];
            unsigned *planes = reinterpret_cast<unsigned *>(sm + c.planes);
            for (int i = threadIdx.x; i < c.n[0]; i += CT) {
                const unsigned o = (unsigned)i * blocks / (unsigned)c.n[0];
                planes[i] = in_block(sm + c.x + (i - first(c, o)) * c.n[1] * c.S, o);
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
        const int i0 = first(c, rank), np = first(c, rank + 1) - i0;
        const int n0 = c.n[0], n1 = c.n[1], S = c.S, njh = (n1 + 1) / 2;
        const int ip = warp / njh, h = warp - ip * njh, i = i0 + ip;
        if (ip >= np) {  // no column: only the barriers (uniform in the warp, as all but the lane)
            for (int s = 0; s < 2 * nu; s++) cluster_sync();
            return;
        }
        LineFactors<R> F[2] = {};
        float f[2][R], w2[R], wj[2], yn[2], ys[2];
        unsigned e[2], w[2];               // the neighbours' rows of this lane
        const float *nn[2], *ss[2];
        float *at[2];
        bool has[2];
        load_seg<R>(L.w2 + R * lane, w2);
        const float wi = L.w0[i], xe = L.cf0[i + 1], xw = L.cf0[i];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int jq = 2 * h + ((i + q) & 1), j = min(jq, n1 - 1), col = j * S + R * lane;
            has[q] = jq < n1;  // (an odd count's last: solved with the others, not stored)
            wj[q] = L.w1[j], yn[q] = L.cf1[j + 1], ys[q] = L.cf1[j];
            at[q] = L.x + ip * n1 * S + col;
            e[q] = i + 1 < n0 ? L.planes[i + 1] + 4 * col : zeros_at;
            w[q] = i > 0 ? L.planes[i - 1] + 4 * col : zeros_at;
            nn[q] = j + 1 < n1 ? at[q] + S : zeros;
            ss[q] = j > 0 ? at[q] - S : zeros;
            load_seg<R>(at[q] + (c.f - c.x), f[q]);
            if (c.tab >= 0)
                F[q].load(tables + c.tab + (L.cls0[i] * c.lky + L.cls1[j]) * mglf_count(R) * 32 + lane);
        }
        auto half = [&](auto colour, bool zero, bool pending) {
            constexpr int q = decltype(colour)::value;  // constant: the arrays stay in registers
            float d[R], x[R];
#pragma unroll
            for (int t = 0; t < R; t++) d[t] = f[q][t];
            if (!zero) {
                float ve[R], vw[R], vn[R], vs[R];
                load_rows<R>(e[q], ve);
                load_rows<R>(w[q], vw);
                load_seg<R>(nn[q], vn);
                load_seg<R>(ss[q], vs);
                if (pending) {
                    // (a level merges one or two cells along an axis)
                    const Lv C = level(l + 1);
                    const int j = min(2 * h + ((i + q) & 1), n1 - 1), s0 = C.c->fac[0] - 1, s1 = C.c->fac[1] - 1;
                    auto add = [&](bool there, int ii, int jj, float (&v)[R]) {
                        if (!there) return;
                        const unsigned xc = C.planes[ii >> s0] + 4 * (jj >> s1) * C.c->S;
#pragma unroll
                        for (int t = 0; t < R; t++) v[t] += load_word(xc + 4 * ((R * lane + t) >> (C.c->fac[2] - 1)));
                    };
                    add(i + 1 < n0, i + 1, j, ve);
                    add(i > 0, i - 1, j, vw);
                    add(j + 1 < n1, i, j + 1, vn);
                    add(j > 0, i, j - 1, vs);
                }
#pragma unroll
                for (int t = 0; t < R; t++)
                    d[t] = mg_line_rhs(d[t], w2[t], wi, wj[q], xe, xw, yn[q], ys[q], ve[t], vw[t], vn[t], vs[t]);
            }
            if (c.tab >= 0) F[q].solve(lane, d, x);
            else line_solve<R>(wi * wj[q], mg_line_sxy(wi, wj[q], xe, xw, yn[q], ys[q]), L.w2, L.cf2, c.n[2], lane, d, x);
            if (has[q]) store_seg<R>(at[q], x);
            cluster_sync();
        };
#pragma unroll 1
        for (int s = 0; s < 2 * nu; s++) {
            const bool begin = s == 0;
            if ((s & 1) == (post ? 1 : 0)) half(Colour<0>{}, begin, false);  // (begin: not after a correction)
            else half(Colour<1>{}, false, begin);
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

    // A cell column's operands for its residual.
    struct Child {
        unsigned x, e, w, n, s;
        float ce, cw, cn, cs, w0, w1, az, sxy;
        __device__ __forceinline__ Child(const Lv &F, int i, int j, unsigned zeros_at) {
            const MgClusterLevel &f = *F.c;
            const unsigned row = 4u * (unsigned)f.S, col = j * row;
            x = F.planes[i] + col;
            e = i + 1 < f.n[0] ? F.planes[i + 1] + col : zeros_at;
            w = i > 0 ? F.planes[i - 1] + col : zeros_at;
            n = j + 1 < f.n[1] ? x + row : zeros_at;
            s = j > 0 ? x - row : zeros_at;
            w0 = F.w0[i], w1 = F.w1[j], az = w0 * w1;
            ce = F.cf0[i + 1], cw = F.cf0[i], cn = F.cf1[j + 1], cs = F.cf1[j];
            sxy = mg_line_sxy(w0, w1, ce, cw, cn, cs);
        }
        // f - K x at k
        __device__ __forceinline__ float residual(const Lv &F, int k) const {
            const unsigned o = 4u * (unsigned)k;
            const float xk = load_word(x + o), rhs = load_word(x + F.to_f + o);
            const float xe = load_word(e + o), xw = load_word(w + o), xn = load_word(n + o), xs = load_word(s + o);
            const float xt = k + 1 < F.c->n[2] ? load_word(x + o + 4) : 0.f, xb = k > 0 ? load_word(x + o - 4) : 0.f;
            const float w2 = F.w2[k], zt = F.cf2[k + 1], zb = F.cf2[k];
            return rhs - mg_cell_apply(w2, w0, w1, az, sxy, ce, cw, cn, cs, zt, zb, xk, xe, xw, xn, xs, xt, xb);
        }
    };

    // f of level l + 1: the sums of the children's residuals f - K x, the
    // children of colour 1 (smoothed last, no residual) left out: of two by
    // two columns two are kept, of two one, of one one or none.
    __device__ __forceinline__ void restrict_to(int l) const {
        const Lv F = level(l), C = level(l + 1);
        const MgClusterLevel &c = *C.c;
        const int I0 = first(c, rank), np = first(c, rank + 1) - I0, fx = c.fac[0], fy = c.fac[1];
        for (int q = warp; q < np * c.n[1]; q += CW) {
            const int ip = q / c.n[1], I = I0 + ip, J = q - ip * c.n[1], i = I * fx, j = J * fy;
            float *out = C.f + q * c.S;
            // the kept column of the first row of children, then of the second
            const int odd = (i + j) & 1;
            const bool one = !odd || fy == 2, two = fx == 2 && (odd || fy == 2);
            const Child A(F, one ? i : i + fx - 1, one ? j + odd : j, zeros_at);
            const Child B(F, i + fx - 1, odd || fy == 1 ? j : j + 1, zeros_at);
#pragma unroll 1
            for (int K = lane; K < c.n[2]; K += 32) {
                const int k = K * c.fac[2];
                const float a0 = A.residual(F, k), b0 = B.residual(F, k);
                float a1 = 0.f, b1 = 0.f;
                if (c.fac[2] == 2) a1 = A.residual(F, k + 1), b1 = B.residual(F, k + 1);
                out[K] = (one ? a0 + a1 : 0.f) + (two ? b0 : 0.f) + (two ? b1 : 0.f);
            }
        }
        cluster_sync();
    }

    // x = K^-1 f on the coarsest level: a warp per row of the dense inverse,
    // the rows dealt out over all blocks
    __device__ __forceinline__ void coarse(int l, const float *kinv, int n) const {
        const Lv L = level(l);
        const MgClusterLevel &c = *L.c;
        float *all = sm + c.gather;  // the level's f in cell order
        const int nk = c.n[2];
        for (int col = warp; col < c.n[0] * c.n[1]; col += CW) {
            const int i = col / c.n[1], j = col - i * c.n[1];
            const unsigned f = L.planes[i] + 4 * j * c.S + L.to_f;
            for (int k = lane; k < nk; k += 32) all[col * nk + k] = load_word(f + 4 * k);
        }
        __syncthreads();
        for (int q = (int)(rank + blocks * warp); q < n; q += (int)blocks * CW) {
            const float *row = kinv + (size_t)q * n;
            float s = 0.f;
            for (int r0 = lane; r0 < n; r0 += MG_COARSE_TARGET) {
                float v[MG_COARSE_TARGET / 32];
#pragma unroll
                for (int t = 0; t < MG_COARSE_TARGET / 32; t++) v[t] = r0 + 32 * t < n ? row[r0 + 32 * t] : 0.f;
#pragma unroll
                for (int t = 0; t < MG_COARSE_TARGET / 32; t++)
                    if (r0 + 32 * t < n) s += v[t] * all[r0 + 32 * t];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            const int k = q % nk, col = q / nk, i = col / c.n[1], j = col - i * c.n[1];
            if (lane == 0) store_word(L.planes[i] + 4 * (j * c.S + k), s);
        }
        cluster_sync();
    }
};

// RMAX: rows per lane of the first level's columns (32 RMAX cells at most)
template <int RMAX>
__global__ void __launch_bounds__(CT, 1)
k_mg_cluster(MgCluster M, const float *f, float *x, const KrylovState *st) {
    extern __shared__ __align__(16) float cluster_smem[];
    float *sm = cluster_smem;
    // the level table and its coefficients; x and f zeroed (the lanes' rows
    // past a column's end stay zero)
    for (int n = threadIdx.x; n < M.words; n += CT) sm[n] = M.image[n];
    for (int n = M.words + threadIdx.x; n < M.total; n += CT) sm[n] = 0.f;
    __syncthreads();
    Cycle y;
    y.rank = cluster_rank();
    y.blocks = M.blocks;
    y.sm = sm;
    y.lv = reinterpret_cast<const MgClusterLevel *>(sm);
    y.tables = M.tables;
    y.zeros = sm + M.zeros;
    y.zeros_at = in_block(y.zeros, y.rank);
    y.lane = threadIdx.x & 31;
    y.warp = threadIdx.x >> 5;
    y.map_planes(M.levels);
    const MgClusterLevel &c = y.lv[0];
    const int i0 = y.first(c, y.rank), np = y.first(c, y.rank + 1) - i0;
    pdl_wait();
    if (st->done) return;  // the same in every block
    for (int q = y.warp; q < np * c.n[1]; q += CW) {
        const int ip = q / c.n[1], j = q - ip * c.n[1];
        const float *src = f + M.top.at(i0 + ip, j, 0);
        for (int k = y.lane; k < c.n[2]; k += 32) copy_async(sm + c.f + q * c.S + k, src + k);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_sync();
    const int last = M.levels - 1;
    // down the levels, the coarsest solve, and up again
#pragma unroll 1
    for (int t = 0; t <= 2 * last; t++) {
        if (t == last) {
            y.coarse(last, M.kinv, M.ncoarse);
            continue;
        }
        const int l = t < last ? t : 2 * last - t;
        y.smooth<RMAX>(l, mg_nu(M.first + l), t > last);
        if (t < last) y.restrict_to(l);
    }
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

// the kernel for this cycle
auto kernel_of(const MgCluster &M) {
    const int R = (M.top.n[2] + 31) / 32;
    return R == 1 ? k_mg_cluster<1> : R == 2 ? k_mg_cluster<2> : R == 3 ? k_mg_cluster<3> : k_mg_cluster<4>;
}

}  // namespace

bool mg_cluster_fits(const MgCluster &M) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = config(M, attr, 0);
    cfg.numAttrs = 1;
    int n = 0;
    auto k = kernel_of(M);
    allow_shared(k, MG_CLUSTER_SMEM);
    DALM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
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
