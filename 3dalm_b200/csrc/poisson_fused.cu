// BiCGStab iterations of large grids as three kernels: the two halves
// (poisson_half.cuh), each followed by its scalar update in the last block,
// and the x / r update.  20 vectors per cell and iteration pass through HBM
// (P half: r, p, q, r0 in, p, pp, q out; S half: r, q in, s, ss, t out; x / r
// update 8) against 35 with one kernel per reference loop.  p and q are
// ping-pong buffers, because a block reads its neighbours' old p and q as its
// halo while it writes its own new ones.
//
// One block per SM, each marching an equal range of (tile, plane) units, so
// the last wave is always full.
//
// 512 x 256 x 128, per iteration: P half 263 us, S half 200 us, x / r update
// 214 us (its 1.07 GB at 5.0 TB/s), against 860 us for the nine launches of one
// kernel per loop.  The halves' bytes would take 144 and 103 us.
#include "poisson_half.cuh"

namespace dalm {

namespace {

template <int KIND, typename G>
__global__ void __launch_bounds__(G::THREADS, 1)
k_half(Grid g, PoissonCoef C, HalfPlan H, const __grid_constant__ CUtensorMap mr,
       const __grid_constant__ CUtensorMap mp, const __grid_constant__ CUtensorMap mq, HalfArgs A,
       Partials<2> part, KrylovState *st) {
    if (st->done) return;
    extern __shared__ __align__(128) unsigned char half_smem[];
    __shared__ __align__(8) unsigned long long bar[4];
    HalfRing R(bar);
    const long long u0 = H.units * blockIdx.x / gridDim.x,
                    u1 = H.units * (blockIdx.x + 1) / gridDim.x;
    double acc[2] = {0.0, 0.0};
    const bool ok = half_march<KIND, G>(g, C, H, &mr, &mp, &mq, A, KIND == HALF_P ? st->beta : st->alpha,
                                        st->omega, st->it == 0, u0, u1, half_smem, R, acc);
    if (!ok) {
        if (threadIdx.x == 0) {
            st->wait_error = 1;
            st->done = 1;
        }
        return;
    }
    if (grid_reduce<2>(acc, 0u, part) && threadIdx.x == 0) {
        if (KIND == HALF_P) fin_q(st, acc[0]);
        else fin_t(st, acc[0], acc[1]);
    }
}

template <int KIND, typename G>
void half_launch(const LaunchCtx &L, int kind_tag, const Grid &g, const PoissonCoef &C,
                 const PoissonConfig &cfg, const double *r, const double *p, const double *q,
                 const HalfArgs &A, Partials<2> part, KrylovState *st) {
    const HalfPlan H = HalfPlan::make(cfg.seg.box, G::BJ, G::BK);
    const int blocks = (int)(H.units < cfg.sm_count ? H.units : cfg.sm_count);
    const MapTable &M = *cfg.maps;
    // an attribute of the function in the current device's context: set on
    // every launch, so handles on several devices or threads share no flag
    DALM_CUDA(cudaFuncSetAttribute(k_half<KIND, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   G::SMEM));
    L.pre(kind_tag);
    k_half<KIND, G><<<blocks, G::THREADS, G::SMEM, L.s>>>(g, C, H, M.of(r).half, M.of(p).half,
                                                          M.of(q).half, A, part, st);
    L.post(kind_tag);
}

template <typename G>
void iteration(const LaunchCtx &L, const Grid &g, const PoissonCoef &C, const PoissonBufs &B,
               long long n, const PoissonConfig &cfg, Partials<2> part, KrylovState *st) {
    double *pk[2] = {B.pk, B.tp}, *q[2] = {B.q, B.ts};
    const int a = (int)(n & 1), b = 1 - a;
    half_launch<HALF_P, G>(L, KK_BICG_PF, g, C, cfg, B.r, pk[a], q[a],
                           HalfArgs{B.r0, pk[b], B.pp, q[b]}, part, st);
    half_launch<HALF_S, G>(L, KK_BICG_SF, g, C, cfg, B.r, B.r, q[b],
                           HalfArgs{nullptr, B.s, B.ss, B.t}, part, st);
    launch_bicg_xr(L, g, B, B.pp, B.ss, cfg, part, st);
}

}  // namespace

bool fused_bicg_available(const PoissonConfig &cfg) {
    return cfg.method == PM_BICG && cfg.pc == PC_JACOBI && cfg.pc_sweeps == HH &&
           !cfg.reference_sums;
}

void launch_bicg_iteration_fused(const LaunchCtx &L, const Grid &g, const PoissonCoef &C,
                                 const PoissonBufs &B, long long n, const PoissonConfig &cfg,
                                 Partials<2> part, KrylovState *st) {
    if (g.nk() > HalfNarrow::BK)
        iteration<HalfWide>(L, g, C, B, n, cfg, part, st);
    else
        iteration<HalfNarrow>(L, g, C, B, n, cfg, part, st);
}

}  // namespace dalm
