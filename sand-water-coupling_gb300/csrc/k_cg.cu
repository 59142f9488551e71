// k_cg.cu -- matrix-free virtual Laplacian and CG of the dual-particle SPH
// projection (reference: VirtualParticle::calculateCoef / solveLinearSystem,
// Cores/Structures/VirtualParticle.cpp:149-169,105-108, and the Eigen CG behind
// Cores/Solvers/IterativeSolver.h:21-40).
//
// Because virtual particles sit on lattice nodes, alpha_IJ = c(|k|^2) V_J with a
// radial coefficient table c, so
//     (A v)_I = alpha_hat_I v_I + sum_{0 < |k|^2 < 16} c(|k|^2) (V v)_{I+k}
// on active rows; inactive rows are identity rows with zero right-hand side and
// zero start, so CG over whole bricks is CG over the active set.
//
// Here: the start of a solve (residual sums, start state, the choice between two
// starts) and the block-per-brick operator kernels of the true residual and of
// swc_apply_operator; the solve itself and the residual / alpha_hat row passes are in
// k_cg_solve.cu.  Dot products use exact FP32 products summed in float-float below
// the warp and FP64 above, reduced
// deterministically.  A is not symmetric (alpha_IJ carries V_J) and the
// reference runs Hestenes-Stiefel CG on the full matrix, so single-reduction
// rearrangements that rely on symmetry (Chronopoulos-Gear, pipelined CG) are
// not equivalent here: on a 2D dam break the Chronopoulos-Gear form stalls
// after ~10 iterations where this form converges.
#include "swc_kernels.h"
#include "swc_tiles.cuh"

namespace swc {

template<int DIM> struct KG {
    static constexpr int NT = RowGeom<DIM>::NT;         // rows per brick
    static constexpr int BT = NT < 32 ? 32 : NT;        // threads per block
};
constexpr int kUT = 256;  // threads per block of the streaming update

__device__ __forceinline__ float4 ld4(const float * a, long long s) { return *reinterpret_cast<const float4 *>(a + s); }
__device__ __forceinline__ void st4(float * a, long long s, float4 v) { *reinterpret_cast<float4 *>(a + s) = v; }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 fma4(float s, float4 a, float4 b) {
    return make_float4(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y), fmaf(s, a.z, b.z), fmaf(s, a.w, b.w));
}
__device__ __forceinline__ float comp(const float4 & v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }
__device__ __forceinline__ unsigned char compb(const uchar4 & v, int j) {
    return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
}

// Slot of the first node of brick row (ly, lz).
template<int DIM> __device__ __forceinline__ long long row_base(int b, int ly, int lz) {
    using G = BrickGeom<DIM>;
    return (long long) b * G::BN + G::BX * (ly + G::BY * lz);
}

// y = A v (test hook).
template<int DIM>
__global__ void __launch_bounds__(KG<DIM>::BT) k_apply_operator(Lattice L, const int * __restrict__ blist,
                                                                const int * __restrict__ bcount,
                                                                const unsigned char * __restrict__ bflag, NodeArrays N,
                                                                Stencil S, const float * __restrict__ in,
                                                                float * __restrict__ out) {
    using G = BrickGeom<DIM>;
    __shared__ __align__(16) float tile[G::TILE];
    const int nb = *bcount;
    const int t = threadIdx.x, ly = t % G::BY, lz = t / G::BY;
    for (int bi = blockIdx.x; bi < nb; bi += gridDim.x) {
        const int b   = blist[bi];
        const int3 bc = brick_coords(L, b);
        __syncthreads();
        load_tile4<DIM>(L, bflag, bc, tile, [&](long long s) { return mul4(ld4(N.V, s), ld4(in, s)); });
        __syncthreads();
        if (t < KG<DIM>::NT) {
            float acc[G::BX];
            stencil_row<DIM>(tile, ly, lz, S, acc);
            const long long base = row_base<DIM>(b, ly, lz);
#pragma unroll
            for (int k = 0; k < G::BX / 4; k++) {
                const float4 v = ld4(in, base + 4 * k), a = ld4(N.ahat, base + 4 * k);
                const uchar4 f = *reinterpret_cast<const uchar4 *>(N.flag + base + 4 * k);
                float4 o;
                o.x = f.x ? fmaf(a.x, v.x, acc[4 * k]) : v.x;
                o.y = f.y ? fmaf(a.y, v.y, acc[4 * k + 1]) : v.y;
                o.z = f.z ? fmaf(a.z, v.z, acc[4 * k + 2]) : v.z;
                o.w = f.w ? fmaf(a.w, v.w, acc[4 * k + 3]) : v.w;
                st4(out, base + 4 * k, o);
            }
        }
    }
}

// The base start won the residual test: x = xb, r = d = rb (all slots of the
// active bricks, 16-byte streaming).
template<int DIM>
__global__ void __launch_bounds__(kUT) k_cg_pick_base(const int * __restrict__ blist, const int * __restrict__ bcount,
                                                      NodeArrays N, const float * __restrict__ xb,
                                                      const float * __restrict__ rb, const CgState * __restrict__ cg) {
    pdl_wait_and_release();
    using G = BrickGeom<DIM>;
    constexpr int Q = G::BN / 4;
    if (cg->start != 1) return;
    const int nb = *bcount;
    for (long long e = blockIdx.x * (long long) kUT + threadIdx.x; e < (long long) nb * Q; e += (long long) gridDim.x * kUT) {
        const long long s = (long long) blist[e / Q] * G::BN + 4 * (e % Q);
        const float4 r = ld4(rb, s);
        st4(N.x, s, ld4(xb, s));
        st4(N.r, s, r);
        st4(N.d, s, r);
    }
}

// u = V x over the slots of the active bricks (16-byte streaming).
template<int DIM>
__global__ void __launch_bounds__(kUT) k_vmul(const int * __restrict__ blist, const int * __restrict__ bcount,
                                              const float * __restrict__ V, const float * __restrict__ x,
                                              float * __restrict__ u) {
    pdl_wait_and_release();
    using G = BrickGeom<DIM>;
    constexpr int Q = G::BN / 4;
    const long long total = (long long) (*bcount) * Q;
    for (long long e = blockIdx.x * (long long) kUT + threadIdx.x; e < total; e += (long long) gridDim.x * kUT) {
        const long long s = (long long) blist[e / Q] * G::BN + 4 * (e % Q);
        st4(u, s, mul4(ld4(V, s), ld4(x, s)));
    }
}

// CG start state from the residual sums (Eigen's stopping rule:
// |r|^2 < max(tol, eps/|b|)^2 |b|^2, cap 2 N_v).  With a second candidate
// (sums_b, the base start of the learned warm start) the prediction is kept
// when the network reported no error, its residual is finite and, unless
// keep_prediction, not larger than the base's; cg->start records the choice
// (0 prediction, 1 base) for k_cg_pick_base and the host.
__global__ void k_cg_start(CgState * cg, const double * __restrict__ sums_l, const double * __restrict__ sums_b,
                           const int * __restrict__ mlp_err, int keep_prediction, double tol, int max_iterations,
                           const int * __restrict__ nv) {
    pdl_wait_and_release();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double srr_l = sums_l[0], sbb = sums_l[1];
    bool keep = true;
    if (sums_b) {
        const double srr_b = sums_b[0];
        keep = (!mlp_err || *mlp_err == 0) && srr_l == srr_l && (keep_prediction || srr_l <= srr_b);
    }
    const double srr = keep ? srr_l : sums_b[0];
    cg->failed  = 0;
    cg->start   = keep ? 0 : 1;
    cg->bb      = sbb;
    cg->rr      = srr;
    cg->rr0     = srr;
    cg->iter    = 0;
    const int n  = *nv;
    cg->max_iter = max_iterations >= 0 ? max_iterations : 2 * n;
    const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
    if (n == 0 || sbb == 0.0) {
        cg->threshold = 0;
        cg->done      = sbb == 0.0 ? 4 : 1;  // 4: zero right-hand side -> x = 0
    } else {
        const double tt = fmax(tol, eps / sqrt(sbb));
        cg->threshold   = fmax(tt * tt * sbb, dmin);
        cg->done        = srr < cg->threshold ? 1 : (srr != srr ? 3 : 0);
        if (cg->done == 0 && cg->max_iter <= 0) cg->done = 2;
    }
}

// True residual |b - A x|^2 and |b|^2 (FP64, out2[0], out2[1]).
// |b|^2 = sum_I D_I^2 into cg->bb (the learned start's scale sD before the
// solve, when no fallback residual of the node-mapped start is needed).
template<int DIM>
__global__ void __launch_bounds__(kUT) k_rhs_norm(const int * __restrict__ blist, const int * __restrict__ bcount,
                                                  NodeArrays N, CgState * cg, double * __restrict__ partials) {
    pdl_wait_and_release();
    using G = BrickGeom<DIM>;
    constexpr int Q = G::BN / 4;
    __shared__ double red[kUT / 32 + 1];
    __shared__ int last;
    const long long total = (long long) (*bcount) * Q;
    FF bb{0.f, 0.f};
    for (long long i = blockIdx.x * (long long) kUT + threadIdx.x; i < total; i += (long long) gridDim.x * kUT) {
        const float4 d = ld4(N.D, (long long) blist[i / Q] * G::BN + 4 * (i % Q));
        ff_add_prod(bb, d.x, d.x);
        ff_add_prod(bb, d.y, d.y);
        ff_add_prod(bb, d.z, d.z);
        ff_add_prod(bb, d.w, d.w);
    }
    double part[1] = {block_sum_ff<kUT>(bb, red)};
    double tot[1];
    if (grid_reduce<kUT, 1>(part, partials, &cg->ticket[3], tot, red, &last) && threadIdx.x == 0) cg->bb = tot[0];
}

template<int DIM>
__global__ void __launch_bounds__(KG<DIM>::BT) k_true_residual(Lattice L, const int * __restrict__ blist,
                                                               const int * __restrict__ bcount,
                                                               const unsigned char * __restrict__ bflag, NodeArrays N,
                                                               Stencil S, CgState * cg, double * __restrict__ partials,
                                                               double * __restrict__ out2) {
    using G = BrickGeom<DIM>;
    constexpr int BT = KG<DIM>::BT;
    __shared__ __align__(16) float tile[G::TILE];
    __shared__ double red[BT / 32 + 1];
    __shared__ int last;
    const int nb = *bcount;
    const int t = threadIdx.x, ly = t % G::BY, lz = t / G::BY;
    double rr = 0, bb = 0;
    for (int bi = blockIdx.x; bi < nb; bi += gridDim.x) {
        const int b   = blist[bi];
        const int3 bc = brick_coords(L, b);
        __syncthreads();
        load_tile4<DIM>(L, bflag, bc, tile, [&](long long s) { return mul4(ld4(N.V, s), ld4(N.x, s)); });
        __syncthreads();
        if (t < KG<DIM>::NT) {
            float acc[G::BX];
            stencil_row<DIM>(tile, ly, lz, S, acc);
            const long long base = row_base<DIM>(b, ly, lz);
#pragma unroll
            for (int i = 0; i < G::BX; i++) {
                if (!N.flag[base + i]) continue;
                const double q = double(N.ahat[base + i]) * N.x[base + i] + double(acc[i]);
                const double r = double(N.D[base + i]) - q;
                rr += r * r;
                bb += double(N.D[base + i]) * N.D[base + i];
            }
        }
    }
    double part[2] = {block_sum_double<BT>(rr, red), 0.0};
    part[1]        = block_sum_double<BT>(bb, red);
    double tot[2];
    if (grid_reduce<BT, 2>(part, partials, &cg->ticket[3], tot, red, &last) && threadIdx.x == 0) {
        out2[0] = tot[0];
        out2[1] = tot[1];
    }
}

// ---------------------------------------------------------------------------
// Launchers (sgrid: blocks of the row-stencil kernels; ugrid: of the update)
// ---------------------------------------------------------------------------
template<int DIM>
void launch_apply_operator(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                           const float * in, float * out, int sgrid, cudaStream_t st) {
    k_apply_operator<DIM><<<sgrid, KG<DIM>::BT, 0, st>>>(L, B.list, B.count, B.flag, N, S, in, out);
}
// Residual of one candidate start x: r = b - A x into r (and d when non-null),
// |r|^2 and |b|^2 into sums[0..1] (u = V x staged in N.u).
template<int DIM>
void launch_cg_residual(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                        const float * x, float * r, float * d, double * sums, CgState * cg, double * partials,
                        int rblocks, int ugrid, cudaStream_t st) {
    launch_pdl(k_vmul<DIM>, ugrid, kUT, 0, st, B.list, B.count, N.V, x, N.u);
    launch_rows_residual<DIM>(L, B, N, S, x, r, d, sums, cg, partials, rblocks, st);
}
// Start state keeping the better of the prediction (residual in cg->sums[0..1],
// already in N.x / N.r / N.d) and the base start xb (cg->sums[2..3], residual rb),
// and the base copied in when it wins.
template<int DIM>
void launch_cg_pick(const BrickArrays & B, const NodeArrays & N, const float * xb, const float * rb,
                    const int * mlp_err, bool keep_prediction, CgState * cg, double tol, int max_iterations,
                    const int * nv, int ugrid, cudaStream_t st) {
    launch_pdl(k_cg_start, 1, 32, 0, st, cg, cg->sums, cg->sums + 2, mlp_err, keep_prediction ? 1 : 0, tol,
               max_iterations, nv);
    launch_pdl(k_cg_pick_base<DIM>, ugrid, kUT, 0, st, B.list, B.count, N, xb, rb, cg);
}
template<int DIM>
void launch_true_residual(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                          CgState * cg, double * partials, double * out2, int sgrid, cudaStream_t st) {
    k_true_residual<DIM><<<sgrid, KG<DIM>::BT, 0, st>>>(L, B.list, B.count, B.flag, N, S, cg, partials, out2);
}
template<int DIM>
void launch_rhs_norm(const BrickArrays & B, const NodeArrays & N, CgState * cg, double * partials, int ugrid,
                     cudaStream_t st) {
    launch_pdl(k_rhs_norm<DIM>, ugrid, kUT, 0, st, B.list, B.count, N, cg, partials);
}

#define SWC_INST(D)                                                                                                    \
    template void launch_apply_operator<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,   \
                                           const float *, float *, int, cudaStream_t);                                 \
    template void launch_cg_residual<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,     \
                                        const float *, float *, float *, double *, CgState *, double *, int, int,      \
                                        cudaStream_t);                                                                 \
    template void launch_cg_pick<D>(const BrickArrays &, const NodeArrays &, const float *, const float *, const int *, \
                                    bool, CgState *, double, int, const int *, int, cudaStream_t);                     \
    template void launch_true_residual<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,   \
                                          CgState *, double *, double *, int, cudaStream_t);                           \
    template void launch_rhs_norm<D>(const BrickArrays &, const NodeArrays &, CgState *, double *, int, cudaStream_t);
SWC_INST(2)
SWC_INST(3)
#undef SWC_INST

}  // namespace swc
