// k_cg_solve.cu -- the CG solve of the projection as one resident kernel, and the
// other row-stencil passes on the same warp-per-brick stencil (alpha_hat, residuals
// of the CG start).
//
// CG (Eigen's Hestenes-Stiefel form on the full matrix, k_cg.cu) from the start
// state to its end in one cooperative launch, one block per SM (or, for lattices of few
// bricks, one cluster).  A group of W warps
// (fewer where bricks are many) owns its bricks in both phases of an iteration:
//   step      x += alpha d, r -= alpha q, d = r + beta d, u = V d       (streaming)
//   product   q = A d from the halo tile of u (swc_stencil.cuh), and the four dot
//             products d.q, r.q, q.q, r.r
// (before the first: u = V x, r = d = b - A x, r.r and b.b, and the stopping threshold,
// unless the caller queued a start of its own.  As three launches, with the sums in FP64
// in every block, the start took 19 us at 15,625 particles, against 7 here.)
// alpha = r.r / d.q, and |r - alpha q|^2 = r.r - 2 alpha r.q + alpha^2 q.q gives beta
// without a second trip: the sums hold 44 bits and more, so at a quotient of two
// successive norms of a tenth, below which it seldom is, the prediction is good to 2^-44
// and at kPredict to 2^-40, where the rounding of the stored r alone makes 2^-31 (at 1e-6,
// where the line lay first, 2^-28).  Below kPredict, and where the prediction ends the
// solve, the norm is summed from r - alpha q itself: the stopping test and the residual
// that is reported are of the r that is stored.  r.r is summed from r in every
// iteration, so nothing of a prediction is carried on.  q.q is summed times a power of two
// near 1 / |A| (CgStart::qscale), so that its FP32 products hold over the range of lengths and
// velocities that those of d.q do.
// Before a warp copies a tile it waits for the flags of the brick's neighbours; the
// blocks meet once per iteration, for the sums, and each decides by itself whether to
// go on, with no host check.  Dot products use exact FP32 products in float-float per
// lane and triple floats above (the start's |r|^2 and |b|^2: FP64 above the block), in a
// fixed order.
#include <type_traits>

#include "swc_kernels.h"
#include "swc_stencil.cuh"

namespace swc {

namespace {

__device__ __forceinline__ float4 ld4(const float * a, long long s) { return *reinterpret_cast<const float4 *>(a + s); }
__device__ __forceinline__ void st4(float * a, long long s, float4 v) { *reinterpret_cast<float4 *>(a + s) = v; }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 fma4(float s, float4 a, float4 b) {
    return make_float4(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y), fmaf(s, a.z, b.z), fmaf(s, a.w, b.w));
}
__device__ __forceinline__ float comp(const float4 & v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }

constexpr int kSums = 4;  // values of a meeting

// Triple floats (three error-free terms, about 70 bits) hold the sums above the lane and
// the scalars of the iteration.  GB300 adds or converts two FP64 values per SM and
// clock, with a latency of 65 clocks and far more for a quotient: with FP64 here a meeting
// took 7,100 clocks in a block alone.  The sums are scaled by a power of two that brings
// |b|^2, and later r.r when it has left 2^-48 .. 2^48 (decide), to about 1, so they stay in
// the range of the FP32 products however far the solve goes.
struct F3 {
    float h, m, l;
};
__device__ __forceinline__ F3 f3_add(const F3 & a, const F3 & b) {
    float s, e, t, f, u, g;
    F3 o;
    two_sum(a.h, b.h, s, e);
    two_sum(a.m, b.m, t, f);
    two_sum(e, t, u, g);
    o.l = __fadd_rn(__fadd_rn(a.l, b.l), __fadd_rn(f, g));
    fast_two_sum(s, u, o.h, o.m);
    return o;
}
__device__ __forceinline__ F3 f3_shfl(const F3 & a, int o) {
    return F3{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.m, o),
              __shfl_xor_sync(0xffffffffu, a.l, o)};
}
// Sums of four float-float values, scaled, over the warp: lanes 8 k .. 8 k + 7 get value k's.
__device__ __forceinline__ F3 warp_sum4(const FF (&p)[kSums], float scale) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16, odd = lane & 8;
    F3 q[kSums];
#pragma unroll
    for (int k = 0; k < kSums; k++) q[k] = F3{p[k].hi * scale, p[k].lo * scale, 0.f};
    // the halves of the warp, then its quarters, exchange the values that they give up
    const F3 a = f3_add(up ? q[2] : q[0], f3_shfl(up ? q[0] : q[2], 16));
    const F3 b = f3_add(up ? q[3] : q[1], f3_shfl(up ? q[1] : q[3], 16));
    F3 c       = f3_add(odd ? b : a, f3_shfl(odd ? a : b, 8));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) c = f3_add(c, f3_shfl(c, o));
    return c;
}
// a * k (k a float)
__device__ __forceinline__ F3 f3_scale(const F3 & a, float k) {
    const float p = __fmul_rn(a.h, k), e = __fmaf_rn(a.h, k, -p), q = __fmul_rn(a.m, k);
    const float f = __fmaf_rn(a.m, k, -q);
    float s, t;
    F3 o;
    two_sum(e, q, s, t);
    o.l = __fmaf_rn(a.l, k, __fadd_rn(f, t));
    fast_two_sum(p, s, o.h, o.m);
    return o;
}
// float(a / b): the FP32 quotient and one correction from the exact remainder (about 44
// bits before the last rounding)
__device__ __forceinline__ float f3_quotient(const F3 & a, const F3 & b) {
    const float q = __fdiv_rn(a.h, b.h);
    const F3 r    = f3_add(a, f3_scale(b, -q));
    return __fadd_rn(q, __fdiv_rn(__fadd_rn(r.h, r.m), b.h));
}
__device__ __forceinline__ double f3_double(const F3 & a) { return (double(a.h) + double(a.m)) + double(a.l); }
__device__ __forceinline__ F3 f3_of(double v) {
    F3 o;
    o.h = float(v);
    o.m = float(v - double(o.h));
    o.l = float((v - double(o.h)) - double(o.m));
    return o;
}

// A meeting's words are 16 bytes, value and tag written and read as one.
__device__ __forceinline__ void word_put(ulonglong2 * p, unsigned long long a, unsigned long long b) {
    asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ ulonglong2 word_get(const ulonglong2 * p) {
    ulonglong2 v;
    asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p)
                 : "memory");
    return v;
}
// A block's partial sum and its tag.
__device__ __forceinline__ void slot_put(ulonglong2 * p, const F3 & v, unsigned tag) {
    word_put(p, (unsigned long long) __float_as_uint(v.m) << 32 | __float_as_uint(v.h),
             (unsigned long long) tag << 32 | __float_as_uint(v.l));
}
__device__ __forceinline__ bool slot_get(const ulonglong2 * p, unsigned tag, F3 & v) {
    const ulonglong2 w = word_get(p);
    v = F3{__uint_as_float(unsigned(w.x)), __uint_as_float(unsigned(w.x >> 32)), __uint_as_float(unsigned(w.y))};
    return unsigned(w.y >> 32) == tag;
}
// What block 0 made of the sums: the step's factors and how to go on.
enum : unsigned { kGoOn = 0, kFailed = 5, kMeasure = 6 };  // 1, 2, 3: CgState::done
struct Outcome {
    float    alpha, beta;
    unsigned code;
    int      shift = 0;  // the sums' scale grows by 2^shift
};
__device__ __forceinline__ void outcome_put(ulonglong2 * p, const Outcome & o, unsigned tag) {
    word_put(p, (unsigned long long) __float_as_uint(o.beta) << 32 | __float_as_uint(o.alpha),
             (unsigned long long) tag << 32 | unsigned(o.shift) << 8 | o.code);
}
__device__ __forceinline__ bool outcome_get(const ulonglong2 * p, unsigned tag, Outcome & o) {
    const ulonglong2 w = word_get(p);
    o.alpha            = __uint_as_float(unsigned(w.x));
    o.beta             = __uint_as_float(unsigned(w.x >> 32));
    o.code             = unsigned(w.y) & 0xffu;
    o.shift            = int(unsigned(w.y)) >> 8;
    return unsigned(w.y >> 32) == tag;
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned * p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned * p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(v));
    return v;
}

// Block 0's view of the solve (scaled).
struct CgScalars {
    F3    rr, rr_next;
    float threshold_h, threshold_l;  // times 2^threshold_e
    int   threshold_e;
    float qinv;  // 1 / qscale
    int   it, max_iter;
};
// 2^e, 0 where it is below the normal floats
__device__ __forceinline__ float pow2(int e) { return __int_as_float(max(0, min(254, 127 + e)) << 23); }
constexpr int kCluster = 16;  // blocks of a cluster's solve, at most
template<int WARPS> struct MeetSmem {
    F3        part[WARPS][kSums];
    F3        sum[kSums];
    double    start[2];
    int       nv;  // block 0
    int       full[kSums];
    Outcome   out;
    CgScalars cg;  // block 0
};
// A cluster's partials, by the meeting's parity: two meetings may have no other barrier
// between them.
template<int WARPS> struct ClusterSmem : MeetSmem<WARPS> {
    F3     all[2][kCluster][kSums];
    double all_start[kCluster][2];
};
// The power of two that brings |b|^2 to about 1.
__device__ __forceinline__ float sum_scale(double bb) { return exp2f(float(-max(-120, min(120, ilogb(bb))))); }
__device__ __forceinline__ CgScalars scalars_of(double rr, double threshold, int max_iter, float scale, float qscale) {
    const F3 r = f3_of(rr * double(scale));
    const int e = threshold > 0 ? ilogb(threshold) : 0;
    const F3 t  = f3_of(scalbn(threshold, -e));
    return CgScalars{r, r, t.h, t.m, e + ilogbf(scale), 1.f / qscale, 0, max_iter};
}
constexpr float kPredict = 1.f / 128.f;  // of r.r: a smaller norm is measured, not predicted
constexpr int kRescale = 48;             // bits that r.r may move before the sums' scale follows it
constexpr int kCopies = 8;               // copies of a meeting's outcome, so that fewer blocks poll one line

// How to go on (Outcome's code, the shift in the bits above its 8) where an iteration's norm
// n calls for a closer look: its measurement first.  Out of line: few iterations come here,
// and the code of the others is at the size of the instruction caches (with these cases in
// the decision itself CG took 267 us a step at 87,025 particles in 2D and 211 in the 2D dam
// break, 247 and 204 without).
__device__ __noinline__ int decide_seldom(float nh, float nm, float pq, float th, float tl, int left, bool measured,
                                          bool timed) {
    if (timed) return left > 0 ? int(kGoOn) : 2;  // no end but the cap
    if (!measured) return !(pq != 0.f) || pq != pq ? 3 : int(kMeasure);
    if (nh != nh) return 3;
    // (r = 0 is below any threshold, also one that the scale takes to 0 in FP32)
    if (!(nh > 0.f) || nh < th || (nh == th && nm < tl)) return 1;
    if (left <= 0) return 2;
    const int e = int(__float_as_uint(nh) >> 23) - 127;
    return abs(e) > kRescale ? max(-120, min(120, -e)) * 256 : int(kGoOn);
}
// The factors and the stopping test from the sums d.q, r.q, q.q (times qscale), r.r (after
// kMeasure: from |r - alpha q|^2).  An iteration goes on at once where its predicted norm is
// above kPredict r.r and, by a margin far above the prediction's error, the threshold,
// within the scale's range, and not the cap's last.
__device__ __forceinline__ Outcome decide(CgScalars & c, const F3 (&sum)[kSums], float alpha, bool measured,
                                          bool timed) {
    Outcome o{alpha, 0.f, kGoOn};
    if (!measured) {
        c.rr       = sum[3];
        o.alpha    = f3_quotient(c.rr, sum[0]);
        const F3 t = f3_add(f3_scale(sum[2], o.alpha * c.qinv), f3_scale(sum[1], -2.f));
        c.rr_next  = f3_add(c.rr, f3_scale(t, o.alpha));
    } else c.rr_next = sum[0];
    const F3 & n   = c.rr_next;
    const float t2 = pow2(c.threshold_e), th = c.threshold_h * t2;
    const int left = c.max_iter - c.it - 1;
    const float lo = fmaxf(fmaxf(kPredict * c.rr.h, th * (1.f + 0x1p-16f)), pow2(-kRescale));
    if (measured || !(n.h > lo && n.h < pow2(kRescale)) || left <= 0) {
        const int what = decide_seldom(n.h, n.m, sum[0].h, th, c.threshold_l * t2, left, measured, timed);
        o.code         = unsigned(what) & 0xffu;
        o.shift        = what >> 8;
        if (!measured && o.code >= 3) return o;  // (kMeasure among them)
        c.threshold_e += o.shift;
    }
    c.it++;
    o.beta = f3_quotient(n, c.rr);
    return o;
}

// Start state from |r|^2 and |b|^2 (Eigen's stopping rule: |r|^2 < max(tol, eps/|b|)^2
// |b|^2, cap 2 N_v), into *cg when given.  The outcome's alpha is the power of two that
// scales the sums.
__device__ __forceinline__ Outcome decide_start(CgState * cg, CgScalars & c, double rr, double bb, int nv,
                                               const CgStart & from) {
    const int cap = from.max_iterations >= 0 ? from.max_iterations : 2 * nv;
    const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
    int done = 0;
    double threshold = 0;
    if (nv == 0 || bb == 0.0) done = bb == 0.0 ? 4 : 1;  // 4: zero right-hand side -> x = 0
    else {
        // (the quotient only where it may be the larger one)
        double tt = from.tolerance;
        if (!(tt * tt * bb > 4 * eps * eps)) tt = fmax(tt, eps / sqrt(bb));
        threshold = fmax(tt * tt * bb, dmin);
        done      = rr < threshold ? 1 : (rr != rr ? 3 : 0);
        if (done == 0 && cap <= 0) done = 2;
    }
    if (from.timed) done = 0;
    if (cg) {
        cg->start     = 0;
        cg->bb        = bb;
        cg->rr        = rr;
        cg->rr0       = rr;
        cg->iter      = 0;
        cg->max_iter  = cap;
        cg->threshold = threshold;
        cg->done      = done;
    }
    const float scale = sum_scale(bb);
    c = scalars_of(rr, threshold, cap, scale, from.qscale);
    return Outcome{scale, 0.f, unsigned(done)};
}

// Meeting of the blocks in use: v (value lane / 8 of the warp, as warp_sum4 gives it)
// summed over their first `active` warps, and what block 0 decides on the sums, the
// same on every thread.  Every block publishes its four partials under the meeting's
// tag; block 0 reads them all and publishes the outcome, one word that the others poll.
// (With every block polling every slot the polls themselves, 64 B x blocks^2 a round, kept
// the slots from being written: 13 us a meeting of 152 blocks; with the sums published and
// FP64 quotients formed by every thread, 5 us.)  One set of
// slots serves: a block publishes again only after it has the outcome, and block 0
// only after every block has published again.
// START: values 0 and 1 are |r|^2 and |b|^2, unscaled, in FP64 above the block (once a
// solve, by one warp each); `decided` makes the outcome of the sums.  A wait ends after
// `polls` more looks at its word, with kFailed.
template<bool START, int WARPS, class Decide>
__device__ __forceinline__ Outcome meet(const F3 & v, ulonglong2 * slots, int stride, int blocks, int active,
                                        int polls, unsigned & tag, MeetSmem<WARPS> & M, Decide decided) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ulonglong2 * outcome = slots + (long long) stride * kSums;
    if ((lane & 7) == 0) M.part[warp][lane >> 3] = v;
    __syncthreads();
    if (warp == 0) {
        const int k = lane >> 3, w = lane & 7;
        F3 part{0.f, 0.f, 0.f};
        for (int j = w; j < active; j += 8) part = f3_add(part, M.part[j][k]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) part = f3_add(part, f3_shfl(part, o));
        if (w == 0) {
            ulonglong2 * p = slots + (long long) blockIdx.x * kSums + k;
            if constexpr (START) {
                if (k < 2)
                    word_put(p, (unsigned long long) __double_as_longlong(f3_double(part)), (unsigned long long) tag << 32);
            } else slot_put(p, part, tag);
        }
        if (blockIdx.x != 0 && lane == 0) {
            const ulonglong2 * p = outcome + blockIdx.x % kCopies;
            Outcome o;
            bool there;
            int n = polls;
            do there = outcome_get(p, tag, o);
            while (!there && n-- > 0);
            if (!there) o.code = kFailed;
            M.out = o;
        }
    }
    if (blockIdx.x == 0) {
        // a warp per value, five slots a lane at once
        if constexpr (START) {
            if (warp < 2) {
                double s  = 0;
                bool full = true;
                for (int j = lane; j < blocks; j += 32) {
                    ulonglong2 w{0, 0};
                    bool there;
                    int n = polls;
                    do {
                        w     = word_get(slots + (long long) j * kSums + warp);
                        there = unsigned(w.y >> 32) == tag;
                    } while (!there && n-- > 0);
                    full = full && there;
                    s += __longlong_as_double((long long) w.x);
                }
                __syncwarp();
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
                full = __all_sync(0xffffffffu, full);
                if (lane == 0) M.start[warp] = s, M.full[warp] = full;
            }
        } else if (warp < kSums) {
            F3 s{0.f, 0.f, 0.f};
            bool full = true;
            for (int j0 = lane; j0 < blocks; j0 += 32 * 5) {
                F3 e[5];
                bool there;
                int n = polls;
                do {
                    there = true;
#pragma unroll
                    for (int q = 0; q < 5; q++) {
                        const int j = j0 + 32 * q;
                        e[q]        = F3{0.f, 0.f, 0.f};
                        if (j < blocks) there = slot_get(slots + (long long) j * kSums + warp, tag, e[q]) && there;
                    }
                } while (!there && n-- > 0);
                full = full && there;
                if (blocks > 32) e[0] = f3_add(f3_add(f3_add(e[0], e[1]), f3_add(e[2], e[3])), e[4]);
                s = f3_add(s, e[0]);
            }
            __syncwarp();
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) s = f3_add(s, f3_shfl(s, d));
            full = __all_sync(0xffffffffu, full);
            if (lane == 0) {
                M.sum[warp]  = s;
                M.full[warp] = full;
            }
        }
        __syncthreads();
        if (warp == 0) {
            if (!START || lane == 0) {
                CgScalars c = M.cg;
                Outcome o   = decided(c);
                const bool full = M.full[0] && M.full[1] && (START || (M.full[2] && M.full[3]));
                if (!full) o.code = kFailed;
                if (!START && lane < kCopies) outcome_put(outcome + lane, o, tag);
                __syncwarp(START ? 1u : 0xffffffffu);
                if (lane == 0) M.cg = c, M.out = o;
            }
            if (START) {
                __syncwarp();
                if (lane < kCopies) outcome_put(outcome + lane, M.out, tag);
            }
        }
    }
    __syncthreads();
    tag++;
    return M.out;
}

// The cluster's barrier, with its blocks' writes before it visible after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// v to the same place in the shared memory of block `rank` of the cluster.
__device__ __forceinline__ void cluster_put(float * p, int rank, float v) {
    unsigned at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(unsigned(__cvta_generic_to_shared(p))), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_put(double * p, int rank, double v) {
    unsigned at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(unsigned(__cvta_generic_to_shared(p))), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
// The meeting of a cluster: every block has all partials in its own shared memory and
// decides for itself, in the same order on the same values.
template<bool START, int WARPS, class Decide>
__device__ __forceinline__ Outcome meet_cluster(const F3 & v, int active, unsigned & tag, ClusterSmem<WARPS> & M,
                                                Decide decided) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, blocks = gridDim.x;
    const int k = lane >> 3, w = lane & 7;
    if (w == 0) M.part[warp][k] = v;
    __syncthreads();
    F3(&all)[kCluster][kSums] = M.all[tag & 1u];
    if (warp == 0) {
        F3 part{0.f, 0.f, 0.f};
        for (int j = w; j < active; j += 8) part = f3_add(part, M.part[j][k]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) part = f3_add(part, f3_shfl(part, o));
        for (int r = w; r < blocks; r += 8) {
            if constexpr (START) {
                if (k < 2) cluster_put(&M.all_start[blockIdx.x][k], r, f3_double(part));
            } else {
                F3 & to = all[blockIdx.x][k];
                cluster_put(&to.h, r, part.h);
                cluster_put(&to.m, r, part.m);
                cluster_put(&to.l, r, part.l);
            }
        }
    }
    cluster_sync();
    if (warp == 0) {
        if constexpr (START) {
            double s = 0;
            for (int r = w; r < blocks; r += 8) s += M.all_start[r][k & 1];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (w == 0 && k < 2) M.start[k] = s;
        } else {
            F3 s{0.f, 0.f, 0.f};
            for (int r = w; r < blocks; r += 8) s = f3_add(s, all[r][k]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s = f3_add(s, f3_shfl(s, o));
            if (w == 0) M.sum[k] = s;
        }
        __syncwarp();
        if (!START || lane == 0) {
            CgScalars c     = M.cg;
            const Outcome o = decided(c);
            __syncwarp(START ? 1u : 0xffffffffu);
            if (lane == 0) M.cg = c, M.out = o;
        }
    }
    __syncthreads();
    tag++;
    return M.out;
}

// A warp's wait for the flags of a brick's active neighbours (tab); false when they did
// not come in time.
__device__ __forceinline__ bool wait_neighbours(const unsigned * flags, const int * tab, int polls, unsigned tag) {
    const int lane = threadIdx.x & 31;
    const int b    = lane < 27 ? tab[lane] : -1;
    bool there     = b < 0;
    int n          = polls;
    while (!there) {
        there = ld_relaxed(flags + b) == tag;
        if (n-- <= 0) break;
    }
    fence_gpu();
    return __all_sync(0xffffffffu, there);
}

// The state to host memory (pinned), but for `failed`, which any block sets there.
__device__ __forceinline__ void to_host(const CgState * cg, CgState * host) {
    if (!host) return;
    host->bb      = cg->bb;
    host->rr      = cg->rr;
    host->rr0     = cg->rr0;
    host->iter    = cg->iter;
    host->done    = cg->done;
    host->start   = cg->start;
    host->nv      = cg->nv;
    host->nbricks = cg->nbricks;
}

template<int DIM, bool CLUSTER>
using MeetSmemOf = std::conditional_t<CLUSTER, ClusterSmem<WarpBrick<DIM>::WARPS>, MeetSmem<WarpBrick<DIM>::WARPS>>;
// Dynamic shared memory of the tiles: a cluster uses the larger groups alone.
template<int DIM, bool CLUSTER>
constexpr size_t kSolveTiles = CLUSTER ? sizeof(float) * WarpBrick<DIM>::T::TILE * (WarpBrick<DIM>::WARPS / WarpBrick<DIM>::WMAX)
                                       : WarpBrick<DIM>::kTileBytes;
template<int DIM, bool CLUSTER>
constexpr size_t kSolveSmem = WarpBrick<DIM>::kSmem - WarpBrick<DIM>::kTileBytes + kSolveTiles<DIM, CLUSTER>;

// Groups of W warps own the bricks c + P (g + COUNT k): the solve's loop.  CLUSTER: the
// grid is one cluster, whose barrier and shared memory take the place of the flags and the
// slots.
template<int DIM, int W, bool CLUSTER>
__device__ __forceinline__ void solve(const Lattice & L, const int * __restrict__ blist, int nb, int P,
                                      const unsigned char * __restrict__ bflag, const NodeArrays & N, const Stencil & S,
                                      CgState * cg, const CgStart & from, ulonglong2 * slots, unsigned * flags,
                                      CgPhases * phases, CgState * host, MeetSmemOf<DIM, CLUSTER> & M) {
    using B  = WarpBrick<DIM>;
    using G  = typename B::G;
    using Gr = Group<DIM, W>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int grp = Gr::index(), gl = Gr::lane();
    const bool idle  = grp >= Gr::COUNT;
    float * tile     = reinterpret_cast<float *>(smem) + B::T::TILE * grp;
    int * tab        = reinterpret_cast<int *>(smem + kSolveTiles<DIM, CLUSTER>) + 27 * (B::TABS + 1) * grp;
    unsigned * seg   = reinterpret_cast<unsigned *>(smem + kSolveTiles<DIM, CLUSTER> + B::kTabBytes);
    const int bfirst = idle ? nb : int(blockIdx.x) + P * grp, bstep = P * Gr::COUNT;
    constexpr int Q  = G::BN / 4 / Gr::NT;  // float4 per thread of a brick
    fill_segments<DIM>(seg);
    for (int k = 0, bi = bfirst; k < B::TABS && bi < nb; k++, bi += bstep)
        fill_neighbours<DIM>(L, bflag, blist[bi], gl, tab + 27 * k);
    float scale = 1.f;
    if (!from.own) {
        scale = sum_scale(cg->bb);
        if (threadIdx.x == 0) M.cg = scalars_of(cg->rr, cg->threshold, cg->max_iter, scale, from.qscale);
    }
    __syncthreads();
    const int active = W * min(Gr::COUNT, (nb - int(blockIdx.x) + P - 1) / P);  // warps with bricks

    Outcome o{0.f, 0.f, kGoOn};
    bool first = true, ok = true;
    unsigned tag = cg->tick + 1;
    CgPhases spent{0, 0, 0};
    unsigned long long mark = phases ? global_ns() : 0;
    auto lap = [&](unsigned long long & sum) {
        if (phases) {
            const unsigned long long now = global_ns();
            sum += now - mark;
            mark = now;
        }
    };
    // u is there: the bricks' flags
    auto publish = [&]() {
        if constexpr (CLUSTER) cluster_sync();
        else if (!idle) {
            Gr::sync();
            if (gl == 0) {
                fence_gpu();
                for (int bi = bfirst; bi < nb; bi += bstep) st_relaxed(flags + blist[bi], tag);
            }
        }
    };
    auto product = [&](auto start, FF (&part)[kSums]) {
        constexpr bool START = decltype(start)::value;
        for (int k = 0, bi = bfirst; bi < nb; bi += bstep, k++) {
            const int b = blist[bi];
            int * t     = tab + 27 * min(k, B::TABS);
            if (k >= B::TABS) {
                Gr::sync();
                fill_neighbours<DIM>(L, bflag, b, gl, t);
                __syncwarp();
            }
            if (!CLUSTER && gl < 32 && !wait_neighbours(flags, t, from.polls, tag)) ok = false;
            Gr::sync();  // also past the last brick's reads of the tile
            tile_copy<DIM, W>(seg, t, N.u, tile);
            const long long base = (long long) b * G::BN;
            float q[Gr::NOUT];
            // with few bricks the row's own operands are loaded under the tile's copy
            constexpr bool FEW  = W == B::WMAX;
            constexpr int AHEAD = FEW ? Gr::NOUT / 4 : 1;
            float4 d_[AHEAD], a_[AHEAD], r_[AHEAD];
            unsigned f_[AHEAD];
            auto operands = [&](int i, int at) {  // (x and b for the start)
                const long long s = base + Gr::row(i / Gr::NX) + i % Gr::NX;
                d_[at] = ld4(START ? N.x : N.d, s), a_[at] = ld4(N.ahat, s), r_[at] = ld4(START ? N.D : N.r, s);
                f_[at] = *reinterpret_cast<const unsigned *>(N.flag + s);
            };
            if constexpr (FEW) {
#pragma unroll
                for (int i = 0; i < Gr::NOUT; i += 4) operands(i, i / 4);
            }
            tile_wait<DIM, W>();
            group_stencil<DIM, W>(tile, S, q);
#pragma unroll
            for (int i = 0; i < Gr::NOUT; i += 4) {
                const long long s = base + Gr::row(i / Gr::NX) + i % Gr::NX;
                const int at      = FEW ? i / 4 : 0;
                if constexpr (!FEW) operands(i, 0);
                const unsigned fl = f_[at];
                const float4 d = d_[at], a = a_[at], r = r_[at];
                float p[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    p[j] = (fl >> (8 * j)) & 0xffu ? fmaf(comp(a, j), comp(d, j), q[i + j]) : comp(d, j);
                if constexpr (START) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        p[j] = comp(r, j) - p[j];
                        ff_add_prod(part[0], p[j], p[j]);
                        ff_add_prod(part[1], comp(r, j), comp(r, j));
                    }
                    st4(N.r, s, make_float4(p[0], p[1], p[2], p[3]));
                    st4(N.d, s, make_float4(p[0], p[1], p[2], p[3]));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        ff_add_prod(part[0], comp(d, j), p[j]);
                        ff_add_prod(part[1], comp(r, j), p[j]);
                        ff_add_prod(part[2], p[j], p[j] * from.qscale);
                        ff_add_prod(part[3], comp(r, j), comp(r, j));
                    }
                    st4(N.q, s, make_float4(p[0], p[1], p[2], p[3]));
                }
            }
        }
    };
    auto meeting = [&](auto start, const F3 & v, auto decided) {
        constexpr bool START = decltype(start)::value;
        if constexpr (CLUSTER) return meet_cluster<START, B::WARPS>(v, active, tag, M, decided);
        else return meet<START, B::WARPS>(v, slots, gridDim.x, P, active, from.polls, tag, M, decided);
    };
    if (from.own) {
        for (int bi = bfirst; bi < nb; bi += bstep) {
            const long long base = (long long) blist[bi] * G::BN + 4 * gl;
#pragma unroll 2
            for (int k = 0; k < Q; k++) {
                const long long s = base + 4 * Gr::NT * k;
                st4(N.u, s, mul4(ld4(N.V, s), ld4(N.x, s)));
            }
        }
        publish();
        FF part[kSums] = {};
        product(std::true_type{}, part);
        o = meeting(std::true_type{}, warp_sum4(part, 1.f), [&](CgScalars & c) {
            return decide_start(blockIdx.x == 0 ? cg : nullptr, c, M.start[0], M.start[1], M.nv, from);
        });
        scale = o.alpha;
        mark  = phases ? global_ns() : 0;
    }
    const bool started = o.code == kGoOn;
    while (o.code == kGoOn) {
        for (int bi = bfirst; bi < nb; bi += bstep) {
            const long long base = (long long) blist[bi] * G::BN + 4 * gl;
#pragma unroll 2
            for (int k = 0; k < Q; k++) {
                const long long s = base + 4 * Gr::NT * k;
                const float4 v    = ld4(N.V, s);
                float4 d          = ld4(N.d, s);
                if (!first) {
                    const float4 q = ld4(N.q, s), x = ld4(N.x, s);
                    float4 r = ld4(N.r, s);
                    r        = fma4(-o.alpha, q, r);
                    st4(N.x, s, fma4(o.alpha, d, x));
                    st4(N.r, s, r);
                    d = fma4(o.beta, d, r);
                    st4(N.d, s, d);
                }
                st4(N.u, s, mul4(v, d));
            }
        }
        if constexpr (CLUSTER) lap(spent.step);
        publish();
        if constexpr (!CLUSTER) lap(spent.step);

        FF part[kSums] = {};
        product(std::false_type{}, part);
        lap(spent.product);
        o = meeting(std::false_type{}, warp_sum4(part, scale), [&](CgScalars & c) {
            const F3 sum[kSums] = {M.sum[0], M.sum[1], M.sum[2], M.sum[3]};
            return decide(c, sum, 0.f, false, from.timed);
        });
        first = false;
        if (o.code == kMeasure) {
#pragma unroll
            for (int k = 0; k < kSums; k++) part[k] = FF{0.f, 0.f};
            for (int bi = bfirst; bi < nb; bi += bstep) {
                const long long base = (long long) blist[bi] * G::BN + 4 * gl;
                for (int k = 0; k < Q; k++) {
                    const long long s = base + 4 * Gr::NT * k;
                    const float4 r    = fma4(-o.alpha, ld4(N.q, s), ld4(N.r, s));
#pragma unroll
                    for (int j = 0; j < 4; j++) ff_add_prod(part[0], comp(r, j), comp(r, j));
                }
            }
            const float alpha = o.alpha;
            o = meeting(std::false_type{}, warp_sum4(part, scale), [&](CgScalars & c) {
                const F3 sum[kSums] = {M.sum[0], M.sum[1], M.sum[2], M.sum[3]};
                return decide(c, sum, alpha, true, false);
            });
        }
        if (o.code == kGoOn && o.shift) scale *= pow2(o.shift);
        lap(spent.meeting);
    }
    if (!__syncthreads_and(ok)) o.code = kFailed;
    // the last step of x (none after a start that is the solution already, or a cap of no
    // iterations); a breakdown, a start that is not a number and b = 0 leave x = 0
    const bool zero = o.code >= 3;
    if (o.code != kFailed && (started || zero))
        for (int bi = bfirst; bi < nb; bi += bstep) {
            const long long base = (long long) blist[bi] * G::BN + 4 * gl;
#pragma unroll
            for (int k = 0; k < Q; k++) {
                const long long s = base + 4 * Gr::NT * k;
                st4(N.x, s, zero ? make_float4(0.f, 0.f, 0.f, 0.f) : fma4(o.alpha, ld4(N.d, s), ld4(N.x, s)));
            }
        }
    if (threadIdx.x == 0) {
        if (blockIdx.x == 0) {
            if (started) {
                cg->rr      = f3_double(M.cg.rr_next) / double(scale);
                cg->iter    = M.cg.it;
                if (o.code != kFailed) cg->done = int(o.code);
            }
            cg->tick = tag;
            if (phases) *phases = spent;
            to_host(cg, host);
        }
        if (o.code == kFailed) {
            atomicExch(&cg->failed, 1);
            if (host) host->failed = 1;
        }
    }
}

// Few bricks: the larger groups take all bricks of a block at once (3D: at most three,
// where their reads, 2,160 shared-memory wavefronts a brick against 1,250, still cost no
// more than the longer chain of the smaller groups: an iteration with the larger and the
// smaller takes 7.9 and 8.8 us at 125 bricks, 10.2 and 11.3 at 216, 12.4 and 12.4 at 343,
// 14.1 and 12.7 at 528).
template<int DIM> __device__ __forceinline__ bool few_bricks(int nb, int blocks) {
    return nb <= blocks * (DIM == 3 ? 3 : Group<DIM, WarpBrick<DIM>::WMAX>::COUNT);
}

}  // namespace

template<int DIM, bool CLUSTER>
__global__ void __launch_bounds__(WarpBrick<DIM>::NT, 1)
    k_cg_solve(Lattice L, const int * __restrict__ blist, const int * __restrict__ bcount,
               const unsigned char * __restrict__ bflag, NodeArrays N, Stencil S, CgState * cg, CgStart from,
               ulonglong2 * slots, unsigned * flags, CgPhases * phases, CgState * host) {
    if constexpr (CLUSTER) pdl_wait_and_release();
    using B = WarpBrick<DIM>;
    constexpr int Q = B::G::BN / 4;
    __shared__ MeetSmemOf<DIM, CLUSTER> M;
    const int nb   = *bcount;
    const int done = from.own ? 0 : cg->done;
    if (CLUSTER && threadIdx.x == 0) M.nv = *from.nv;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        M.nv        = *from.nv;
        cg->nv      = M.nv;
        cg->nbricks = nb;
        if (from.own && nb == 0) {
            CgScalars none;
            decide_start(cg, none, 0.0, 0.0, 0, from);
        }
        if (done || nb == 0) to_host(cg, host);
    }
    if (done) {
        // no solve: a zero right-hand side (4) or a start that is not a number (3) leaves x = 0
        if (done >= 3)
            for (long long e = blockIdx.x * (long long) B::NT + threadIdx.x; e < (long long) nb * Q;
                 e += (long long) gridDim.x * B::NT)
                st4(N.x, (long long) blist[e / Q] * B::G::BN + 4 * (e % Q), make_float4(0.f, 0.f, 0.f, 0.f));
        return;
    }
    if constexpr (CLUSTER) {
        if (nb == 0) return;
        solve<DIM, B::WMAX, true>(L, blist, nb, int(gridDim.x), bflag, N, S, cg, from, slots, flags, phases, host, M);
    } else {
        const int P = min(int(gridDim.x), nb);
        if (int(blockIdx.x) >= P) return;
        if (few_bricks<DIM>(nb, gridDim.x))
            solve<DIM, B::WMAX, false>(L, blist, nb, P, bflag, N, S, cg, from, slots, flags, phases, host, M);
        else solve<DIM, B::WMIN, false>(L, blist, nb, P, bflag, N, S, cg, from, slots, flags, phases, host, M);
    }
}

// Row-stencil passes outside the iteration, the bricks strided over the warps of a
// resident grid:
//   kRowsAhat:  alpha_hat = max(-sum_J alpha_IJ, alpha0) from src = V
//               (calculateCoef, VirtualParticle.cpp:149-169).
//   kRowsResid: r = b - A x from src = V x: r (and d when non-null) written,
//               |r|^2 and |b|^2 summed (deterministic) into sums[0..1].
//   kRowsDiag:  the diagonal -sum_J alpha_IJ itself (0 on inactive nodes) into N.ahat and
//               its maximum, as the bits of a non-negative float, into *top.
enum { kRowsAhat = 0, kRowsResid = 1, kRowsDiag = 2 };
template<int DIM, int OP, int W>
__device__ __forceinline__ void rows_of_bricks(const Lattice & L, float alpha0, const int * __restrict__ blist, int nb,
                                               const unsigned char * __restrict__ bflag, const NodeArrays & N,
                                               const Stencil & S, const float * __restrict__ src,
                                               const float * __restrict__ xin, float * __restrict__ r_out,
                                               float * __restrict__ d_out, FF & rr, FF & bb) {
    using B  = WarpBrick<DIM>;
    using Gr = Group<DIM, W>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int grp = Gr::index();
    if (grp >= Gr::COUNT) return;
    float * tile   = reinterpret_cast<float *>(smem) + B::T::TILE * grp;
    int * tab      = reinterpret_cast<int *>(smem + B::kTileBytes) + 27 * (B::TABS + 1) * grp;
    unsigned * seg = reinterpret_cast<unsigned *>(smem + B::kTileBytes + B::kTabBytes);
    for (int bi = int(blockIdx.x) + int(gridDim.x) * grp; bi < nb; bi += int(gridDim.x) * Gr::COUNT) {
        const int b = blist[bi];
        Gr::sync();  // the last brick's reads of the tile and the table
        fill_neighbours<DIM>(L, bflag, b, Gr::lane(), tab);
        Gr::sync();
        tile_copy<DIM, W>(seg, tab, src, tile);
        tile_wait<DIM, W>();
        float q[Gr::NOUT];
        group_stencil<DIM, W>(tile, S, q);
#pragma unroll
        for (int i = 0; i < Gr::NOUT; i += 4) {
            const long long s = (long long) b * B::G::BN + Gr::row(i / Gr::NX) + i % Gr::NX;
            const unsigned fl = *reinterpret_cast<const unsigned *>(N.flag + s);
            float o[4];
            if (OP == kRowsAhat) {
#pragma unroll
                for (int j = 0; j < 4; j++) o[j] = (fl >> (8 * j)) & 0xffu ? fmaxf(-q[i + j], alpha0) : 1.f;
                st4(N.ahat, s, make_float4(o[0], o[1], o[2], o[3]));
            } else if (OP == kRowsDiag) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    o[j]  = (fl >> (8 * j)) & 0xffu ? fmaxf(-q[i + j], 0.f) : 0.f;
                    rr.hi = fmaxf(rr.hi, o[j]);
                }
                st4(N.ahat, s, make_float4(o[0], o[1], o[2], o[3]));
            } else {
                const float4 xv = ld4(xin, s), a = ld4(N.ahat, s), bv = ld4(N.D, s);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    o[j] = comp(bv, j) - ((fl >> (8 * j)) & 0xffu ? fmaf(comp(a, j), comp(xv, j), q[i + j]) : comp(xv, j));
                    ff_add_prod(rr, o[j], o[j]);
                    ff_add_prod(bb, comp(bv, j), comp(bv, j));
                }
                st4(r_out, s, make_float4(o[0], o[1], o[2], o[3]));
                if (d_out) st4(d_out, s, make_float4(o[0], o[1], o[2], o[3]));
            }
        }
    }
}
template<int DIM, int OP>
__global__ void __launch_bounds__(WarpBrick<DIM>::NT, 1)
    k_rows_tiled(Lattice L, float alpha0, const int * __restrict__ blist, const int * __restrict__ bcount,
                 const unsigned char * __restrict__ bflag, NodeArrays N, Stencil S, const float * __restrict__ src,
                 const float * __restrict__ xin, float * __restrict__ r_out, float * __restrict__ d_out,
                 double * __restrict__ sums, double * __restrict__ partials, unsigned int * __restrict__ ticket,
                 unsigned int * __restrict__ top) {
    using B = WarpBrick<DIM>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[B::WARPS + 1];
    __shared__ int last;
    fill_segments<DIM>(reinterpret_cast<unsigned *>(smem + B::kTileBytes + B::kTabBytes));
    __syncthreads();
    pdl_wait_and_release();
    const int nb = *bcount;
    FF rr{0.f, 0.f}, bb{0.f, 0.f};
    if (few_bricks<DIM>(nb, gridDim.x))
        rows_of_bricks<DIM, OP, B::WMAX>(L, alpha0, blist, nb, bflag, N, S, src, xin, r_out, d_out, rr, bb);
    else rows_of_bricks<DIM, OP, B::WMIN>(L, alpha0, blist, nb, bflag, N, S, src, xin, r_out, d_out, rr, bb);
    if (OP == kRowsDiag) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(rr.hi));
        if ((threadIdx.x & 31) == 0) atomicMax(top, m);
    }
    if (OP == kRowsResid) {
        double part[2] = {block_sum_ff<B::NT>(rr, red), 0.0};
        part[1]        = block_sum_ff<B::NT>(bb, red);
        double tot[2];
        if (grid_reduce<B::NT, 2>(part, partials, ticket, tot, red, &last) && threadIdx.x == 0) {
            sums[0] = tot[0];
            sums[1] = tot[1];
        }
    }
}

// alpha0 calibration (VirtualParticle::setAlpha, VirtualParticle.cpp:64-73): the maximum
// over active nodes of -sum_J alpha_IJ in FP64, among the nodes whose FP32 diagonal
// (kRowsDiag) is within 1e-4 of the largest one.  The FP32 value is a sum of at most 250
// terms of one sign, so it is within 250 x 2^-24 = 1.5e-5 of the FP64 value and the node
// of the FP64 maximum is one of them.  (All nodes in FP64: 250 multiply-adds a node on a
// pipe of two per SM and clock, 2.26 ms at 2.25M nodes; this pass with the FP32 one
// takes 0.06.)
template<int DIM>
__global__ void __launch_bounds__(256)
    k_diag_max_f64(Lattice L, const int * __restrict__ blist, const int * __restrict__ bcount,
                   const unsigned char * __restrict__ bflag, NodeArrays N, StencilD S,
                   const unsigned int * __restrict__ top, unsigned long long * __restrict__ out_bits) {
    pdl_wait_and_release();
    using G           = BrickGeom<DIM>;
    constexpr int ZR  = DIM == 3 ? 3 : 0;
    const float bound = __uint_as_float(*top) * (1.f - 1e-4f);
    const long long n = (long long) *bcount * G::BN;
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < n; e += (long long) gridDim.x * 256) {
        const int b = blist[e / G::BN], l = int(e % G::BN);
        const long long s = (long long) b * G::BN + l;
        if (!N.flag[s] || N.ahat[s] < bound) continue;
        const int3 bc = brick_coords(L, b);
        const int x = bc.x * G::BX + l % G::BX, y = bc.y * G::BY + (l / G::BX) % G::BY,
                  z = DIM == 3 ? bc.z * G::BZ + l / (G::BX * G::BY) : 0;
        double acc = 0;
        for (int dz = -ZR; dz <= ZR; dz++)
            for (int dy = -3; dy <= 3; dy++)
                for (int dx = -3; dx <= 3; dx++) {
                    const int r2 = dx * dx + dy * dy + dz * dz, X = x + dx, Y = y + dy, Z = z + dz;
                    if (r2 == 0 || r2 >= 16 || X < 0 || X >= L.nx || Y < 0 || Y >= L.ny || Z < 0 || Z >= L.nz) continue;
                    if (!bflag[brick_of(L, X, Y, Z, G::BX, G::BY, G::BZ)]) continue;
                    acc += S.c[r2] * double(N.V[node_slot<DIM>(L, X, Y, Z)]);
                }
        // positive doubles order like their bit patterns; the diagonal is >= 0
        if (-acc >= 0) atomicMax(out_bits, (unsigned long long) __double_as_longlong(-acc));
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
template<int DIM> int cg_solve_prepare() {
    const int bytes = int(WarpBrick<DIM>::kSmem);
    auto set = [bytes](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
    };
    return set(k_cg_solve<DIM, false>) && set(k_rows_tiled<DIM, kRowsAhat>) && set(k_rows_tiled<DIM, kRowsResid>) &&
                   set(k_rows_tiled<DIM, kRowsDiag>)
               ? 0
               : -1;
}
template<int DIM>
void launch_ahat(const Lattice & L, const Phys & P, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                 int blocks, cudaStream_t st) {
    using W = WarpBrick<DIM>;
    launch_pdl(k_rows_tiled<DIM, kRowsAhat>, blocks, W::NT, W::kSmem, st, L, P.alpha0, B.list, B.count, B.flag, N, S,
               N.V, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
}
template<int DIM>
void launch_diag_max_f64(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                         const StencilD & SD, unsigned int * top, unsigned long long * out_bits, int blocks, int grid,
                         cudaStream_t st) {
    using W = WarpBrick<DIM>;
    cudaMemsetAsync(top, 0, sizeof(unsigned int), st);
    cudaMemsetAsync(out_bits, 0, sizeof(unsigned long long), st);
    launch_pdl(k_rows_tiled<DIM, kRowsDiag>, blocks, W::NT, W::kSmem, st, L, 0.f, B.list, B.count, B.flag, N, S, N.V,
               nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, top);
    launch_pdl(k_diag_max_f64<DIM>, grid, 256, 0, st, L, B.list, B.count, B.flag, N, SD, top, out_bits);
}
template<int DIM>
void launch_rows_residual(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S,
                          const float * x, float * r, float * d, double * sums, CgState * cg, double * partials,
                          int blocks, cudaStream_t st) {
    using W = WarpBrick<DIM>;
    launch_pdl(k_rows_tiled<DIM, kRowsResid>, blocks, W::NT, W::kSmem, st, L, 0.f, B.list, B.count, B.flag, N, S, N.u, x,
               r, d, sums, partials, &cg->ticket[0], nullptr);
}
template<int DIM> int cg_cluster_blocks() {
    auto kernel = k_cg_solve<DIM, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSolveSmem<DIM, true>)) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (int blocks = kCluster; blocks >= 8; blocks /= 2) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at[1];
        cfg.gridDim          = blocks;
        cfg.blockDim         = WarpBrick<DIM>::NT;
        cfg.dynamicSmemBytes = kSolveSmem<DIM, true>;
        at[0].id               = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs    = at;
        cfg.numAttrs = 1;
        int n        = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) return blocks;
        cudaGetLastError();
    }
    return 0;
}
template<int DIM>
int launch_cg_solve(const Lattice & L, const BrickArrays & B, const NodeArrays & N, const Stencil & S, CgState * cg,
                    const CgStart & from, ulonglong2 * slots, unsigned * flags, int blocks, int cluster,
                    CgPhases * phases, CgState * host, cudaStream_t st) {
    using W = WarpBrick<DIM>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = cluster ? cluster : blocks;
    cfg.blockDim         = W::NT;
    cfg.dynamicSmemBytes = cluster ? kSolveSmem<DIM, true> : W::kSmem;
    cfg.stream           = st;
    cudaLaunchAttribute at[2];
    if (cluster) {
        at[0].id               = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        at[1].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
    } else {
        at[0].id              = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs    = at;
    cfg.numAttrs = cluster ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, cluster ? k_cg_solve<DIM, true> : k_cg_solve<DIM, false>, L, (const int *) B.list,
                              (const int *) B.count, (const unsigned char *) B.flag, N, S, cg, from, slots, flags, phases,
                              host) == cudaSuccess
               ? 0
               : -1;
}

#define SWC_INST(D)                                                                                                    \
    template int cg_solve_prepare<D>();                                                                                \
    template void launch_ahat<D>(const Lattice &, const Phys &, const BrickArrays &, const NodeArrays &,               \
                                 const Stencil &, int, cudaStream_t);                                                  \
    template void launch_rows_residual<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,   \
                                          const float *, float *, float *, double *, CgState *, double *, int,         \
                                          cudaStream_t);                                                               \
    template void launch_diag_max_f64<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,    \
                                         const StencilD &, unsigned int *, unsigned long long *, int, int,             \
                                         cudaStream_t);                                                                \
    template int cg_cluster_blocks<D>();                                                                              \
    template int launch_cg_solve<D>(const Lattice &, const BrickArrays &, const NodeArrays &, const Stencil &,         \
                                    CgState *, const CgStart &, ulonglong2 *, unsigned *, int, int, CgPhases *,        \
                                    CgState *, cudaStream_t);
SWC_INST(2)
SWC_INST(3)
#undef SWC_INST

}  // namespace swc
