// swc_stencil.cuh -- the radial virtual-Laplacian stencil of one brick computed by a
// group of W warps from a halo tile that the group copies into shared memory.
//
// 3D, W = 2 is the form for many bricks, between FP32 issue and shared-memory reads:
// rows at the same |dy| share their coefficients, so per z-plane the rows y - j and
// y + j are added first and the x-convolution runs once per (j, |dz|), the nodes at
// +-dx added first too; a thread computes four nodes of two rows next to each other in
// z, whose 8 planes serve both: 8 outputs cost 52 row reads of 12 floats (156 LDS.128,
// 19.5 per output, against 22.5 of one row of 8 per thread) and 1,130 FP32
// instructions.  14 tiles of 15.7 KB fill an SM's shared memory, so two warps per tile
// are 28 warps per SM: with one warp per tile (eight nodes of two rows per lane, 13
// LDS.128 per output) 14 warps left 64% of the issue slots empty on the latency of the
// tile copy and of the row reads: 46 us a product against 38 at 2.25M nodes.
// 3D, W = 4 (2D: 2) is the form for few bricks, where the chain of one group's
// instructions per brick is what a product takes: half a row of 4 per thread, rows
// summed by class of dy^2 + dz^2 (stencil_row_t).  2D, W = 1: 8 nodes of a row.
// Lanes 0-7 of a quarter-warp read 8 consecutive rows of pitch 20 (3D) or 28 (2D)
// floats: all 32 banks once.
#pragma once

#include "swc_tiles.cuh"

namespace swc {

template<int DIM> struct WarpBrick {
    using G = BrickGeom<DIM>;
    using T = SpmvTile<DIM>;
    static constexpr int SEGX  = T::TX / 4;
    static constexpr int NSEG  = SEGX * T::TY * T::TZ; // 16-byte segments of a halo tile
    static constexpr int WMIN  = DIM == 3 ? 2 : 1;     // warps per brick where bricks are many
    static constexpr int WARPS = DIM == 3 ? 28 : 16;   // warps of a block
    static constexpr int NT    = 32 * WARPS;
    static constexpr int WMAX  = DIM == 3 ? 4 : 2;     // warps per brick where bricks are few
    static constexpr int TABS  = 4;                    // bricks per group whose neighbour tables are kept
    // dynamic shared memory: tiles, neighbour tables (one more for bricks past TABS), segment table
    static constexpr int TILES = WARPS / WMIN;         // 3D: 14 tiles of 15.7 KB fill the SM
    static constexpr size_t kTileBytes = sizeof(float) * T::TILE * TILES;
    static constexpr size_t kTabBytes  = sizeof(int) * 27 * (TABS + 1) * TILES;
    static constexpr size_t kSmem      = kTileBytes + kTabBytes + sizeof(unsigned) * NSEG;
};

// A thread's place among the groups of W warps of its block.
template<int DIM, int W> struct Group {
    static constexpr int COUNT = WarpBrick<DIM>::WARPS / W;  // groups of a block (left-over warps hold none)
    static constexpr int NT    = 32 * W;
    static constexpr int NOUT  = BrickGeom<DIM>::BN / NT;    // outputs per thread
    static constexpr int NX    = DIM == 3 ? 4 : NOUT;        // of one row
    static __device__ __forceinline__ int index() { return int(threadIdx.x) / NT; }
    static __device__ __forceinline__ int lane() { return int(threadIdx.x) % NT; }
    static __device__ __forceinline__ void sync() {
        if constexpr (W == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(index() + 1), "r"(NT) : "memory");
    }
    // node offset (in the brick) of the thread's outputs: NX nodes of row k from there
    static __device__ __forceinline__ int row(int k) {
        const int l = lane();
        if constexpr (DIM == 3) {
            // y = l % 8, half row, then z (W = 4) or a pair of z (W = 2)
            const int z = W == 2 ? 2 * (l >> 4) + k : l >> 4;
            return 8 * ((l & 7) + 8 * z) + 4 * ((l >> 3) & 1);
        } else return 16 * (l & 15) + NX * (l >> 4);
    }
};

// Copy table of a halo tile, the same for every brick: segment -> neighbour index
// (27 codes), offset in that brick and (in 16-byte units) in the tile.
template<int DIM> __device__ __forceinline__ void fill_segments(unsigned * seg) {
    using W = WarpBrick<DIM>;
    using G = typename W::G;
    using T = typename W::T;
    for (int t = threadIdx.x; t < W::NSEG; t += W::NT) {
        const int sx = t % W::SEGX, row = t / W::SEGX, ty = row % T::TY, tz = row / T::TY;
        const int tx = 4 * sx;
        const int oi = (tx - T::HX + G::BX) / G::BX - 1, oj = (ty - T::HY + G::BY) / G::BY - 1;
        const int ok = DIM == 3 ? (tz - T::HZ + G::BZ) / G::BZ - 1 : 0;
        const int lx = tx - T::HX - G::BX * oi, ly = ty - T::HY - G::BY * oj;
        const int lz = DIM == 3 ? tz - T::HZ - G::BZ * ok : 0;
        const unsigned code = unsigned((ok + 1) * 9 + (oj + 1) * 3 + (oi + 1));
        seg[t] = unsigned((tx + T::PX * row) / 4) << 16 | code << 9 | unsigned(lx + G::BX * (ly + G::BY * lz));
    }
}

// Neighbour table of brick b (ids of the active ones of the 27 bricks, else -1), by the
// group's first lanes; the caller synchronises the group.
template<int DIM>
__device__ __forceinline__ void fill_neighbours(const Lattice & L, const unsigned char * __restrict__ bflag, int b, int t,
                                                int * tab) {
    if (t < 27) {
        const int3 bc = brick_coords(L, b);
        const int i = t % 3 - 1, j = (t / 3) % 3 - 1, k = t / 9 - 1;
        const int x = bc.x + i, y = bc.y + j, z = bc.z + k;
        int id = -1;
        if (x >= 0 && x < L.bnx && y >= 0 && y < L.bny && z >= 0 && z < L.bnz && (DIM == 3 || k == 0)) {
            const int nb = x + L.bnx * (y + L.bny * z);
            if (bflag[nb]) id = nb;
        }
        tab[t] = id;
    }
}

// The group's asynchronous copy of the halo tile of `src` (zero outside the active
// bricks), and the wait for it.
template<int DIM, int W>
__device__ __forceinline__ void tile_copy(const unsigned * seg, const int * tab, const float * src, float * tile) {
    using B = WarpBrick<DIM>;
#pragma unroll 5
    for (int t = Group<DIM, W>::lane(); t < B::NSEG; t += 32 * W) {
        const unsigned e = seg[t];
        const int nb     = tab[(e >> 9) & 127u];
        cp_async16(tile + 4 * (e >> 16), src + ((long long) (nb < 0 ? 0 : nb) * B::G::BN + (e & 511u)), nb >= 0);
    }
    cp_async_commit();
}
template<int DIM, int W> __device__ __forceinline__ void tile_wait() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    Group<DIM, W>::sync();
}

// W = 2, 3D: one half of the two rows' planes (plane K at distance 3 - K from the first
// row f and 4 - K from the second s) in 15 stages (K, J = |dy|), each the rows y - J and
// y + J of one plane.
struct PlaneStages {
    static constexpr int COUNT = 15;
    static constexpr int K[COUNT] = {0, 0, 0, 1, 1, 1, 1, 2, 2, 2, 2, 3, 3, 3, 3};
    static constexpr int J[COUNT] = {0, 1, 2, 0, 1, 2, 3, 0, 1, 2, 3, 0, 1, 2, 3};
};
__device__ __forceinline__ void row_load(const float * row, float (&T)[12]) {
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const float4 v = reinterpret_cast<const float4 *>(row)[s];
        T[4 * s] = v.x, T[4 * s + 1] = v.y, T[4 * s + 2] = v.z, T[4 * s + 3] = v.w;
    }
}
template<int PX, int I>
__device__ __forceinline__ void stages(const float * row, int step, const Stencil & S, float (&f)[4], float (&s)[4]) {
    constexpr int K = PlaneStages::K[I], J = PlaneStages::J[I];
    constexpr int M1 = J * J + (3 - K) * (3 - K), M2 = J * J + (4 - K) * (4 - K);
    float T[12];
    row_load(row + K * step - PX * J, T);
    if constexpr (J > 0) {
        float U[12];
        row_load(row + K * step + PX * J, U);
#pragma unroll
        for (int k = 1; k < 11; k++) T[k] += U[k];
    }
    if constexpr (M1 > 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) f[i] = fmaf(S.c[M1], T[i + 4], f[i]);
    }
    if constexpr (M2 < 16) {
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = fmaf(S.c[M2], T[i + 4], s[i]);
    }
    // the nodes at +-dx share their coefficients
#pragma unroll
    for (int dx = 1; dx <= 3; dx++) {
        if (dx * dx + M1 >= 16) continue;  // M1 < M2
        float t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) t[i] = T[i + 4 - dx] + T[i + 4 + dx];
#pragma unroll
        for (int i = 0; i < 4; i++) f[i] = fmaf(S.c[dx * dx + M1], t[i], f[i]);
        if (dx * dx + M2 < 16) {
#pragma unroll
            for (int i = 0; i < 4; i++) s[i] = fmaf(S.c[(dx * dx + M2) & 15], t[i], s[i]);
        }
    }
    if constexpr (I + 1 < PlaneStages::COUNT) stages<PX, I + 1>(row, step, S, f, s);
}

// The stencil sums at the thread's outputs (Group::row).
template<int DIM, int W>
__device__ __forceinline__ void group_stencil(const float * tile, const Stencil & S, float (&out)[Group<DIM, W>::NOUT]) {
    using T     = typename WarpBrick<DIM>::T;
    using Gr    = Group<DIM, W>;
    const int l = Gr::lane();
    if constexpr (DIM == 3 && W == 2) {
        constexpr int PZ = T::PX * T::TY;
        // planes 0..3 from below, then 7..4 from above with the rows' roles exchanged
        const float * row = tile + T::PX * ((l & 7) + T::HY) + PZ * (2 * (l >> 4)) + 4 * ((l >> 3) & 1);
        float f[4], s[4];
#pragma unroll
        for (int i = 0; i < 4; i++) f[i] = s[i] = 0.f;
        int step = PZ;
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            stages<T::PX, 0>(row, step, S, f, s);
            row += 7 * PZ;
            step = -PZ;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float v = f[i];
                f[i]          = s[i];
                s[i]          = v;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = f[i], out[4 + i] = s[i];
    } else if constexpr (DIM == 3) {
        const int o = Gr::row(0), y = (o >> 3) & 7, z = o >> 6;
        stencil_row_t<3, T::PX, T::TY, Gr::NX>(tile + T::PX * ((y + T::HY) + T::TY * (z + T::HZ)) + (o & 7), S, out);
    } else {
        stencil_row_t<2, T::PX, T::TY, Gr::NX>(tile + T::PX * ((l & 15) + T::HY) + Gr::NX * (l >> 4), S, out);
    }
}

}  // namespace swc
