// Particle/grid transfer kernels of one substep:
//   k_p2g          APIC/MLS particle-to-grid scatter
//   k_grid_update  momentum -> velocity, gravity, clamping, collider BCs
//   k_g2p_update   grid-to-particle gather fused with the particle update
//   k_rigid        rigid-body pose integration
#pragma once

#include "grid_build.cuh"
#include "models.cuh"
#include "scene.cuh"
#include "trimesh.cuh"

namespace slosh {

// Coordinates of tile node t (tile edge TW) and the rank + local node id of
// the grid block that owns it (the block itself or one of its +1
// neighbours, in slosh's associated-block order).
template <int D>
__device__ __forceinline__ bool tile_node_owner(const DevScene &s, uint32_t r, int t, uint32_t &rank, uint32_t &local) {
    constexpr int TW = Geo<D>::TW, BW = Geo<D>::BW, NN = Geo<D>::NASSOC - 1;
    int c[D];
    c[0] = t % TW;
    if constexpr (D == 3) {
        c[1] = (t / TW) % TW;
        c[2] = t / (TW * TW);
    } else {
        c[1] = t / TW;
    }
    int oct = 0;
    uint32_t loc = 0, mul = 1;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int o = c[k] >= BW ? 1 : 0;
        oct = oct * 2 + o;
        loc += (uint32_t)(c[k] - o * BW) * mul;
        mul *= BW;
    }
    rank = (oct == 0) ? r : s.bnbh[r * NN + oct - 1];
    local = loc;
    return rank != NONE;
}

// The quadratic B-spline weights of one axis (kernel.slang:62-68), each
// duplicated into both lanes of a pair for the paired FMAs below.
__device__ __forceinline__ void bspline_pairs(float x, float2 (&w)[3]) {
    const float2 f = pair(x), half = pair(0.5f);
    const float2 a = __fadd2_rn(pair(1.5f), make_float2(-f.x, -f.y)), b = __fadd2_rn(f, pair(-1.0f)),
                 c = __fadd2_rn(f, pair(-0.5f));
    w[0] = __fmul2_rn(__fmul2_rn(half, a), a);
    w[1] = __ffma2_rn(make_float2(-b.x, -b.y), b, pair(0.75f));
    w[2] = __fmul2_rn(__fmul2_rn(half, c), c);
}

// Adds one particle to a lane's stencil sums.  The lane owns cell `assoc`
// (its base node, in cells) and one half of the node values: half 0 the
// momentum's (x, y), half 1 (z, mass), (0, mass) in 2D.  p = (x, m), vv = (v,
// C22), cq = C's planes, fdt = the pending force impulse (zeros when none).
// The weights use -d0 / h = -d0 * (1/h) like slosh's p2g (dpt *
// inv_cell_width) with d0 = assoc h - x exact from the sorted cell.  Returns
// false for a particle outside the cell (packed-key aliasing far outside the
// key range).
//
// Paired FP32 arithmetic (sm_100's f32x2 FMA) throughout: a node's value is
// b + sx h C0 + sy h C1 + sz h C2 with C's columns restricted to the half
// (the mass lane's are zero, so it stays m exactly), formed slab by slab and
// row by row; 27 nodes cost 27 weight products, 26 value and 27 sum pairs.
template <int D>
__device__ __forceinline__ bool p2g_particle(const float4 p, const float4 vv, const float4 *cq, const float (&fdt)[3],
                                             const float (&assoc)[D], float h, float inv_h, int half,
                                             float2 (&acc)[Geo<D>::NST]) {
    const float x[3] = {p.x, p.y, p.z};
    float d0[D];
    bool in_cell = true;
    float2 w[D][3];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        d0[k] = fmaf(assoc[k], h, -x[k]);
        const float f = -d0[k] * inv_h;
        in_cell = in_cell && fabsf(f - 1.0f) <= 0.51f;
        bspline_pairs(f, w[k]);
    }
    if (!in_cell) return false;
    float C[D][D];
    mat_from<D>(cq, vv.w, C);
    // columns of C and the base value, restricted to this half
    float2 col[D], b;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        if constexpr (D == 3) col[k] = half ? make_float2(C[2][k], 0.f) : make_float2(C[0][k], C[1][k]);
        else col[k] = half ? make_float2(0.f, 0.f) : make_float2(C[0][k], C[1][k]);
    }
    const float m = p.w;
    if constexpr (D == 3) b = half ? make_float2(vv.z * m + fdt[2], m) : make_float2(vv.x * m + fdt[0], vv.y * m + fdt[1]);
    else b = half ? make_float2(0.f, m) : make_float2(vv.x * m + fdt[0], vv.y * m + fdt[1]);
#pragma unroll
    for (int k = 0; k < D; ++k) b = __ffma2_rn(col[k], pair(d0[k]), b);
    const float2 h2 = pair(h), two = pair(2.0f);
#pragma unroll
    for (int k = 0; k < D; ++k) col[k] = __fmul2_rn(h2, col[k]);
#pragma unroll
    for (int sz = 0; sz < (D == 3 ? 3 : 1); ++sz) {
        float2 bz = b;
        if constexpr (D == 3) bz = sz == 0 ? b : (sz == 1 ? __fadd2_rn(b, col[2]) : __ffma2_rn(two, col[2], b));
#pragma unroll
        for (int sy = 0; sy < 3; ++sy) {
            const float2 by = sy == 0 ? bz : (sy == 1 ? __fadd2_rn(bz, col[1]) : __ffma2_rn(two, col[1], bz));
            float2 wyz = w[1][sy];
            if constexpr (D == 3) wyz = __fmul2_rn(w[1][sy], w[2][sz]);
#pragma unroll
            for (int sx = 0; sx < 3; ++sx) {
                const float2 v = sx == 0 ? by : (sx == 1 ? __fadd2_rn(by, col[0]) : __ffma2_rn(two, col[0], by));
                float2 &a = acc[sx + 3 * (sy + 3 * sz)];
                a = __ffma2_rn(__fmul2_rn(w[0][sx], wyz), v, a);
            }
        }
    }
    return true;
}

// Particle-to-grid over the blocks of the sorted grid.
//
// A block's 64 cells x 2 halves of the node values are 128 items, taken in
// bord's order (cells by decreasing particle count) in 4 passes of 32: the
// lanes of a pass hold 16 cells of similar count, so they finish their
// particle loops together, and a pass whose first (largest) cell is empty
// ends the block.  A lane owns cell c, sums the c's particles -- contiguous
// in the canonical order, staged NBUF deep through cp.async, the two lanes of
// a cell copying half of the particle each -- into its 27 (9) stencil nodes'
// half values in registers.
//
// Why halves: every lane of a cell computes the particle's weights and base
// value again, so fewer lanes a cell means less of that; a whole node value a
// lane (108 sums) does not fit the registers.  With three z slabs a cell
// (nine nodes, whole values) the same sums took a quarter more instructions
// (22.2 warp instructions a particle against 17.9) and the block three slab
// tiles: 161 against 157 us a launch on the 4.74 M-particle sand column, 41
// against 35.5 on the 524,288-particle elastic drop.
//
// Reduction, fixed order (the substep is bit-reproducible): after a pass the
// lanes add their sums into the warp's (block + 2)^D tile, one stencil offset
// at a time; for a fixed offset the lanes of a pass hit distinct node halves,
// so only __syncwarp is needed.  With a block per warp the passes follow each
// other on one tile; where a group of warps shares a block (small scenes) the
// warps' tiles are summed in warp order.  The tile goes to the block's own
// `partial` slot; k_grid_update adds the (up to 2^D) tiles overlapping each
// node in a fixed order.
//
// FORCE: the substep adds the particles' pending force impulses (the first
// substep after they were set); the other substeps compile without them.
// NBUF: particles of a cell staged ahead through cp.async (batches tune it;
// the results do not depend on it).
constexpr int P2G_WARPS = 4;
constexpr uint32_t P2G_PASSES = 4;
template <int D, int NBUF> struct P2gWarp {
    float4 tile[Geo<D>::TILE];
    float4 pm[NBUF][16], vv[NBUF][16], cq[NBUF][MQ<D>::Q][16];
};
// Shared memory of W warps (one group).
template <int D, int NBUF, int W = P2G_WARPS> struct P2gSmem {
    P2gWarp<D, NBUF> w[W];
};

// One pass of block r: 32 (cell, half) items (`ord` their cells) summed into
// the warp's tile.  Returns false when the pass's cells are empty (and so are
// the later passes').  With `next`, `ord` is reloaded with the next pass's
// cells once this pass's are read.  `src`: storage index of the block's first
// particle when its particles are one shifted range of storage, else NONE
// (`perm`, the block's part of the permutation, is read).
template <int D, bool FORCE, int NBUF>
__device__ __forceinline__ bool p2g_pass(const DevScene &s, P2gWarp<D, NBUF> &wm, uint32_t r, const uint32_t *perm,
                                         uint32_t src, const int (&bv)[D], float h, float inv_h, uint32_t pass,
                                         uint2 &ord, bool next) {
    constexpr int TW = Geo<D>::TW, BW = Geo<D>::BW, NST = Geo<D>::NST;
    constexpr int Q = MQ<D>::Q;
    static_assert(NBUF >= 2, "at least two staged particles");
    const uint32_t lane = lane_id();
    const size_t n = s.n;
    const int half = (int)(lane & 1u);
    const uint32_t cs = lane >> 1;  // the cell's staging slot
    const uint32_t lo = ord.x >> 6, cnt = ord.y;
    const int cell = (int)(ord.x & 63u);
    const uint32_t kmax = __shfl_sync(FULL_MASK, cnt, 0);
    if (kmax == 0u) return false;
    if (next) ord = s.bord[(size_t)r * CELLS + 16u * (pass + 1u) + cs];
    int ca[D];
    if constexpr (D == 3) {
        ca[0] = cell & 3;
        ca[1] = (cell >> 2) & 3;
        ca[2] = cell >> 4;
    } else {
        ca[0] = cell & 7;
        ca[1] = cell >> 3;
    }
    float assoc[D];
#pragma unroll
    for (int k = 0; k < D; ++k) assoc[k] = (float)(bv[k] * BW + ca[k]);
    float2 acc[NST];
#pragma unroll
    for (int k = 0; k < NST; ++k) acc[k] = make_float2(0.f, 0.f);
    // the lanes step through particle k together (k up to the pass's largest
    // count, lane 0's), so the warp can sync around the copies
    auto stage = [&](uint32_t k, int b, uint32_t i) {  // particle k into buffer b = k mod NBUF
        if (k < cnt) {
            if (half == 0) {
                cp_async16(&wm.pm[b][cs], &s.pm[i]);
                cp_async16(&wm.vv[b][cs], &s.vv[i]);
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q) cp_async16(&wm.cq[b][q][cs], &s.cq[q * n + i]);
            }
        }
        cp_async_commit();
    };
    auto index = [&](uint32_t k) { return k < cnt ? (src != NONE ? src + lo + k : perm[lo + k]) : 0u; };
#pragma unroll
    for (uint32_t k = 0; k + 1 < (uint32_t)NBUF; ++k) stage(k, (int)k, index(k));
    uint32_t i_next = index(NBUF - 1u);  // loaded one iteration before its copies
    int b = 0, fill = NBUF - 1;
    for (uint32_t k = 0; k < kmax; ++k) {
        stage(k + NBUF - 1u, fill, i_next);
        fill = b;
        i_next = index(k + NBUF);
        cp_async_wait<NBUF - 1>();
        __syncwarp();  // both lanes' copies of particle k have landed
        if (k < cnt) {
            float fdt[3] = {0.f, 0.f, 0.f};
            if constexpr (FORCE) {
                const uint32_t i = src != NONE ? src + lo + k : perm[lo + k];
#pragma unroll
                for (int d = 0; d < D; ++d) fdt[d] = s.fdt[d * n + i];
            }
            float4 cv[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) cv[q] = wm.cq[b][q][cs];
            if (!p2g_particle<D>(wm.pm[b][cs], wm.vv[b][cs], cv, fdt, assoc, h, inv_h, half, acc))
                atomicOr(s.err, ERR_KEY_RANGE);
        }
        b = b + 1 == NBUF ? 0 : b + 1;
        __syncwarp();  // the buffer just read is refilled by the next iteration's copies
    }
    cp_async_wait<0>();
    __syncwarp();
    float2 *pt = reinterpret_cast<float2 *>(wm.tile) + half;
    int base = ca[0] + TW * ca[1];
    if constexpr (D == 3) base += TW * TW * ca[2];
#pragma unroll
    for (int k = 0; k < NST; ++k) {
        const int idx = base + k % 3 + TW * ((k / 3) % 3) + TW * TW * (k / 9);
        pt[2 * idx] = __fadd2_rn(pt[2 * idx], acc[k]);
        __syncwarp();
    }
    return true;
}

// The block of rank r as P2G needs it: cell width, cell origin, first entry.
// False for a block without particles, or with stale counts (left by an
// earlier overflow).
template <int D, bool B> struct P2gBlock {
    float h, inv_h;
    int bv[D];
    uint32_t first, src;
    __device__ __forceinline__ bool load(const DevScene &s, uint32_t r, bool report) {
        const uint32_t np = s.bnp[r];
        if (np == 0) return false;
        first = s.bfirst[r];
        if ((size_t)first + np > s.n) {
            if (report) atomicOr(s.err, ERR_BLOCK_OVERFLOW);
            return false;
        }
        h = s.h;
        if constexpr (B) h = s.scenes[s.bscene[r]].h;
        inv_h = 1.0f / h;
        unpack_key<D>(s.bkey[r], bv);
        src = (!B && s.reuse && s.bsrc != nullptr) ? s.bsrc[r] : NONE;
        return true;
    }
};
template <int D, int NBUF> __device__ __forceinline__ void p2g_zero_tile(P2gWarp<D, NBUF> &wm) {
    for (int q = (int)lane_id(); q < Geo<D>::TILE; q += 32) wm.tile[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
}

// Block r by one warp.
template <int D, bool B, bool FORCE, int NBUF>
__device__ __forceinline__ void p2g_warp_block(const DevScene &s, P2gWarp<D, NBUF> &wm, uint32_t r) {
    P2gBlock<D, B> k;
    if (!k.load(s, r, lane_id() == 0)) return;
    p2g_zero_tile<D>(wm);
    uint2 ord = s.bord[(size_t)r * CELLS + (lane_id() >> 1)];
    for (uint32_t pass = 0; pass < P2G_PASSES; ++pass)
        if (!p2g_pass<D, FORCE>(s, wm, r, s.perm + k.first, k.src, k.bv, k.h, k.inv_h, pass, ord, pass + 1u < P2G_PASSES)) break;
    __syncwarp();
    for (int t = (int)lane_id(); t < Geo<D>::TILE; t += 32) s.partial[(size_t)r * Geo<D>::TILE + t] = wm.tile[t];
    __syncwarp();
}

// Block r by a group of P2G_WARPS warps, a pass each; thread `t` of the
// group, which `sync` synchronises.  `perm`: the block's part of the
// permutation where the group holds it, else null.
template <int D, bool FORCE, int NBUF, typename Sync>
__device__ __forceinline__ void p2g_group_block(const DevScene &s, P2gSmem<D, NBUF> &sm, uint32_t r, uint32_t t,
                                                const uint32_t *perm, Sync sync) {
    constexpr int TILE = Geo<D>::TILE;
    static_assert(P2G_WARPS == P2G_PASSES, "a pass a warp");
    const uint32_t wl = t >> 5;
    P2gBlock<D, false> k;
    if (!k.load(s, r, t == 0)) return;  // the same for the whole group
    p2g_zero_tile<D>(sm.w[wl]);
    uint2 ord = s.bord[(size_t)r * CELLS + 16u * wl + (lane_id() >> 1)];
    p2g_pass<D, FORCE>(s, sm.w[wl], r, perm ? perm : s.perm + k.first, k.src, k.bv, k.h, k.inv_h, wl, ord, false);
    sync();
    for (int q = (int)t; q < TILE; q += 32 * P2G_WARPS) {
        float4 sum = sm.w[0].tile[q];
#pragma unroll
        for (int w = 1; w < P2G_WARPS; ++w) {
            const float4 v = sm.w[w].tile[q];
            sum.x += v.x;
            sum.y += v.y;
            sum.z += v.z;
            sum.w += v.w;
        }
        s.partial[(size_t)r * TILE + q] = sum;
    }
    sync();  // the tiles are zeroed for the next block
}

template <int D, bool B = false, bool FORCE = false, int NBUF = 3>
__device__ __forceinline__ void p2g_body(const DevScene &s, P2gSmem<D, NBUF> &sm) {
    const uint32_t nb = s.ctr->n_blocks;
    // blocks are taken from a queue (one atomic a block), so warps that get
    // light blocks take more of them
    auto next = [&]() {
        const uint32_t q = atomicAdd(&s.ctr->p2g_next, 1u);
        return q < nb ? (s.p2g_heavy_first ? s.qorder[q] : q) : nb;
    };
    if (!B && nb < s.p2g_coop_below) {  // few blocks (a small scene): the CTA's warps share a block
        __shared__ uint32_t coop_r;
        for (;;) {
            __syncthreads();
            if (threadIdx.x == 0) coop_r = next();
            __syncthreads();
            const uint32_t r = coop_r;
            if (r >= nb) return;
            p2g_group_block<D, FORCE>(s, sm, r, threadIdx.x, nullptr, [] { __syncthreads(); });
        }
    }
    for (;;) {
        uint32_t r = 0;
        if (lane_id() == 0) r = next();
        r = __shfl_sync(FULL_MASK, r, 0);
        if (r >= nb) return;
        p2g_warp_block<D, B, FORCE>(s, sm.w[threadIdx.x >> 5], r);
    }
}
constexpr int P2G_CTAS_PER_SM = 4;
template <int D, bool B = false, bool FORCE = false, int NBUF = 3>
__global__ void __launch_bounds__(32 * P2G_WARPS, P2G_CTAS_PER_SM) k_p2g(DevScene s) {
    pdl_enter();
    __shared__ P2gSmem<D, NBUF> sm;
    p2g_body<D, B, FORCE, NBUF>(s, sm);
}

// Particle-to-grid with float atomics, kept for comparison (SLOSH_P2G=direct):
// one CTA of 128 threads a block, thread (cell, half) sums its nodes like
// k_p2g and adds them through shared-memory atomics into the block's tile,
// then 16-byte global atomics into the nodes.  Not bit-reproducible.
constexpr int P2G_ATOMIC_THREADS = 128;
template <int D> __global__ void __launch_bounds__(P2G_ATOMIC_THREADS, 4) k_p2g_atomic(DevScene s) {
    pdl_enter();
    constexpr int TW = Geo<D>::TW, TILE = Geo<D>::TILE, BW = Geo<D>::BW, NST = Geo<D>::NST;
    constexpr int NT = P2G_ATOMIC_THREADS;
    constexpr int Q = MQ<D>::Q;
    __shared__ float4 tile[TILE];
    const uint32_t nb = s.ctr->n_blocks;
    const float h = s.h, inv_h = 1.0f / s.h;
    const size_t n = s.n;
    const uint32_t tid = threadIdx.x;
    const int mycell = (int)(tid >> 1), half = (int)(tid & 1u);
    int ca[D];
    if constexpr (D == 3) {
        ca[0] = mycell & 3;
        ca[1] = (mycell >> 2) & 3;
        ca[2] = mycell >> 4;
    } else {
        ca[0] = mycell & 7;
        ca[1] = mycell >> 3;
    }
    for (uint32_t r = blockIdx.x; r < nb; r += gridDim.x) {
        const uint32_t np = s.bnp[r];
        if (np == 0) continue;
        const uint32_t first = s.bfirst[r];
        if (first + np > s.n) {
            if (tid == 0) atomicOr(s.err, ERR_BLOCK_OVERFLOW);
            continue;
        }
        for (int t = tid; t < TILE; t += NT) tile[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        int bv[D];
        unpack_key<D>(s.bkey[r], bv);
        const uint32_t lo = s.bcell[(size_t)r * CELLS + mycell];
        const uint32_t hi = (mycell < 63) ? s.bcell[(size_t)r * CELLS + mycell + 1] : np;
        float assoc[D];
#pragma unroll
        for (int k = 0; k < D; ++k) assoc[k] = (float)(bv[k] * BW + ca[k]);
        float2 acc[NST];
#pragma unroll
        for (int k = 0; k < NST; ++k) acc[k] = make_float2(0.f, 0.f);
        __syncthreads();
        for (uint32_t j = lo; j < hi; ++j) {
            const uint32_t i = s.perm[first + j];
            float fdt[3] = {0.f, 0.f, 0.f};
            if (s.force_pending) {
#pragma unroll
                for (int k = 0; k < D; ++k) fdt[k] = s.fdt[k * n + i];
            }
            float4 cv[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) cv[q] = s.cq[q * n + i];
            if (!p2g_particle<D>(s.pm[i], s.vv[i], cv, fdt, assoc, h, inv_h, half, acc)) atomicOr(s.err, ERR_KEY_RANGE);
        }
        if (hi > lo) {
            float *pt = reinterpret_cast<float *>(tile) + 2 * half;
            int base = ca[0] + TW * ca[1];
            if constexpr (D == 3) base += TW * TW * ca[2];
#pragma unroll
            for (int k = 0; k < NST; ++k) {
                const int idx = base + k % 3 + TW * ((k / 3) % 3) + TW * TW * (k / 9);
                atomicAdd(&pt[4 * idx], acc[k].x);
                atomicAdd(&pt[4 * idx + 1], acc[k].y);
            }
        }
        __syncthreads();
        for (int t = tid; t < TILE; t += NT) {
            const float4 val = tile[t];
            if (val.x == 0.f && val.y == 0.f && val.z == 0.f && val.w == 0.f) continue;
            uint32_t rank, local;
            if (!tile_node_owner<D>(s, r, t, rank, local)) continue;
            atomicAdd(&s.nodes[(size_t)rank * 64u + local], val);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Colliders: Sim3/Sim2 poses, ball and cuboid projections, collide() and the
// boundary-condition projection.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void quat_rotate(const float *q, const float *v, float *out) {
    const float t0 = 2.f * products_diff(q[1], v[2], q[2], v[1]);
    const float t1 = 2.f * products_diff(q[2], v[0], q[0], v[2]);
    const float t2 = 2.f * products_diff(q[0], v[1], q[1], v[0]);
    out[0] = fmaf(q[3], t0, v[0]) + products_diff(q[1], t2, q[2], t1);
    out[1] = fmaf(q[3], t1, v[1]) + products_diff(q[2], t0, q[0], t2);
    out[2] = fmaf(q[3], t2, v[2]) + products_diff(q[0], t1, q[1], t0);
}

template <int D> __device__ __forceinline__ void pose_mul_pt(const DevBody &b, const float *p, float *out) {
    if constexpr (D == 3) {
        const float sp[3] = {p[0] * b.scale, p[1] * b.scale, p[2] * b.scale};
        float r[3];
        quat_rotate(b.rot, sp, r);
        for (int i = 0; i < 3; ++i) out[i] = r[i] + b.tra[i];
    } else {
        const float sp0 = p[0] * b.scale, sp1 = p[1] * b.scale;
        out[0] = products_diff(b.rot[0], sp0, b.rot[1], sp1) + b.tra[0];
        out[1] = products_sum(b.rot[1], sp0, b.rot[0], sp1) + b.tra[1];
    }
}

// The inverse pose of the grid node at cell * h.  Differences with a node's
// position are formed from its cell, rounded once (here and in collide): the
// product rounded first moves a node near a surface by a visible part of its
// distance.
template <int D>
__device__ __forceinline__ void pose_inv_mul_node(const DevBody &b, const float *cell, float h, float *out) {
    if constexpr (D == 3) {
        const float d[3] = {fmaf(cell[0], h, -b.tra[0]), fmaf(cell[1], h, -b.tra[1]), fmaf(cell[2], h, -b.tra[2])};
        const float qi[4] = {-b.rot[0], -b.rot[1], -b.rot[2], b.rot[3]};
        float r[3];
        quat_rotate(qi, d, r);
        for (int i = 0; i < 3; ++i) out[i] = r[i] / b.scale;
    } else {
        const float d0 = fmaf(cell[0], h, -b.tra[0]), d1 = fmaf(cell[1], h, -b.tra[1]);
        out[0] = products_sum(b.rot[0], d0, b.rot[1], d1) / b.scale;
        out[1] = products_diff(b.rot[0], d1, b.rot[1], d0) / b.scale;
    }
}

// Closest point of the segment a-b (shaders/slosh/rbd/shapes/segment.slang:9-28):
// an end point in its Voronoi region, else the orthogonal projection.
template <int D> __device__ __forceinline__ void segment_closest(const float *a, const float *b, const float *p,
                                                                 float *q) {
    float ab[D], ap_ab = 0.f, ab2 = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        ab[k] = b[k] - a[k];
        ap_ab += ab[k] * (p[k] - a[k]);
        ab2 += ab[k] * ab[k];
    }
    if (ap_ab <= 0.f) {
#pragma unroll
        for (int k = 0; k < D; ++k) q[k] = a[k];
    } else if (ap_ab >= ab2) {
#pragma unroll
        for (int k = 0; k < D; ++k) q[k] = b[k];
    } else {
        const float u = ap_ab / ab2;
#pragma unroll
        for (int k = 0; k < D; ++k) q[k] = a[k] + ab[k] * u;
    }
}

// Capsule = segment a-b inflated by `radius` (capsule.slang:38-55): the
// closest axis point pushed out by the radius.  A point exactly on the axis
// goes out along a fixed unit vector orthogonal to the axis: in 3D the first
// vector of the branchless orthonormal basis of Duff et al., "Building an
// Orthonormal Basis, Revisited" (JCGT 2017).  Returns "inside".
template <int D>
__device__ __forceinline__ bool capsule_boundary(const float *a, const float *b, float radius, const float *p,
                                                 float *out) {
    float q[D], d[D], n2 = 0.f;
    segment_closest<D>(a, b, p, q);
#pragma unroll
    for (int k = 0; k < D; ++k) {
        d[k] = p[k] - q[k];
        n2 += d[k] * d[k];
    }
    const float dist = sqrtf(n2);
    if (dist > 0.f) {
#pragma unroll
        for (int k = 0; k < D; ++k) out[k] = q[k] + d[k] * (radius / dist);
        return dist <= radius;
    }
    float ax[D], l2 = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        ax[k] = b[k] - a[k];
        l2 += ax[k] * ax[k];
    }
    const float len = sqrtf(l2);
#pragma unroll
    for (int k = 0; k < D; ++k) ax[k] /= len;
    float o[D];
    if constexpr (D == 2) {
        o[0] = ax[1];
        o[1] = -ax[0];
    } else {
        const float sg = ax[2] >= 0.f ? 1.f : -1.f;
        const float aa = -1.0f / (sg + ax[2]);
        const float bb = ax[0] * ax[1] * aa;
        o[0] = 1.0f + sg * ax[0] * ax[0] * aa;
        o[1] = sg * bb;
        o[2] = -sg * ax[0];
    }
#pragma unroll
    for (int k = 0; k < D; ++k) out[k] = q[k] + o[k] * radius;
    return true;
}

// Cylinder of half height hh and radius r around the local y axis
// (cylinder.slang:72-125): inside, the nearest of the two caps and the
// side; outside, the cap disc, the cap rim or the side.  Returns "inside".
__device__ __forceinline__ bool cylinder_boundary(float hh, float r, const float *p, float *out) {
    const float rxz = sqrtf(products_sum(p[0], p[0], p[2], p[2]));
    const float dx = rxz > 0.f ? p[0] / rxz : 1.f, dz = rxz > 0.f ? p[2] / rxz : 0.f;
    const float sx = dx * r, sz = dz * r;
    if (p[1] >= -hh && p[1] <= hh && rxz <= r) {
        const float to_top = hh - p[1], to_bottom = p[1] + hh, to_side = r - rxz;
        if (to_top < to_bottom && to_top < to_side) {
            out[0] = p[0], out[1] = hh, out[2] = p[2];
        } else if (to_bottom < to_top && to_bottom < to_side) {
            out[0] = p[0], out[1] = -hh, out[2] = p[2];
        } else {
            out[0] = sx, out[1] = p[1], out[2] = sz;
        }
        return true;
    }
    if (p[1] > hh || p[1] < -hh) {
        const float y = p[1] > hh ? hh : -hh;
        if (rxz <= r) out[0] = p[0], out[1] = y, out[2] = p[2];
        else out[0] = sx, out[1] = y, out[2] = sz;
    } else {
        out[0] = sx, out[1] = p[1], out[2] = sz;
    }
    return false;
}

// Cone of half height hh and base radius r, apex at +hh on the local y axis
// (cone.slang:82-131): below the base disc, the disc; otherwise the closest
// point of the generatrix through the point's azimuth, or (inside) the base
// when that is nearer.  Returns "inside".
__device__ __forceinline__ bool cone_boundary(float hh, float r, const float *p, float *out) {
    const float rxz = sqrtf(products_sum(p[0], p[0], p[2], p[2]));
    const float dx = rxz > 0.f ? p[0] / rxz : 1.f, dz = rxz > 0.f ? p[2] / rxz : 0.f;
    const float base[3] = {p[0], -hh, p[2]};
    if (p[1] < -hh && rxz <= r) {
#pragma unroll
        for (int k = 0; k < 3; ++k) out[k] = base[k];
        return false;
    }
    const float rim[3] = {dx * r, -hh, dz * r};
    const float apex[3] = {0.f, hh, 0.f};
    float proj[3];
    segment_closest<3>(apex, rim, p, proj);
    const float gen[3] = {rim[0] - apex[0], rim[1] - apex[1], rim[2] - apex[2]};
    const float ap[3] = {p[0] - apex[0], p[1] - apex[1], p[2] - apex[2]};
    const float axis[3] = {0.f, -2.0f * hh, 0.f};
    const float c1[3] = {products_diff(gen[1], ap[2], gen[2], ap[1]), products_diff(gen[2], ap[0], gen[0], ap[2]),
                         products_diff(gen[0], ap[1], gen[1], ap[0])};
    const float c2[3] = {products_diff(gen[1], axis[2], gen[2], axis[1]), products_diff(gen[2], axis[0], gen[0], axis[2]),
                         products_diff(gen[0], axis[1], gen[1], axis[0])};
    const bool in = p[1] >= -hh && p[1] <= hh && fmaf(c1[2], c2[2], products_sum(c1[0], c2[0], c1[1], c2[1])) >= 0.f;
    if (in) {
        float d_side = 0.f, d_base = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            d_side += (proj[k] - p[k]) * (proj[k] - p[k]);
            d_base += (base[k] - p[k]) * (base[k] - p[k]);
        }
        const float *src = d_side > d_base ? base : proj;
#pragma unroll
        for (int k = 0; k < 3; ++k) out[k] = src[k];
        return true;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = proj[k];
    return false;
}

// Shape::project_point_on_boundary for balls, cuboids, capsules, cylinders
// and cones (shaders/slosh/rbd/shapes/shape.slang:152-175; ball.slang:39-52,
// cuboid.slang:14-63, capsule.slang, cylinder.slang, cone.slang), and the
// triangle-mesh query of collide (collision/collide.slang:124-134): a mesh
// point is returned only within `cap` of the surface.
template <int D>
__device__ __forceinline__ bool project_on_boundary(const DevBody &b, const float *cell, float h, float *proj,
                                                    bool &inside, const float4 *mvtx, const uint32_t *midx, float cap) {
    float local[D], lp[D];
    pose_inv_mul_node<D>(b, cell, h, local);
    if (b.shape_type == SLOSH_SHAPE_CUBOID) {
        float outp[D], sgn[D], diff[D], inp[D];
        bool in = true;
#pragma unroll
        for (int i = 0; i < D; ++i) {
            const float shift = fmaxf(-b.sa[i] - local[i], 0.f) - fmaxf(local[i] - b.sa[i], 0.f);
            outp[i] = local[i] + shift;
            const float sw = (local[i] > 0.f) ? 1.f : ((local[i] < 0.f) ? -1.f : 0.f);
            sgn[i] = sw + (fabsf(sw) - 1.f);
            diff[i] = fmaf(-sgn[i], local[i], b.sa[i]);
            inp[i] = local[i];
            in = in && (local[i] == outp[i]);
        }
        if constexpr (D == 3) {
            const bool px = diff[0] <= diff[1] && diff[0] <= diff[2];
            const bool py = diff[1] <= diff[0] && diff[1] <= diff[2];
            if (px) inp[0] = fmaf(diff[0], sgn[0], local[0]);
            else if (py) inp[1] = fmaf(diff[1], sgn[1], local[1]);
            else inp[2] = fmaf(diff[2], sgn[2], local[2]);
        } else {
            if (diff[0] <= diff[1]) inp[0] = fmaf(diff[0], sgn[0], local[0]);
            else inp[1] = fmaf(diff[1], sgn[1], local[1]);
        }
#pragma unroll
        for (int i = 0; i < D; ++i) lp[i] = in ? inp[i] : outp[i];
        inside = in;
    } else if (b.shape_type == SLOSH_SHAPE_BALL) {
        float n2 = 0.f;
#pragma unroll
        for (int i = 0; i < D; ++i) n2 += local[i] * local[i];
        const float dist = sqrtf(n2), rad = b.sa[0];
#pragma unroll
        for (int i = 0; i < D; ++i) lp[i] = (dist != 0.f) ? local[i] * (rad / dist) : 0.f;
        if (dist == 0.f) lp[1] = rad;
        inside = dist <= rad;
    } else if (b.shape_type == SLOSH_SHAPE_CAPSULE) {
        inside = capsule_boundary<D>(b.sa, b.sb, b.sb[3], local, lp);
    } else if constexpr (D == 3) {
        if (b.shape_type == SLOSH_SHAPE_CYLINDER) inside = cylinder_boundary(b.sa[0], b.sa[1], local, lp);
        else if (b.shape_type == SLOSH_SHAPE_CONE) inside = cone_boundary(b.sa[0], b.sa[1], local, lp);
        else if (b.shape_type == SLOSH_SHAPE_TRIMESH && mvtx) {
            if (!trimesh_project(trimesh_ref(b.sa, b.sb), mvtx, midx, local, cap, lp, inside)) return false;
        } else
            return false;
    } else {
        return false;
    }
    pose_mul_pt<D>(b, lp, proj);
    return true;
}

// collide (shaders/slosh/collision/collide.slang:87-153).  Returns the
// collider id or NONE; `nd` = (normal, dot(point_node - proj, normal)).
template <int D>
__device__ __forceinline__ uint32_t collide(const DevBody *bodies, uint32_t n_bodies, float h, const float *cell,
                                            float4 &nd, const float4 *mvtx, const uint32_t *midx) {
    const float cap = h * 1.5f;
    float best = 1.0e10f;
    uint32_t id = NONE;
    float bn[D] = {}, bp[D] = {};
    for (uint32_t i = 0; i < n_bodies && i < MAX_BODIES; ++i) {
        float proj[D];
        bool inside = false;
        if (!project_on_boundary<D>(bodies[i], cell, h, proj, inside, mvtx, midx, cap)) continue;
        float dpt[D], n2 = 0.f;
        bool within = true;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            dpt[k] = fmaf(-cell[k], h, proj[k]);
            within = within && (fabsf(dpt[k]) <= cap);
            n2 += dpt[k] * dpt[k];
        }
        if (inside || within) {
            const float sign = inside ? -1.f : 1.f;
            const float dist = sqrtf(n2);
            if (sign * dist < best && dist != 0.f) {
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    bn[k] = dpt[k] / (dist * -sign);
                    bp[k] = proj[k];
                }
                id = i;
                best = dist;
            }
        }
    }
    float dd = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) dd = fmaf(fmaf(cell[k], h, -bp[k]), bn[k], dd);
    nd = make_float4(bn[0], bn[1], D == 3 ? bn[D - 1] : 0.f, dd);
    return id;
}

// BoundaryCondition::project_velocity (boundary_condition.slang:31-89),
// keeping slosh's use of the collider friction for FrictionZUp.
template <int D>
__device__ __forceinline__ void project_velocity(uint32_t type, float friction, float *vel, const float *n, float dist,
                                                 float dt) {
    if (type == SLOSH_BC_STICK) {
        if (dist <= 0.f)
#pragma unroll
            for (int k = 0; k < D; ++k) vel[k] = 0.f;
    } else if (type == SLOSH_BC_SLIP) {
        if (dist <= 0.f) {
            float nv = 0.f;
#pragma unroll
            for (int k = 0; k < D; ++k) nv += vel[k] * n[k];
#pragma unroll
            for (int k = 0; k < D; ++k) vel[k] = vel[k] - n[k] * nv;
        }
    } else if (type == SLOSH_BC_SEPARATE || type == SLOSH_BC_FRICTION_Z_UP) {
        float nv = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) nv += vel[k] * n[k];
        if (nv < 0.f) {
            if (dist <= 0.f) {
                float tv[D], tl2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    tv[k] = vel[k] - n[k] * nv;
                    tl2 += tv[k] * tv[k];
                }
                const float tl = sqrtf(tl2);
                const float sc = fmaxf(0.f, tl + friction * nv);
#pragma unroll
                for (int k = 0; k < D; ++k) vel[k] = ((tl > 1.0e-8f) ? tv[k] / tl : 0.f) * sc;
            } else if (-nv * dt > dist) {
                const float a = dist / dt + nv;
#pragma unroll
                for (int k = 0; k < D; ++k) vel[k] = vel[k] - a * n[k];
            }
        }
    }
}

// Grid update (shaders/slosh/solver/grid_update.slang:38-163), one thread per
// node.  The collision of a node is reused from the previous substep when
// its block was active there (slosh's cache, which assumes static colliders),
// otherwise collide() runs; both are recorded for the next substep.
// 8 CTAs of 256 per SM (64 warps): the node gather is a chain of dependent
// loads, so occupancy pays; the register cap (32) leaves the rare collision
// queries (nodes without a cached collision) to spill, not the common path.
template <int D, bool B = false> __device__ __forceinline__ void grid_update_body(const DevScene &s, Cta g) {
    constexpr int BW = Geo<D>::BW;
    const uint32_t nb = s.ctr->n_blocks;
    const uint32_t stride = g.n * blockDim.x;
    float h = s.h, dt = s.dt, grav[3] = {s.gravity[0], s.gravity[1], s.gravity[2]};
    const DevBody *bodies = s.bodies;
    uint32_t n_bodies = s.n_bodies, sc = 0;
    for (uint32_t t = g.id * blockDim.x + threadIdx.x; t < nb * 64u; t += stride) {
        const uint32_t r = t >> 6, node = t & 63u;
        if constexpr (B) {
            sc = s.bscene[r];
            const SceneRec &rec = s.scenes[sc];
            h = rec.h;
            dt = rec.dt;
            for (int k = 0; k < 3; ++k) grav[k] = rec.gravity[k];
            bodies = s.bodies + rec.body_first;
            n_bodies = rec.n_bodies;
        }
        const float vlim = h / dt;
        const uint32_t key = s.bkey[r];
        int bv[D], lc[D];
        unpack_key<D>(key, bv);
        if constexpr (D == 3) {
            lc[0] = node & 3;
            lc[1] = (node >> 2) & 3;
            lc[2] = node >> 4;
        } else {
            lc[0] = node & 7;
            lc[1] = node >> 3;
        }
        float cell[D];  // the node's position is cell * h
#pragma unroll
        for (int k = 0; k < D; ++k) cell[k] = (float)(bv[k] * BW + lc[k]);
        float4 nv;
        if (s.use_partial) {
            // Node sums of the deterministic P2G: the tiles of this block and
            // of its -1 neighbours b - o that cover the node (local
            // coordinate + BW o inside the tile), added in the fixed order
            // of o.
            constexpr int TW = Geo<D>::TW, NN = Geo<D>::NASSOC - 1;
            nv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < Geo<D>::NASSOC; ++q) {
                int o[D];
                assoc_offset<D>(q, o);
                bool inside = true;
                int tix = 0, mul = 1;
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const int tc = lc[k] + BW * o[k];
                    inside = inside && tc < TW;
                    tix += tc * mul;
                    mul *= TW;
                }
                if (!inside) continue;
                // blocks without particles have no tile (their -1
                // neighbour ranks are NONE)
                const uint32_t ra = (q == 0) ? (s.bnp[r] != 0u ? r : NONE) : s.bnbh_rev[r * NN + q - 1];
                if (ra >= nb) continue;
                const float4 v = s.partial[(size_t)ra * Geo<D>::TILE + tix];
                nv.x += v.x;
                nv.y += v.y;
                nv.z += v.z;
                nv.w += v.w;
            }
            if (s.gather_only) {
                s.nodes[t] = nv;
                continue;
            }
        } else {
            nv = s.nodes[t];
        }
        const float pm[3] = {nv.x, nv.y, nv.z};
        const float mass = nv.w;
        const float inv_mass = mass > 0.f ? 1.0f / mass : 0.f;
        float vel[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const float v = (pm[k] + mass * grav[k] * dt) * inv_mass;
            vel[k] = fminf(fmaxf(v, -vlim), vlim);
        }
        // The cached normal and distance are read, and recorded, only for a
        // node that has a collision (cid != NONE), their only readers.
        float4 cn = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t cid;
        const uint32_t prank = s.bprev[r];
        if (prank != NONE && !s.coll_dynamic) {
            cid = s.prev_coll_id[(size_t)prank * 64u + node];
            if (cid != NONE) cn = s.prev_coll[(size_t)prank * 64u + node];
        } else {
            cid = collide<D>(bodies, n_bodies, h, cell, cn, s.mesh_vtx, s.mesh_idx);
        }
        if (cid != NONE) s.coll[t] = cn;
        s.coll_id[t] = cid;
        if (cid != NONE) {
            const DevBody &bd = bodies[cid];
            const float n[3] = {cn.x, cn.y, cn.z};
            if (bd.coupling == SLOSH_COUPLING_TWO_WAY) {
                // project in the body's frame; the momentum the node loses
                // goes to the body as an impulse at the node
                float com[3] = {0.f, 0.f, 0.f}, r[3] = {0.f, 0.f, 0.f}, vb[3] = {0.f, 0.f, 0.f};
                pose_mul_pt<D>(bd, bd.local_com, com);
#pragma unroll
                for (int k = 0; k < D; ++k) r[k] = fmaf(cell[k], h, -com[k]);
                if constexpr (D == 3) {
                    vb[0] = fmaf(-bd.angvel[2], r[1], fmaf(bd.angvel[1], r[2], bd.linvel[0]));
                    vb[1] = fmaf(-bd.angvel[0], r[2], fmaf(bd.angvel[2], r[0], bd.linvel[1]));
                    vb[2] = fmaf(-bd.angvel[1], r[0], fmaf(bd.angvel[0], r[1], bd.linvel[2]));
                } else {
                    vb[0] = bd.linvel[0] - bd.angvel[0] * r[1];
                    vb[1] = bd.linvel[1] + bd.angvel[0] * r[0];
                }
                float rel[D];
#pragma unroll
                for (int k = 0; k < D; ++k) rel[k] = vel[k] - vb[k];
                project_velocity<D>(bd.bc_type, bd.friction, rel, n, cn.w - h, dt);
                float J[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < D; ++k) {
                    const float nvk = rel[k] + vb[k];
                    J[k] = mass * (vel[k] - nvk);
                    vel[k] = nvk;
                }
                if (mass > 0.f) {
                    float A[3];
                    int na;
                    if constexpr (D == 3) {
                        A[0] = products_diff(r[1], J[2], r[2], J[1]);
                        A[1] = products_diff(r[2], J[0], r[0], J[2]);
                        A[2] = products_diff(r[0], J[1], r[1], J[0]);
                        na = 3;
                    } else {
                        A[0] = products_diff(r[0], J[1], r[1], J[0]);
                        na = 1;
                    }
                    unsigned long long *acc = s.body_imp + (size_t)(&bd - s.bodies) * 6u;
#pragma unroll
                    for (int k = 0; k < D; ++k)
                        if (J[k] != 0.f) atomicAdd(acc + k, (unsigned long long)__double2ll_rn((double)J[k] * IMPULSE_UNITS));
                    for (int k = 0; k < na; ++k)
                        if (A[k] != 0.f)
                            atomicAdd(acc + 3 + k, (unsigned long long)__double2ll_rn((double)A[k] * IMPULSE_UNITS));
                }
            } else {
                project_velocity<D>(bd.bc_type, bd.friction, vel, n, cn.w - h, dt);
            }
        }
        s.nodes[t] = make_float4(vel[0], vel[1], D == 3 ? vel[D - 1] : 0.f, mass);
    }
}
template <int D, bool B = false> __global__ void __launch_bounds__(256, 8) k_grid_update(DevScene s) {
    pdl_enter();
    grid_update_body<D, B>(s, launch_cta());
}

// Clears the next substep's hash map and the key histogram / per-scene
// block counts (their readers in this substep have all run), thread g0 of
// gs.  Done by the fused G2P / particle update, or by k_clear_next when a
// stage hook replaced it.
// hist: also the key histogram (a build that did not count in it leaves it
// clear).
template <bool B>
__device__ __forceinline__ void clear_next_map(const DevScene &s, uint32_t g0, uint32_t gs, bool hist = true) {
    for (uint32_t q = g0; q < s.hcap; q += gs) {
        if constexpr (B) s.clr_hkeys64[q] = NONE64;
        else s.clr_hkeys[q] = NONE;
        s.clr_hvals[q] = NONE;
    }
    if constexpr (B) {
        for (uint32_t q = g0; q < s.n_scenes; q += gs) s.scene_nblk[q] = 0u;
    } else if (hist) {
        for (uint32_t q = g0; q < HIST_BINS; q += gs) s.hist[q] = 0u;
        if (g0 < HIST_COARSE) s.hist_coarse[g0] = 0u;
    }
    if (*s.err != 0u) {
        for (size_t q = g0; q < (size_t)s.hcap * CELLS; q += gs) s.slot_counts[q] = 0u;
        if (!B && s.slot_total)
            for (uint32_t q = g0; q < s.hcap; q += gs) s.slot_total[q] = 0u;
    }
}

// After a stage hook replaced the fused G2P / particle update: the next
// map cleared as G2P would, and the original-index plane of the next
// storage taken from its flags plane.
__global__ void k_after_replaced_g2p(DevScene s) {
    pdl_enter();
    const uint32_t g0 = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
    clear_next_map<false>(s, g0, gs);
    for (uint32_t i = g0; i < s.count; i += gs) s.out_oid[i] = s.out_fo[i].y;
}

// Grid-reuse bookkeeping of one particle that G2P has just moved from xo to
// xn (storage position in block r of this substep's grid): when its base
// cell changed, the per-cell count deltas and touched-cell bits of the old
// and new blocks, which the next substep's k_grid_reuse applies; when the
// change is one the kept grid cannot hold (a move of more than one cell, or
// into a block without particles or outside the grid), the next substep's
// full build.  The cells are the ones k_touch would compute from the stored
// positions.
template <int D, bool POW2>
__device__ __forceinline__ void note_cell_change(const DevScene &s, uint32_t r, const float4 &xo4, const float4 &xn4,
                                                 float h, float inv_h, uint32_t h_pow2) {
    const float xo[3] = {xo4.x, xo4.y, xo4.z}, xn[3] = {xn4.x, xn4.y, xn4.z};
    // round(x / h) per axis, as locate() computes it (the base cell is one less)
    int co[D], cn[D];
    bool moved = false;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        co[k] = __float2int_rn(POW2 ? xo[k] * inv_h : div_h(xo[k], h, inv_h, h_pow2));
        cn[k] = __float2int_rn(POW2 ? xn[k] * inv_h : div_h(xn[k], h, inv_h, h_pow2));
        moved = moved || co[k] != cn[k];
    }
    if (!moved) return;
    constexpr int SHIFT = Geo<D>::BW == 4 ? 2 : 3, BW = Geo<D>::BW;
    int bo[D], bn[D], lo[D], ln[D];
    bool far = false, same_block = true;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const int dc = cn[k] - co[k];
        far = far || dc > 1 || dc < -1;
        bo[k] = (co[k] - 1) >> SHIFT;
        bn[k] = (cn[k] - 1) >> SHIFT;
        lo[k] = (co[k] - 1) & (BW - 1);
        ln[k] = (cn[k] - 1) & (BW - 1);
        same_block = same_block && bo[k] == bn[k];
    }
    uint32_t r2 = r;
    bool ok = !far;
    if (ok && !same_block) {
        const uint32_t slot = hash_find(s.hkeys, s.hcap, pack_key<D>(bn));
        const uint32_t v = slot == NONE ? NONE : s.hvals[slot];
        ok = v != NONE && (v & RANK_EXTRA) == 0u;
        r2 = v;
    }
    if (!ok) {
        s.ctr->rebuild[s.par ^ 1u] = 1u;
        return;
    }
    const uint32_t c_old = cell_index<D>(lo), c_new = cell_index<D>(ln);
    atomicAdd(&s.cell_delta[(size_t)r * CELLS + c_old], -1);
    atomicAdd(&s.cell_delta[(size_t)r2 * CELLS + c_new], 1);
    atomicOr(&s.touch[r], 1ull << c_old);
    atomicOr(&s.touch[r2], 1ull << c_new);
}

// G2P fused with the particle update.  One CTA per active block with
// primaries: the block's (block + 2)^D tile of node velocities is staged in
// shared memory, then each thread gathers v, grad v and div v for its
// particles (g2p.slang:150-265) and applies the particle update of
// particle_update.slang:48-159 with the constitutive model, writing the new
// position, velocity, APIC matrix C and F.  The inputs of a thread's next
// particle (x, m, F, V0, flags, original id, plastic state, damping) are
// staged into shared memory with cp.async while the current particle is
// computed; each thread consumes only its own staged slot, so the particle
// loop has no barrier.
// POW2: the cell width is a power of two (known at launch), so x / h is
// exactly x * (1/h) and no division is compiled in.  MODEL >= 0: every
// particle of the scene uses that model tag (known at upload), so only its
// constitutive code is compiled in; MODEL < 0 reads each particle's tag.
// Shared memory of k_g2p_update's CTA (NT threads): the block's node tile
// (velocity, mass: one 16-byte load a node) and two buffers of staged
// particles, one particle a thread.
template <int D, int NT> struct G2pSmem {
    float4 tv[Geo<D>::TILE];
    float4 st_pm[2][NT];
    float4 st_fq[2][MQ<D>::Q][NT];
    uint4 st_fo[2][NT];
    float4 st_ps[2][NT];
    uint32_t next_r;
};

// Particles e0, e0 + stride, ... (a thread's own) of block r, by a group of NT
// threads (`tid` the thread in it) that `sync` synchronises.
template <int D, int NT, bool B, bool POW2, int MODEL, typename Sync>
__device__ __forceinline__ void g2p_block(const DevScene &s, G2pSmem<D, NT> &sm, uint32_t r, uint32_t np, uint32_t tid,
                                          uint32_t e0, uint32_t stride, Sync sync) {
    constexpr int TW = Geo<D>::TW, TILE = Geo<D>::TILE, BW = Geo<D>::BW;
    constexpr int Q = MQ<D>::Q;
    auto &tv = sm.tv;
    auto &st_pm = sm.st_pm;
    auto &st_fq = sm.st_fq;
    auto &st_fo = sm.st_fo;
    auto &st_ps = sm.st_ps;
    const size_t n = s.n;
    // Issues the copies of sorted entry e (storage index i) of the block into
    // buffer b (an empty group when e is past the block's particles).  The
    // storage index is loaded one iteration before the copies that need it.
    auto stage = [&](int b, uint32_t e, uint32_t i) {
        if (e < np) {
            cp_async16(&st_pm[b][tid], &s.pm[i]);
#pragma unroll
            for (int q = 0; q < Q; ++q) cp_async16(&st_fq[b][q][tid], &s.fq[q * n + i]);
            cp_async16(&st_fo[b][tid], &s.fo[i]);
            if (s.has_sand | s.has_damping) cp_async16(&st_ps[b][tid], &s.ps[i]);
        }
        cp_async_commit();
    };
    const uint32_t first = s.bfirst[r];
    // storage index of entry e: from the block's storage start when its
    // particles are one shifted range of storage, else the permutation
    const uint32_t src = (!B && s.reuse && s.bsrc != nullptr) ? s.bsrc[r] : NONE;
    auto pidx = [&](uint32_t e) { return src != NONE ? src + e : s.perm[first + e]; };
    stage(0, e0, e0 < np ? pidx(e0) : 0u);
    uint32_t i_next = e0 + stride < np ? pidx(e0 + stride) : 0u;
    float h = s.h, dt = s.dt, inv_h = s.inv_h;
    uint32_t h_pow2 = s.h_pow2;
    if constexpr (B) {
        const SceneRec &rec = s.scenes[s.bscene[r]];
        h = rec.h;
        dt = rec.dt;
        inv_h = rec.inv_h;
        h_pow2 = rec.h_pow2;
    }
    const float inv_d = 4.0f / (h * h), vmax = h / dt;
    for (uint32_t t = tid; t < TILE; t += NT) {
        uint32_t rank, local;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tile_node_owner<D>(s, r, (int)t, rank, local)) v = s.nodes[(size_t)rank * 64u + local];
        tv[t] = v;
    }
    sync();
    int bv[D];
    unpack_key<D>(s.bkey[r], bv);
    int buf = 0;
    for (uint32_t e = e0; e < np; e += stride, buf ^= 1) {
        stage(buf ^ 1, e + stride, i_next);
        i_next = e + 2 * stride < np ? pidx(e + 2 * stride) : 0u;
        cp_async_wait<1>();
        const float4 p = st_pm[buf][tid];
        const float x[3] = {p.x, p.y, p.z};
        float m = p.w;
        const uint4 fo = st_fo[buf][tid];
        uint32_t fl = fo.x;
        // ---- G2P ----
        float vel[D], grad[D][D], div = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            vel[k] = 0.f;
#pragma unroll
            for (int l = 0; l < D; ++l) grad[k][l] = 0.f;
        }
        if (fl & FLAG_ENABLED) {
            float d0[D], w[D][3];
            int a[D];
            bool in_block = true;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const float assoc = rintf(POW2 ? x[k] * inv_h : div_h(x[k], h, inv_h, h_pow2)) - 1.0f;
                a[k] = (int)assoc - bv[k] * BW;
                in_block = in_block && a[k] >= 0 && a[k] < BW;
                d0[k] = fmaf(assoc, h, -x[k]);
                bspline_weights(POW2 ? -d0[k] * inv_h : div_h(-d0[k], h, inv_h, h_pow2), w[k]);
            }
            if (!in_block) {  // packed-key aliasing: gather nothing
                atomicOr(s.err, ERR_KEY_RANGE);
#pragma unroll
                for (int k = 0; k < D; ++k) a[k] = 0, w[k][0] = w[k][1] = w[k][2] = 0.f;
            }
            // Separable gather.  With w_s = wx[sx] wy[sy] wz[sz] and
            // dpt_s = d0 + s h, the sums of g2p.slang:196-244 are
            //   v = M0,  grad v[c][r] = inv_d (d0_r M0_c + h M_r,c),
            //   vel_grad_det = trace(grad v),
            // with M0 = sum_s w_s v_s and M_r = sum_s w_s s_r v_s,
            // accumulated axis by axis.
            // Separable gather in paired FP32 arithmetic: the node
            // velocity (x, y, z, mass) is read as the pairs (x, y) and
            // (z, mass); the mass lane is carried along unused.  Terms
            // with offset 0 (s_r = 0) add nothing and are skipped.
            constexpr int NP = (D == 3) ? 2 : 1;
            float2 M0p[NP], Mrp[D][NP];
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                M0p[q] = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < D; ++k) Mrp[k][q] = make_float2(0.f, 0.f);
            }
            const float2 wx0p = pair(w[0][0]), wx1p = pair(w[0][1]), wx2p = pair(w[0][2]),
                         wx2bp = pair(2.f * w[0][2]);
            auto row = [&](const float4 &n0, const float4 &n1, const float4 &n2, int q, float2 &R0, float2 &Rx) {
                const float2 v0 = q ? hi_pair(n0) : lo_pair(n0), v1 = q ? hi_pair(n1) : lo_pair(n1),
                             v2 = q ? hi_pair(n2) : lo_pair(n2);
                R0 = __ffma2_rn(wx2p, v2, __ffma2_rn(wx1p, v1, __fmul2_rn(wx0p, v0)));
                Rx = __ffma2_rn(wx2bp, v2, __fmul2_rn(wx1p, v1));
            };
            if constexpr (D == 3) {
#pragma unroll
                for (int sz = 0; sz < 3; ++sz) {
                    float2 S0[2], Sx[2], Sy[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) S0[q] = Sx[q] = Sy[q] = make_float2(0.f, 0.f);
#pragma unroll
                    for (int sy = 0; sy < 3; ++sy) {
                        const int idx = a[0] + TW * ((a[1] + sy) + TW * (a[2] + sz));
                        const float2 wyp = pair(w[1][sy]), wysp = pair((float)sy * w[1][sy]);
                        const float4 n0 = tv[idx], n1 = tv[idx + 1], n2 = tv[idx + 2];
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            float2 R0, Rx;
                            row(n0, n1, n2, q, R0, Rx);
                            S0[q] = __ffma2_rn(wyp, R0, S0[q]);
                            Sx[q] = __ffma2_rn(wyp, Rx, Sx[q]);
                            if (sy > 0) Sy[q] = __ffma2_rn(wysp, R0, Sy[q]);
                        }
                    }
                    const float2 wzp = pair(w[2][sz]), wzsp = pair((float)sz * w[2][sz]);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        M0p[q] = __ffma2_rn(wzp, S0[q], M0p[q]);
                        Mrp[0][q] = __ffma2_rn(wzp, Sx[q], Mrp[0][q]);
                        Mrp[1][q] = __ffma2_rn(wzp, Sy[q], Mrp[1][q]);
                        if (sz > 0) Mrp[2][q] = __ffma2_rn(wzsp, S0[q], Mrp[2][q]);
                    }
                }
            } else {
#pragma unroll
                for (int sy = 0; sy < 3; ++sy) {
                    const int idx = a[0] + TW * (a[1] + sy);
                    const float2 wyp = pair(w[1][sy]), wysp = pair((float)sy * w[1][sy]);
                    float2 R0, Rx;
                    row(tv[idx], tv[idx + 1], tv[idx + 2], 0, R0, Rx);
                    M0p[0] = __ffma2_rn(wyp, R0, M0p[0]);
                    Mrp[0][0] = __ffma2_rn(wyp, Rx, Mrp[0][0]);
                    if (sy > 0) Mrp[1][0] = __ffma2_rn(wysp, R0, Mrp[1][0]);
                }
            }
            // v = M0, grad v[c][r] = inv_d (d0_r M0_c + h M_r,c), pairs over c
            const float2 hp = pair(h), invdp = pair(inv_d);
#pragma unroll
            for (int rr = 0; rr < D; ++rr) {
                const float2 d0p = pair(d0[rr]);
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    const float2 g = __fmul2_rn(invdp, __ffma2_rn(d0p, M0p[q], __fmul2_rn(hp, Mrp[rr][q])));
                    grad[2 * q][rr] = g.x;
                    if (2 * q + 1 < D) grad[2 * q + 1][rr] = g.y;
                }
            }
            vel[0] = M0p[0].x;
            vel[1] = M0p[0].y;
            if constexpr (D == 3) vel[2] = M0p[1].x;
            div = grad[0][0] + grad[1][1];
            if constexpr (D == 3) div += grad[2][2];
        }
        // ---- particle update ----
        const Material &mat = s.materials[fl & FLAG_MAT_MASK];
        const uint32_t tag = MODEL >= 0 ? (uint32_t)MODEL : mat.tag;
        const bool fluid = tag == SLOSH_MODEL_FLUID_TAIT;
        const bool sand = tag == SLOSH_MODEL_SAND_LINEAR || tag == SLOSH_MODEL_SAND_NEO_HOOKEAN;
        float len2 = 0.f;
#pragma unroll
        for (int k = 0; k < D; ++k) len2 += vel[k] * vel[k];
        // |v| > h / dt, tested on the squares first (sqrt is monotone; the
        // square root is taken only for a particle near the clamp).  When
        // (h / dt)^2 overflows, every particle takes the exact test.
        const float vclamp2 = vmax * vmax * (1.0f - 4e-7f);
        if (len2 > vclamp2 || isinf(vclamp2)) {
            const float len = sqrtf(len2);
            if (len > vmax)
#pragma unroll
                for (int k = 0; k < D; ++k) vel[k] = vel[k] / len * h / dt;
        }
        const float4 ps = (s.has_sand | s.has_damping) ? st_ps[buf][tid] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (s.has_damping) {
            const float dmp = 1.0f + ps.w * dt;
#pragma unroll
            for (int k = 0; k < D; ++k) vel[k] = vel[k] / dmp;
        }
        const bool fixed = (fl & FLAG_FIXED) != 0;
        if (fixed)
#pragma unroll
            for (int k = 0; k < D; ++k) vel[k] = 0.f;
        float nx[D];
#pragma unroll
        for (int k = 0; k < D; ++k) nx[k] = x[k] + vel[k] * dt;
        float F[D][D];
        {
            float4 fv[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) fv[q] = st_fq[buf][q][tid];
            mat_from<D>(fv, __uint_as_float(fo.w), F);
        }
        if (!fluid) {
            // F <- F + (dt grad v) F, row by row in column pairs (c, c + 1)
            float Fn[D][D];
#pragma unroll
            for (int rr = 0; rr < D; ++rr) {
                float2 g[D];
#pragma unroll
                for (int k = 0; k < D; ++k) g[k] = pair(grad[rr][k] * dt);
#pragma unroll
                for (int c = 0; c < D; c += 2) {
                    const bool two = c + 1 < D;
                    auto col = [&](int k) { return make_float2(F[k][c], two ? F[k][c + 1] : 0.f); };
                    float2 acc = __fmul2_rn(col(0), g[0]);
#pragma unroll
                    for (int k = 1; k < D; ++k) acc = __ffma2_rn(col(k), g[k], acc);
                    const float2 r = __fadd2_rn(make_float2(F[rr][c], two ? F[rr][c + 1] : 0.f), acc);
                    Fn[rr][c] = r.x;
                    if (two) Fn[rr][c + 1] = r.y;
                }
            }
#pragma unroll
            for (int rr = 0; rr < D; ++rr)
#pragma unroll
                for (int c = 0; c < D; ++c) F[rr][c] = Fn[rr][c];
        } else {
            const float f0 = F[0][0];
            const float nf = f0 + f0 * div * dt;
#pragma unroll
            for (int rr = 0; rr < D; ++rr)
#pragma unroll
                for (int c = 0; c < D; ++c) F[rr][c] = (rr == c) ? nf : 0.f;
        }
        if (fixed)
#pragma unroll
            for (int rr = 0; rr < D; ++rr)
#pragma unroll
                for (int c = 0; c < D; ++c) grad[rr][c] = 0.f;
        float st[3] = {0.f, 0.f, 0.f};
        if (sand) {
            st[0] = ps.x;
            st[1] = ps.y;
            st[2] = ps.z;
        }
        float tau[D][D];
        model_update<D>(mat, tag, F, st, tau, &s.ctr->n_svd_fp64);
        const float v0 = __uint_as_float(fo.z);
        const float coef = v0 * inv_d * dt;
        bool finite = true;
#pragma unroll
        for (int k = 0; k < D; ++k) finite = finite && (nx[k] == nx[k]);
        // The particle is stored at its canonical position o in the
        // output buffers (contiguous, coalesced writes).
        const size_t o = (size_t)first + e;
        float Cn[D][D];
        float4 np4 = p;
        if (finite && det<D>(F) > 0.f) {
            np4.x = nx[0];
            np4.y = nx[1];
            if constexpr (D == 3) np4.z = nx[2];
#pragma unroll
            for (int rr = 0; rr < D; ++rr)
#pragma unroll
                for (int c = 0; c < D; ++c) Cn[rr][c] = products_diff(grad[rr][c], m, tau[rr][c], coef);
        } else {
            fl &= ~FLAG_ENABLED;
            m = 0.f;
            np4.w = 0.f;
#pragma unroll
            for (int rr = 0; rr < D; ++rr)
#pragma unroll
                for (int c = 0; c < D; ++c) {
                    F[rr][c] = (rr == c) ? 1.f : 0.f;
                    Cn[rr][c] = 0.f;
                }
#pragma unroll
            for (int k = 0; k < D; ++k) vel[k] = 0.f;
        }
        float4 cv[Q], fv[Q];
        const float c22 = mat_split<D>(Cn, cv), f22 = mat_split<D>(F, fv);
        s.out_pm[o] = np4;
        if constexpr (!B) {
            if (s.reuse && (st_fo[buf][tid].x & FLAG_ENABLED)) note_cell_change<D, POW2>(s, r, st_pm[buf][tid], np4, h, inv_h, h_pow2);
        }
        s.out_vv[o] = make_float4(vel[0], vel[1], D == 3 ? vel[D - 1] : 0.f, c22);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            s.out_cq[q * n + o] = cv[q];
            s.out_fq[q * n + o] = fv[q];
        }
        s.out_fo[o] = make_uint4(fl, fo.y, fo.z, __float_as_uint(f22));
        s.out_oid[o] = fo.y;
        if (s.has_sand | s.has_damping) s.out_ps[o] = make_float4(st[0], st[1], st[2], ps.w);
    }
    cp_async_wait<0>();
}

template <int D, int NT, bool B = false, bool POW2 = false, int MODEL = -1>
__device__ __forceinline__ void g2p_update_body(const DevScene &s, Cta g, G2pSmem<D, NT> &sm) {
    const uint32_t nb = s.ctr->n_blocks;
    const uint32_t tid = threadIdx.x;
    if (s.clear_tail) clear_next_map<B>(s, g.id * NT + tid, g.n * NT);
    // blocks are taken from a queue, one atomic a block
    uint32_t &next_r = sm.next_r;
    for (;;) {
        __syncthreads();  // every thread has read next_r, and the last block's tile
        if (tid == 0) {
            if (B && s.g2p_class >= 0) {  // this launch's class of the batch's blocks
                const uint32_t cls = (uint32_t)s.g2p_class;
                const uint32_t q = atomicAdd(&s.g2p_counts[G2P_CLASSES + cls], 1u);
                next_r = q < s.g2p_counts[cls] ? s.g2p_lists[(size_t)cls * s.cap + q] : nb;
            } else {
                next_r = atomicAdd(&s.ctr->g2p_next, 1u);
            }
        }
        __syncthreads();
        const uint32_t r = next_r;
        if (r >= nb) break;
        const uint32_t np = s.bnp[r];
        if (np == 0) continue;
        g2p_block<D, NT, B, POW2, MODEL>(s, sm, r, np, tid, tid, NT, [] { __syncthreads(); });
    }
}
template <int D, int NT, bool B = false, bool POW2 = false, int MODEL = -1>
__global__ void __launch_bounds__(NT, 512 / NT) k_g2p_update(DevScene s) {
    pdl_enter();
    __shared__ G2pSmem<D, NT> sm;
    g2p_update_body<D, NT, B, POW2, MODEL>(s, launch_cta(), sm);
}

// Rigid-body update (shaders/slosh/solver/rigid_impulses.slang:72-121) with
// integrate_velocity (shaders/slosh/rbd/dynamics/body.slang:117-130).  The
// incremental impulse slosh applies here is never written by any of its
// kernels, so velocity capping (guarded by a non-zero impulse) never runs.
// The last kernel of the substep: it also resets the grid-build counters for
// the next substep.
// Multi-scene batches (B): bodies of all scenes in one table, each with its
// scene's dt and gravity (bodies of dropped scenes are left alone), and the
// particle count in storage becomes this substep's sorted count.
template <int D, bool B = false> __device__ __forceinline__ void move_body(const DevScene &s, uint32_t id) {
    DevBody b = s.bodies[id];
    float dt = s.dt, grav[3] = {s.gravity[0], s.gravity[1], s.gravity[2]};
    if constexpr (B) {
        const SceneRec &rec = s.scenes[b.scene];
        if (!rec.live) return;
        dt = rec.dt;
        for (int k = 0; k < 3; ++k) grav[k] = rec.gravity[k];
    }
    if (b.coupling == SLOSH_COUPLING_TWO_WAY) {
        // apply_impulse (shaders/slosh/rbd/dynamics/body.slang:62-70) of the
        // impulse the grid gave this substep, and the velocity caps of
        // rigid_impulses.slang:99-111; the sums restart at zero
        float h = s.h;
        if constexpr (B) h = s.scenes[b.scene].h;
        unsigned long long *acc = s.body_imp + (size_t)id * 6u;
        float jl[3] = {0.f, 0.f, 0.f}, ja[3] = {0.f, 0.f, 0.f};
        for (int k = 0; k < 3; ++k) {
            jl[k] = (float)((double)(long long)acc[k] / IMPULSE_UNITS);
            ja[k] = (float)((double)(long long)acc[3 + k] / IMPULSE_UNITS);
            acc[k] = 0ull;
            acc[3 + k] = 0ull;
        }
        for (int k = 0; k < D; ++k) b.linvel[k] += b.inv_mass[k] * jl[k];
        if constexpr (D == 3) {
            float R[3][3], Iw[9];
            quat_matrix(b.rot, R);
            rotate_tensor(R, b.inv_inertia, Iw, true);
            for (int i = 0; i < 3; ++i) b.angvel[i] += fmaf(Iw[i * 3 + 2], ja[2], products_sum(Iw[i * 3], ja[0], Iw[i * 3 + 1], ja[1]));
        } else {
            b.angvel[0] += b.inv_inertia[0] * ja[0];
        }
        const bool pushed = jl[0] != 0.f || jl[1] != 0.f || jl[2] != 0.f || ja[0] != 0.f || ja[1] != 0.f || ja[2] != 0.f;
        if (pushed) {
            const float lin_limit = 0.1f * h / dt, ang_limit = 1.0f;
            float l2 = 0.f, a2 = 0.f;
            for (int k = 0; k < D; ++k) l2 += b.linvel[k] * b.linvel[k];
            for (int k = 0; k < (D == 3 ? 3 : 1); ++k) a2 += b.angvel[k] * b.angvel[k];
            const float ln = sqrtf(l2), an = sqrtf(a2);
            if (ln > lin_limit)
                for (int k = 0; k < D; ++k) b.linvel[k] = b.linvel[k] * (lin_limit / ln);
            if (an > ang_limit)
                for (int k = 0; k < (D == 3 ? 3 : 1); ++k) b.angvel[k] = b.angvel[k] * (ang_limit / an);
        }
    }
    float init_com[3] = {0.f, 0.f, 0.f};
    pose_mul_pt<D>(b, b.local_com, init_com);
    if constexpr (D == 3) {
        const float sa[3] = {b.angvel[0] * dt, b.angvel[1] * dt, b.angvel[2] * dt};
        const float ang = sqrtf(fmaf(sa[2], sa[2], products_sum(sa[0], sa[0], sa[1], sa[1])));
        float dq[4] = {0.f, 0.f, 0.f, 1.f};
        if (ang > 0.f) {
            const float sc = sinf(ang * 0.5f) / ang;
            dq[0] = sa[0] * sc;
            dq[1] = sa[1] * sc;
            dq[2] = sa[2] * sc;
            dq[3] = cosf(ang * 0.5f);
        }
        const float rel[3] = {b.tra[0] - init_com[0], b.tra[1] - init_com[1], b.tra[2] - init_com[2]};
        float rr[3];
        quat_rotate(dq, rel, rr);
        for (int k = 0; k < 3; ++k) b.tra[k] = fmaf(b.linvel[k], dt, fmaf(rr[k], b.scale, init_com[k]));
        const float *q = b.rot;
        float nq[4];
        nq[0] = products_sum(dq[3], q[0], dq[0], q[3]) + products_diff(dq[1], q[2], dq[2], q[1]);
        nq[1] = products_diff(dq[3], q[1], dq[0], q[2]) + products_sum(dq[1], q[3], dq[2], q[0]);
        nq[2] = products_sum(dq[3], q[2], dq[0], q[1]) + products_diff(dq[2], q[3], dq[1], q[0]);
        nq[3] = products_diff(dq[3], q[3], dq[0], q[0]) - products_sum(dq[1], q[1], dq[2], q[2]);
        const float n2 = products_sum(nq[0], nq[0], nq[1], nq[1]) + products_sum(nq[2], nq[2], nq[3], nq[3]);
        const float f = 0.5f * (3.0f - n2);
        for (int k = 0; k < 4; ++k) b.rot[k] = nq[k] * f;
    } else {
        const float a = b.angvel[0] * dt;
        const float c = cosf(a), sn = sinf(a);
        const float rel0 = b.tra[0] - init_com[0], rel1 = b.tra[1] - init_com[1];
        const float r0 = products_diff(c, rel0, sn, rel1), r1 = products_sum(sn, rel0, c, rel1);
        b.tra[0] = fmaf(b.linvel[0], dt, fmaf(r0, b.scale, init_com[0]));
        b.tra[1] = fmaf(b.linvel[1], dt, fmaf(r1, b.scale, init_com[1]));
        const float nc = products_diff(c, b.rot[0], sn, b.rot[1]), ns = products_sum(sn, b.rot[0], c, b.rot[1]);
        b.rot[0] = nc;
        b.rot[1] = ns;
    }
    for (int k = 0; k < D; ++k) b.linvel[k] = b.linvel[k] + grav[k] * ((b.inv_mass[k] != 0.f) ? 1.f : 0.f) * dt;
    s.bodies[id] = b;
}
template <int D, bool B = false> __device__ __forceinline__ void rigid_body(const DevScene &s, uint32_t id) {
    if (id == 0 && s.clear_tail) {
        const uint32_t nb = s.ctr->n_blocks;
        s.ctr->last_n_blocks = nb;
        if (!build_skipped(s)) s.ctr->last_n_primary = min(s.ctr->n_primary, s.cap);
        if (s.reuse) s.ctr->rebuild[s.par] = 0u;  // read by this substep only; G2P set the next one's
        if constexpr (B)
            if (s.g2p_lists)
                for (uint32_t c = 0; c < G2P_CLASSES; ++c) s.g2p_counts[c] = 0u;  // the next block setup's lists
        s.ctr->n_primary = 0u;
        s.ctr->n_extra = 0u;
        s.ctr->n_blocks = 0u;
        if constexpr (B) *s.n_dev = nb ? s.bfirst[nb - 1] + s.bnp[nb - 1] : 0u;
    }
    if (id < s.n_bodies) move_body<D, B>(s, id);
}
template <int D, bool B = false> __global__ void k_rigid(DevScene s) {
    pdl_enter();
    rigid_body<D, B>(s, blockIdx.x * blockDim.x + threadIdx.x);
}

}  // namespace slosh
