// Substeps of a small scene as one persistent, cooperative launch.
//
// A scene of tens of thousands of particles has one or two blocks an SM: each
// stage of the substep is a few microseconds of latency, and launching the
// stages one after another (13 kernels in a graph) costs more than running
// them.  Here up to one CTA an SM runs all stages of several substeps, with a
// grid barrier where a stage needs the whole grid's results of the one before:
//
//   touch     particles counted per cell, their blocks and the blocks' +1
//             neighbours inserted                       (k_touch, k_neighbors)
//   rank      a warp per block: its rank and first entry, as the number of
//             smaller keys and the particles in their blocks; its cells
//                              (k_hist_scan .. k_block_setup, k_block_scan).
//             Above STEPS_KEYS blocks all pairs are too many (24,000 blocks:
//             2,970 us a substep): the separate kernels' key histogram, with
//             four barriers more (255 us)
//   scatter   the permutation; the blocks' neighbour ranks     (k_scatter)
//   transfer  four warps per block: canonical order, then P2G  (k_canon, k_p2g)
//   update    the grid nodes                              (k_grid_update)
//   particles a warp per 32 particles of a block, G2P and the particle
//             update; the next map cleared; the bodies moved
//                                                 (k_g2p_update, k_rigid)
//
// The stages are the stand-alone kernels' own device functions (or, in touch
// and rank, leave the same arrays), so the results are theirs bit for bit.
// Six barriers of about 1.4 us replace thirteen launches.  What a substep
// takes then is latency: at 68,921 sand particles, microseconds with each
// stage's barrier, touch 5, rank 5, scatter 6, transfer 15 (the chain of one
// full block: 512 particles, a dozen deep in each cell), update 5, particles
// 15 (every warp runs the update once, from a cold instruction cache).
// Measured, graph of separate kernels against this, us a substep: 8,000
// particles 50 and 38, the 62,628-particle 2D dam break 48 and 30, the
// three-model scene of 59,049 62 and 48, the 68,921-particle sand job 62 and 52.
#pragma once

#include "fused.cuh"

namespace slosh {

constexpr int STEPS_THREADS = 512;
constexpr uint32_t STEPS_GROUPS = STEPS_THREADS / 128;  // groups of four warps: a P2G block, a G2P CTA
constexpr uint32_t STEPS_KEYS = 4096;                   // block keys ranked all against all, from shared memory

// The scene as substeps of either parity see it.
struct ScenePair {
    DevScene s[2];
};

// A block's entries while a group puts them in canonical order.
constexpr uint32_t STEPS_SORT = 768;  // larger blocks are sorted in global memory
struct StepsSort {
    uint32_t id[STEPS_SORT], from[STEPS_SORT], perm[STEPS_SORT];
    uint32_t cell[CELLS + 1];  // first entry of each cell, and the end
};
// P2G with eight particles of a cell staged: at one or two warps a scheduler the
// copies' latency is not hidden by other warps.
template <int D> union StepsSmem {
    struct {
        P2gSmem<D, 8> p2g;
        StepsSort sort;
    } t[STEPS_GROUPS];
    G2pSmem<D, 32> g2p[STEPS_THREADS / 32];
    struct {
        uint32_t key[STEPS_KEYS], count[STEPS_KEYS];
    } rank;
};

// Barrier over the launch's CTAs (all resident: a cooperative launch).  The
// ticket counts arrivals of the whole launch, round k ends at k CTAs times
// k; the launch's last CTA to leave sets it back to zero.  Bounded like the
// batch's grid barrier: a CTA that waits longer than BARRIER_NS sets
// ERR_BARRIER and returns false, and so does, at its next look, every CTA
// that waits for it.
__device__ __forceinline__ bool steps_barrier(const DevScene &s, uint32_t &round, uint32_t *flag) {
    ++round;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t *ticket = &s.ctr->steps_ticket;
        const uint32_t target = round * (gridDim.x + s.bar_extra);
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ticket) : "memory");
        uint32_t ok = 1u, seen;
        unsigned long long t0 = 0;
        for (uint32_t it = 1;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(ticket) : "memory");
            if (seen >= target) break;
            if ((it & 255u) == 0u) {
                const unsigned long long now = global_ns(), limit = s.bar_ns ? s.bar_ns : BARRIER_NS;
                if (t0 == 0) t0 = now;
                if ((*(volatile uint32_t *)s.err & ERR_BARRIER) || now - t0 > limit || it >= BARRIER_SPINS) {
                    atomicOr(s.err, ERR_BARRIER);
                    ok = 0u;
                    break;
                }
            }
        }
        *flag = ok;
    }
    __syncthreads();
    return *flag != 0u;
}

// touch_body, with the +1 neighbours of a block inserted by the warp that
// brings its first particle, all blocks appended to one list, and the blocks'
// particle counts.
template <int D> __device__ __forceinline__ void steps_touch(const DevScene &s) {
    constexpr uint32_t NN = Geo<D>::NASSOC - 1, AT_ONCE = 32u / NN;
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t chunk = (((s.count + warps - 1) / warps) + 31u) & ~31u;
    const uint32_t begin = wid * chunk, end = min(s.count, begin + chunk);
    // appends the lanes' new blocks, one atomic for the warp
    auto append = [&](bool fresh, uint32_t key, uint32_t slot) {
        const unsigned who = __ballot_sync(FULL_MASK, fresh);
        if (who == 0u) return;
        const int first = __ffs(who) - 1;
        uint32_t j = 0;
        if ((int)lane == first) j = atomicAdd(&s.ctr->n_extra, (uint32_t)__popc(who));
        j = __shfl_sync(FULL_MASK, j, first) + __popc(who & lanemask_lt());
        if (!fresh) return;
        if (j < s.cap) {
            s.blist_key[j] = key;
            s.blist_slot[j] = slot;
        } else {
            atomicOr(s.err, ERR_BLOCK_OVERFLOW);
        }
    };
    uint32_t last_key = NONE, last_slot = NONE;
    for (uint32_t base = begin; base < end; base += 32) {
        const uint32_t i = base + lane;
        const bool valid = i < end;
        const unsigned mask = __ballot_sync(FULL_MASK, valid);
        const float4 p = valid ? s.pm[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float x[3] = {p.x, p.y, p.z};
        const CellLoc<D> c = locate<D>(x, s.h, s.inv_h, s.h_pow2);
        const uint32_t key = pack_key<D>(c.block);
        const unsigned peers = __match_any_sync(FULL_MASK, key) & mask;
        const int leader = __ffs(peers) - 1;  // -1: no valid lane with this key
        uint32_t slot = NONE;
        bool fresh = false, first = false;
        if ((int)lane == leader) {
            if (key == last_key && last_slot != NONE) slot = last_slot;
            else slot = hash_insert(s.hkeys, s.hcap, key, fresh, s.err);
            first = slot != NONE && atomicAdd(&s.slot_total[slot], (uint32_t)__popc(peers)) == 0u;
        }
        __syncwarp();
        append(fresh, key, slot);
        // the neighbours of the blocks that got their first particle, a lane each
        unsigned todo = __ballot_sync(FULL_MASK, first);
        while (todo != 0u) {
            const uint32_t mine = lane / NN;
            unsigned rest = todo;
            for (uint32_t q = 0; q < mine; ++q) rest &= rest - 1u;  // drop the lower `mine` blocks
            const bool act = mine < AT_ONCE && rest != 0u;
            const int src = act ? __ffs(rest) - 1 : 0;
            int o[D], b[D];
            assoc_offset<D>((int)(lane % NN) + 1, o);
#pragma unroll
            for (int k = 0; k < D; ++k) b[k] = __shfl_sync(FULL_MASK, c.block[k], src) + o[k];
            const uint32_t nk = pack_key<D>(b);
            bool fresh_n = false;
            uint32_t at = NONE;
            if (act) at = hash_insert(s.hkeys, s.hcap, nk, fresh_n, s.err);
            __syncwarp();
            append(fresh_n, nk, at);
            for (uint32_t q = 0; q < AT_ONCE; ++q) todo &= todo - 1u;
        }
        slot = __shfl_sync(FULL_MASK, slot, max(leader, 0));
        const int top = 31 - __clz(mask);
        last_key = __shfl_sync(FULL_MASK, key, top);
        last_slot = __shfl_sync(FULL_MASK, slot, top);
        const uint32_t bin = (slot == NONE || !valid) ? NONE : (slot << 6) | cell_index<D>(c.local);
        const unsigned peers2 = __match_any_sync(FULL_MASK, bin);
        if (bin != NONE && (int)lane == __ffs(peers2) - 1) atomicAdd(&s.slot_counts[bin], (uint32_t)__popc(peers2));
        if (valid) s.pslot[i] = bin;
    }
}

// Ranks, first entries and cells of up to STEPS_KEYS listed blocks, a warp a
// block: the smaller keys, and the particles in their blocks, counted over all
// keys in shared memory.
template <int D> __device__ __forceinline__ void steps_rank(const DevScene &s, StepsSmem<D> &sm, uint32_t total) {
    const uint32_t lane = lane_id();
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    if (blockIdx.x == 0 && threadIdx.x == 0) s.ctr->n_blocks = total;
    if (blockIdx.x >= total) return;  // no warp of this CTA has a block
    for (uint32_t q = threadIdx.x; q < total; q += blockDim.x) {
        sm.rank.key[q] = s.blist_key[q];
        sm.rank.count[q] = s.slot_total[s.blist_slot[q]];
    }
    __syncthreads();
    for (uint32_t j = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; j < total; j += warps) {
        const uint32_t key = sm.rank.key[j], slot = s.blist_slot[j];
        uint32_t r = 0, first = 0;
#pragma unroll 4
        for (uint32_t q = lane; q < total; q += 32u) {
            const bool less = sm.rank.key[q] < key;
            r += less ? 1u : 0u;
            first += less ? sm.rank.count[q] : 0u;
        }
        r = __reduce_add_sync(FULL_MASK, r);
        first = __reduce_add_sync(FULL_MASK, first);
        const uint32_t np = block_cells(s, r, slot);
        if (lane == 0) {
            s.bkey[r] = key;
            s.bslot[r] = slot;
            s.bfirst[r] = first;
            s.hvals[slot] = r | (np ? 0u : RANK_EXTRA);
            if (np) atomicAdd(&s.ctr->n_primary, 1u);
        }
    }
}

// The same for more blocks, in time linear in them: by the key histogram and
// its bins, as the separate kernels rank (k_neighbors' counts, k_hist_scan,
// k_bin_scatter, k_rank, k_block_scan), with four more barriers.  The histogram
// is clear on entry; steps_clear_hist clears it once the ranks are used.
template <int D>
__device__ __forceinline__ bool steps_rank_many(const DevScene &s, uint32_t total, uint32_t &round, uint32_t *flag) {
    const uint32_t lane = lane_id();
    const uint32_t threads = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (t0 == 0) s.ctr->n_blocks = total;
    for (uint32_t base = t0 - lane; base < total; base += threads) {
        const uint32_t t = base + lane;
        const uint32_t key = t < total ? s.blist_key[t] : 0u, coarse = t < total ? key >> 26 : NONE;
        if (t < total) atomicAdd(&s.hist[key >> 16], 1u);
        const unsigned peers = __match_any_sync(FULL_MASK, coarse);
        if (coarse != NONE && (int)lane == __ffs(peers) - 1) atomicAdd(&s.hist_coarse[coarse], (uint32_t)__popc(peers));
    }
    if (!steps_barrier(s, round, flag)) return false;
    for (uint32_t c = blockIdx.x; c < HIST_COARSE; c += gridDim.x) hist_scan_part<STEPS_THREADS>(s, c);
    if (!steps_barrier(s, round, flag)) return false;
    for (uint32_t t = t0; t < total; t += threads) {
        const uint32_t key = s.blist_key[t], pos = atomicAdd(&s.hist_start[key >> 16], 1u);
        s.tmp_key[pos] = key;
        s.tmp_slot[pos] = s.blist_slot[t];
    }
    if (!steps_barrier(s, round, flag)) return false;
    for (uint32_t t = t0 >> 5; t < total; t += threads >> 5) {
        const uint32_t key = s.tmp_key[t], slot = s.tmp_slot[t];
        const uint32_t end = s.hist_start[key >> 16], start = end - s.hist[key >> 16];  // advanced by the scatter
        uint32_t r = 0;
#pragma unroll 4
        for (uint32_t q = start + lane; q < end; q += 32u) r += s.tmp_key[q] < key ? 1u : 0u;
        r = start + __reduce_add_sync(FULL_MASK, r);
        const uint32_t np = block_cells(s, r, slot);
        if (lane == 0) {
            s.bkey[r] = key;
            s.bslot[r] = slot;
            s.hvals[slot] = r | (np ? 0u : RANK_EXTRA);
            if (np) atomicAdd(&s.ctr->n_primary, 1u);
        }
    }
    if (!steps_barrier(s, round, flag)) return false;
    if (blockIdx.x == 0) block_scan_body<STEPS_THREADS>(s);
    return true;
}
__device__ __forceinline__ void steps_clear_hist(const DevScene &s, uint32_t nb) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nb; r += gridDim.x * blockDim.x) {
        const uint32_t key = s.bkey[r];
        s.hist[key >> 16] = 0u;
        s.hist_coarse[key >> 26] = 0u;
    }
}

// The block's part of the permutation in canonical order (cells in order,
// ascending original id in a cell, as k_canon leaves it), by a group of four
// warps: every entry counts the smaller ids of its cell, all side by side.
// Left in sm.perm and written back for G2P.  False for a block that does not
// fit (or whose counts are stale): canon_block sorts that one in place.
template <typename Sync>
__device__ __forceinline__ bool steps_sort(const DevScene &s, StepsSort &sm, uint32_t r, uint32_t t, Sync sync) {
    const uint32_t first = s.bfirst[r], np = s.bnp[r];
    if (np > STEPS_SORT || (size_t)first + np > s.n) return false;
    for (uint32_t e = t; e < np; e += 128u) {
        sm.id[e] = (uint32_t)s.skey[first + e];
        sm.from[e] = s.perm[first + e];
    }
    if (t < CELLS) sm.cell[t] = s.bcell[(size_t)r * CELLS + t];
    if (t == CELLS) sm.cell[CELLS] = np;
    // an entry's cell, read again from its key (a register a round otherwise)
    sync();
    for (uint32_t e = t; e < np; e += 128u) {
        const uint32_t c = (uint32_t)(s.skey[first + e] >> 32) & 63u;
        const uint32_t b0 = sm.cell[c], b1 = min(sm.cell[c + 1], np), id = sm.id[e];
        uint32_t at = b0;
        for (uint32_t q = b0; q < b1; ++q) at += sm.id[q] < id ? 1u : 0u;
        const uint32_t from = sm.from[e];
        sm.perm[at] = from;
        if (at != e) s.perm[first + at] = from;
    }
    sync();
    return true;
}

template <int D, bool POW2, int MODEL>
__global__ void __launch_bounds__(STEPS_THREADS, 1)
    k_scene_steps(const __grid_constant__ ScenePair pair, uint32_t par, uint32_t n_substeps) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t flag;
    StepsSmem<D> &sm = *reinterpret_cast<StepsSmem<D> *>(smem);
    const Cta cta = launch_cta();
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t warps = gridDim.x * (STEPS_THREADS / 32), w0 = warp * gridDim.x + blockIdx.x;
    const uint32_t group = threadIdx.x >> 7, tid = threadIdx.x & 127u;
    const uint32_t groups = gridDim.x * STEPS_GROUPS, g0 = group * gridDim.x + blockIdx.x;
    auto group_sync = [&]() { named_bar_sync(1u + group, 128u); };
    if (*(volatile uint32_t *)pair.s[0].err & ERR_BARRIER) return;  // an earlier launch gave up: its ticket is void
    uint32_t round = 0;
    bool alive = true;
    for (uint32_t k = 0; k < n_substeps; ++k, par ^= 1u) {
        const DevScene &s = pair.s[par & 1u];
        if (k && !(alive = steps_barrier(s, round, &flag))) break;
        steps_touch<D>(s);
        if (!(alive = steps_barrier(s, round, &flag))) break;
        const uint32_t nb = min(s.ctr->n_extra, s.cap);
        if (nb <= STEPS_KEYS) steps_rank<D>(s, sm, nb);
        else if (!(alive = steps_rank_many<D>(s, nb, round, &flag))) break;
        if (!(alive = steps_barrier(s, round, &flag))) break;
        if (nb > STEPS_KEYS) steps_clear_hist(s, nb);
        scatter_body<false>(s, cta);
        for (uint32_t r = w0; r < nb; r += warps) {
            block_neighbors<D, false>(s, r);
            if (lane == 0) s.slot_total[s.bslot[r]] = 0u;
            // the block's 32-particle parts, at places that need no scan:
            // those before block r are at most first / 32 + r
            const uint32_t first = s.bfirst[r], np = s.bnp[r];
            const uint32_t i0 = first / 32u + r, i1 = (first + np) / 32u + r + 1u;
            for (uint32_t q = i0 + lane; q < i1; q += 32u)
                s.items[q] = make_uint2((q - i0) * 32u < np ? r : NONE, q - i0);
        }
        if (!(alive = steps_barrier(s, round, &flag))) break;
        if (nb < s.p2g_coop_below) {
            for (uint32_t r = g0; r < nb; r += groups) {
                auto &t = sm.t[group];
                const bool held = steps_sort(s, t.sort, r, tid, group_sync);
                if (!held) {
                    canon_block(s, r, tid >> 5, 4u);
                    group_sync();
                }
                p2g_group_block<D, false>(s, t.p2g, r, tid, held ? t.sort.perm : nullptr, group_sync);
            }
        } else {
            for (uint32_t r = w0; r < nb; r += warps) {
                canon_block(s, r, 0u, 1u);
                __syncwarp();
                p2g_warp_block<D, false, false>(s, sm.t[group].p2g.w[warp & 3u], r);
            }
        }
        if (!(alive = steps_barrier(s, round, &flag))) break;
        grid_update_body<D>(s, cta);
        if (!(alive = steps_barrier(s, round, &flag))) break;
        // G2P, a warp per 32 particles of a block with a node tile of its
        // own: parts are spread over all SMs, whatever the blocks' sizes
        const uint32_t n_items = s.count / 32u + nb;
        for (uint32_t it = w0; it < n_items; it += warps) {
            const uint2 item = s.items[it];
            if (item.x >= nb) continue;
            const uint32_t r = item.x, e0 = item.y * 32u + lane;
            const uint32_t np = min(s.bnp[r], item.y * 32u + 32u);
            g2p_block<D, 32, false, POW2, MODEL>(s, sm.g2p[warp], r, np, lane, e0, 32u, [] { __syncwarp(); });
            __syncwarp();  // the tile is read; the next part overwrites it
        }
        clear_next_map<false>(s, blockIdx.x * STEPS_THREADS + threadIdx.x, gridDim.x * STEPS_THREADS, false);
        if (blockIdx.x == gridDim.x - 1u && warp == STEPS_THREADS / 32 - 1) {
            if (lane < s.n_bodies) move_body<D>(s, lane);
            if (lane == 0) {
                s.err[1] = nb;
                s.ctr->last_n_blocks = nb;
                s.ctr->last_n_primary = s.ctr->n_primary;
                s.ctr->n_primary = 0u;
                s.ctr->n_extra = 0u;
            }
        }
    }
    // the last CTA to leave sets the ticket back
    __syncthreads();
    if (threadIdx.x == 0 && alive) {
        const DevScene &s = pair.s[0];
        if (atomicAdd(&s.ctr->steps_left, 1u) == gridDim.x - 1u) {
            s.ctr->steps_ticket = 0u;
            s.ctr->steps_left = 0u;
        }
    }
}

}  // namespace slosh
