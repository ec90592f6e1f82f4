// epp_cells.cuh -- cell-list build: bin (atomic counts, linked lists of the cells or slots in them),
// exclusive scan, rank-by-id gather (a counting sort with a deterministic within-cell order).
//
// Replaces the reference's fixed-capacity buckets (NeighbourSearch.jl:12-47, clean! at
// NeighbourSystem.jl:43-54): the counts, offsets and membership of every cell equal the
// reference's bucket counts, their exclusive scan and the buckets sorted by particle id.
#pragma once
#include "epp_math.cuh"

namespace epp {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;   // 2048 cells per tile
constexpr long long kSpinLimit = 1ll << 22;            // bounded look-back wait

__device__ __forceinline__ void set_status(unsigned* status, unsigned bits) {
    if (bits) atomicOr(status, bits);
}

// What a bin pass leaves for the counting sort, per particle i: its cell and its place among its
// cell's particles.  With `head` the particles of a cell form a linked list of count[c] entries from
// head[c] through link[i] = (next, id), in arrival order (the last one's next, like the head of an empty
// cell, is whatever the memory held: the count ends a walk), and only particles of the dead bin (c =
// n_cells), which can be many, take a slot.  Without it all take a slot of their cell, for a scatter pass
// that brings a cell's particles together.  tile[t] counts the particles of scan tile t (2048 cells).
struct BinOut {
    int2* cs;      // (cell, slot: of the dead bin only where there are lists)
    int2* link;    // (next particle of the cell, id)
    int* count;    // [n_cells + 1] zero on entry
    int* head;     // [n_cells], or null
    int* tile;     // [tiles * stride] zero on entry, or null (family 1, whose scan does not go by it)
    int stride;    // ints between two tile counters: a cache line apart where there is room, since the
                   // atomics of one line are served one after the other (binning 955,668 particles in
                   // lattice order: 29 us packed, 15 a line apart)
};

// Adds particle i of id `id` to cell c.  The tile counters are updated once per group of the warp's
// active lanes with one tile (sorted particles: nearly always all of them).
__device__ __forceinline__ void bin_particle(const BinOut& B, int n_cells, int i, int id, int c) {
    if (B.tile) {
        const int t = c / kScanTile;
        const unsigned same = __match_any_sync(__activemask(), t);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&B.tile[t * B.stride], __popc(same));
    }
    int slot = 0;
    if (!B.head || c == n_cells) {
        slot = atomicAdd(&B.count[c], 1);
    } else {
        atomicAdd(&B.count[c], 1);
        B.link[i] = make_int2(atomicExch(&B.head[c], i), id);
    }
    B.cs[i] = make_int2(c, slot);
}

// Per-call search, pass 1 (insertParticlesIntoCells!, NeighbourSearch.jl:12-47):
//   immovable particles with a cell keep it; others are binned from their position;
//   particles outside the domain are killed (dead bin = n_cells).
// Block 0 also clears the look-back state of the scan that lists occupied cells (n_scan_words > 0).
template <int D>
__global__ void k_bin_count(int n, DevDomain dom, State s, BinOut B, unsigned* status, unsigned long long* scan_state,
                            int n_scan_words) {
    if (blockIdx.x == 0)
        for (int t = threadIdx.x; t < n_scan_words; t += blockDim.x) scan_state[t] = 0ull;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int c = s.cell[i];
    if (c != dom.n_cells) {
        int tm = s.tagm[i];
        if (movable_of(tm) || c < 0) {
            c = cell_of<D>(dom, s.xh[i], inst_of(tm));
            if (c < 0) {
                c = dom.n_cells;
                set_status(status, EPP_STATUS_KILLED);
            }
            s.cell[i] = c;
        }
    }
    bin_particle(B, dom.n_cells, i, s.id[i], c);
}

// What a scan by tile counters resets for the bin pass after the next: the buffer not in use (the two
// alternate).
struct ScanReset {
    int* tile;        // [tiles * stride]
    int stride;
};

// The tile counters as their exclusive sums, in place, by one block: for grids of so many tiles that each
// adding up all counters before its own is the longer way.
constexpr int kPrefixThreads = 1024, kPrefixItems = 4;
static __global__ void __launch_bounds__(kPrefixThreads) k_tile_prefix(int tiles, int* tile, int stride) {
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;   // of the chunks before, in every thread
    for (int t0 = 0; t0 < tiles; t0 += kPrefixThreads * kPrefixItems) {
        const int t = t0 + threadIdx.x * kPrefixItems;
        int v[kPrefixItems], sum = 0;
#pragma unroll
        for (int k = 0; k < kPrefixItems; ++k) v[k] = t + k < tiles ? tile[(size_t)(t + k) * stride] : 0;
#pragma unroll
        for (int k = 0; k < kPrefixItems; ++k) sum += v[k];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        const int w = s_warp[lane];
        int run = carry + incl - sum + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0);
        carry += __reduce_add_sync(0xffffffffu, w);
#pragma unroll
        for (int k = 0; k < kPrefixItems; ++k) {
            if (t + k < tiles) tile[(size_t)(t + k) * stride] = run;
            run += v[k];
        }
        __syncthreads();   // s_warp is written again
    }
}

// Exclusive scan over m = n_cells + 1 counts (the last is the dead bin) from the tile counters of the
// bin pass: start[0..m], with the counts cleared for the next binning pass.  A tile sums the counters
// before it itself, or (PREFIX) reads their sum, so no tile waits for another (the look-back scan below
// is a chain through its tiles: 10 us against 4 at 335,336 cells).  A cell of the domain with more than
// max_cell > 0 particles sets EPP_STATUS_CELL_OVERFLOW.
template <bool PREFIX>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(int m, int* count, const int* tile, int* start,
                                                                   ScanReset R, int max_cell, unsigned* status) {
    __shared__ int s_sum[kScanThreads / 32], s_warp[kScanThreads / 32];
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int base = t * kScanTile + threadIdx.x * kScanItems;
    const bool full = base + kScanItems <= m;   // the thread's 8 cells are all in range (aligned)
    int v[kScanItems];
    if (full) {
        const int4 a = reinterpret_cast<const int4*>(count + base)[0];
        const int4 b = reinterpret_cast<const int4*>(count + base)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < m ? count[base + k] : 0;
    }
    int before = 0;   // particles of the tiles before this one
    if (PREFIX) {
        if (threadIdx.x == 0) before = tile[t * R.stride];
    } else {
        for (int q = threadIdx.x; q < t; q += kScanThreads) before += tile[q * R.stride];
    }
    if (threadIdx.x == 0) R.tile[t * R.stride] = 0;
    if (full) {
        reinterpret_cast<int4*>(count + base)[0] = make_int4(0, 0, 0, 0);
        reinterpret_cast<int4*>(count + base)[1] = make_int4(0, 0, 0, 0);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < m) count[base + k] = 0;
    }
    int sum = 0;
    bool over = false;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        sum += v[k];
        over = over || (max_cell > 0 && base + k < m - 1 && v[k] > max_cell);
    }
    if (over) set_status(status, EPP_STATUS_CELL_OVERFLOW);
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 31) {
        s_warp[warp] = incl;
        s_sum[warp] = before;
    }
    __syncthreads();
    int run = incl - sum;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) run += s_sum[w] + (w < warp ? s_warp[w] : 0);
    int out[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        out[k] = run;
        run += v[k];
        if (base + k == m - 1) start[m] = run;
    }
    if (full) {
        reinterpret_cast<int4*>(start + base)[0] = make_int4(out[0], out[1], out[2], out[3]);
        reinterpret_cast<int4*>(start + base)[1] = make_int4(out[4], out[5], out[6], out[7]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < m) start[base + k] = out[k];
    }
}

// The same for the cell-centric pair passes, which also need the occupied cells: single-pass scan with
// decoupled look-back over m = n_cells + 1 counts (the last is the dead bin).  Writes start[0..m], the list
// of occupied cells occ[0..n_occ) in cell order (meta[0] = n_occ) and clears the counts for the next binning pass.  Tiles take a ticket in
// launch order so every predecessor is already running; the wait on a predecessor is bounded
// and reports EPP_STATUS_SPIN_TIMEOUT instead of hanging.
// scan_state layout: [0] ticket, [1 + t] status word of tile t:
//   (flag << 62) | (occupied cells << 31) | particles,  flag 1 = aggregate, 2 = inclusive prefix.
__device__ __forceinline__ unsigned long long pack_status(unsigned long long flag,
                                                          unsigned long long v) {
    // v = (occ << 32) | count  ->  status word
    return (flag << 62) | ((v >> 32) << 31) | (v & 0x7fffffffull);
}
__device__ __forceinline__ unsigned long long unpack_status(unsigned long long w) {
    return (((w >> 31) & 0x7fffffffull) << 32) | (w & 0x7fffffffull);
}

static __global__ void __launch_bounds__(kScanThreads) k_scan(int m, int* count, int* start, int* occ,
                                                       int* meta, unsigned long long* scan_state, int max_cell,
                                                       unsigned* status) {
    __shared__ int s_tile;
    __shared__ unsigned long long s_warp[kScanThreads / 32];
    __shared__ unsigned long long s_prefix;
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(&scan_state[0], 1ull);
    __syncthreads();
    const int tile = s_tile;
    const int base = tile * kScanTile + threadIdx.x * kScanItems;
    const bool full = base + kScanItems <= m;   // the thread's 8 cells are all in range (aligned)
    int v[kScanItems];
    if (full) {   // two 16-byte loads, then zero the counts for the next step
        const int4 a = reinterpret_cast<const int4*>(count + base)[0];
        const int4 b = reinterpret_cast<const int4*>(count + base)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        reinterpret_cast<int4*>(count + base)[0] = make_int4(0, 0, 0, 0);
        reinterpret_cast<int4*>(count + base)[1] = make_int4(0, 0, 0, 0);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            v[k] = base + k < m ? count[base + k] : 0;
            if (base + k < m) count[base + k] = 0;
        }
    }
    unsigned long long tsum = 0;   // (occupied << 32) | particles
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int idx = base + k;
        tsum += (unsigned long long)v[k] + ((idx < m - 1 && v[k] > 0) ? (1ull << 32) : 0ull);
        if (max_cell > 0 && idx < m - 1 && v[k] > max_cell) set_status(status, EPP_STATUS_CELL_OVERFLOW);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        unsigned long long w = lane < kScanThreads / 32 ? s_warp[lane] : 0ull;
        unsigned long long wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < kScanThreads / 32) s_warp[lane] = wi - w;   // exclusive warp offsets
        const unsigned long long total = __shfl_sync(0xffffffffu, wi, kScanThreads / 32 - 1);   // block total
        unsigned long long prefix = 0;
        if (tile == 0) {
            if (lane == 0) atomicExch(&scan_state[1], pack_status(2, total));
        } else {
            if (lane == 0) atomicExch(&scan_state[1 + tile], pack_status(1, total));
            // decoupled look-back, 32 predecessors per round: lane l reads tile p - l; the round
            // ends at the nearest tile with its inclusive prefix published (flag 2), summing the
            // aggregates (flag 1) of the tiles in between; waits (bounded) while any of those has
            // published nothing yet
            volatile unsigned long long* st = scan_state + 1;
            int p = tile - 1;
            long long spins = 0;
            for (;;) {
                const int q = p - lane;
                const unsigned long long w2 = q >= 0 ? st[q] : (2ull << 62);   // before tile 0: inclusive 0
                const unsigned flag = (unsigned)(w2 >> 62);
                const unsigned incl_mask = __ballot_sync(0xffffffffu, flag == 2);
                const unsigned zero_mask = __ballot_sync(0xffffffffu, flag == 0);
                const unsigned need = incl_mask ? ((incl_mask & (0u - incl_mask)) << 1) - 1u : 0xffffffffu;
                if (zero_mask & need) {
                    if (++spins > kSpinLimit) {
                        if (lane == 0) atomicOr(status, EPP_STATUS_SPIN_TIMEOUT);
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                unsigned long long x = ((need >> lane) & 1u) ? unpack_status(w2) : 0ull;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                prefix += x;
                if (incl_mask) break;
                p -= 32;
            }
            if (lane == 0) {
                __threadfence();
                atomicExch(&scan_state[1 + tile], pack_status(2, prefix + total));
            }
        }
        if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    unsigned long long run = s_prefix + s_warp[warp] + incl - tsum;
    int out[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int idx = base + k;
        out[k] = (int)(run & 0xffffffffull);
        const int oc = (int)(run >> 32);
        if (idx < m - 1 && v[k] > 0) occ[oc] = idx;
        run += (unsigned long long)v[k] + ((idx < m - 1 && v[k] > 0) ? (1ull << 32) : 0ull);
        if (idx == m - 1) {
            start[m] = (int)(run & 0xffffffffull);
            meta[0] = (int)(run >> 32);
        }
    }
    if (full) {
        reinterpret_cast<int4*>(start + base)[0] = make_int4(out[0], out[1], out[2], out[3]);
        reinterpret_cast<int4*>(start + base)[1] = make_int4(out[4], out[5], out[6], out[7]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < m) start[base + k] = out[k];
    }
}

// Rank of each particle within its cell by id, from the cell's linked list, and its move to start +
// rank by the mover (src, dst, cell).  A thread per particle in the old order: reads of the state are
// coalesced, writes nearly so (a step moves few particles to another cell), and no scatter pass has to
// bring a cell's particles together first (8 of 32 us of the sort at 515,018 particles).  The dead bin
// keeps arrival order (dead particles never interact).  A destination outside [0, n) can only come from a failed
// scan; it is reported, never written.
__device__ __forceinline__ int sorted_place(int i, int2 cs, int n_cells, int n, const int2* link, const int* head,
                                            const int* start) {
    const int s = start[cs.x];
    if (cs.x == n_cells) return s + cs.y;
    const int id = link[i].y;
    int rank = 0, j = head[cs.x];
    for (int left = start[cs.x + 1] - s; left > 0 && (unsigned)j < (unsigned)n; --left) {   // the cell's particles
        const int2 e = link[j];
        rank += e.y < id;
        j = e.x;
    }
    return s + rank;
}

template <class Mover>
__global__ void k_rank_gather(int n, int n_cells, const int2* link, const int2* cs, const int* head, const int* start,
                              Mover mv, unsigned* status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 c = cs[i];
    // in flight while the rank is found, and none behind a store (a load cannot pass one): 18.9 -> 14.8 us at
    // 515,018 particles, 182 -> 160 at 6,207,228
    const typename Mover::Item m = mv.load(i);
    const int dst = sorted_place(i, c, n_cells, n, link, head, start);
    if (dst < 0 || dst >= n) {
        atomicOr(status, EPP_STATUS_QUEUE);
        return;
    }
    mv.store(m, dst, c.x);
}

// Scatter in arrival order, for cells in no list: perm[start[c] + slot] = (id, source index).  A destination
// outside [0, n) can only come from a failed scan; it is reported, never written.
__device__ __forceinline__ void scatter_particle(int i, int n, int2 c, const int* start, int id, int2* perm, unsigned* status) {
    const int dst = start[c.x] + c.y;
    if (dst < 0 || dst >= n) atomicOr(status, EPP_STATUS_QUEUE);
    else perm[dst] = make_int2(id, i);
}

// Sorted position of perm's entry p, a particle of cell c: start + rank by id among its cell's entries,
// which lie side by side (independent loads, whatever order the particles came in).
__device__ __forceinline__ int sorted_place_perm(int p, int2 e, int c, int n, int n_cells, const int2* perm, const int* start) {
    if (c == n_cells) return p;
    const int s = start[c], en = min(start[c + 1], n);
    int rank = 0;
    for (int q = max(s, 0); q < en; ++q) rank += perm[q].x < e.x;
    return s + rank;
}

static __global__ void k_scatter(int n, const int2* cs, const int* start, const int* id, int2* perm, unsigned* status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) scatter_particle(i, n, cs[i], start, id[i], perm, status);
}

// The gather of a sort by slots: a thread per entry of perm.
template <class Mover>
__global__ void k_rank_gather_perm(int n, int n_cells, const int2* perm, const int2* cs, const int* start, Mover mv,
                                   unsigned* status) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int2 e = perm[p];
    if (e.y < 0 || e.y >= n) {
        atomicOr(status, EPP_STATUS_QUEUE);
        return;
    }
    const int c = cs[e.y].x;
    const typename Mover::Item m = mv.load(e.y);
    const int dst = sorted_place_perm(p, e, c, n, n_cells, perm, start);
    if (dst < 0 || dst >= n) {
        atomicOr(status, EPP_STATUS_QUEUE);
        return;
    }
    mv.store(m, dst, c);
}

// The occupied cells of a finished order, in no order of their own (family 1 taken up between searches;
// *n_occ is zero on entry).
static __global__ void k_list_occupied(int n_cells, const int* start, int* occ, int* n_occ) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const bool mine = c < n_cells && start[c + 1] > start[c];
    const unsigned all = __ballot_sync(0xffffffffu, mine);
    int base = 0;
    if (lane == 0 && all) base = atomicAdd(n_occ, __popc(all));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (mine) occ[base + __popc(all & ((1u << lane) - 1u))] = c;
}

// Mover of the per-call search: every state array follows the particle.
struct MoverAll {
    State a, b;
    struct Item {
        float4 xh, vm, dv, comp;
        float rho, drho, vol, p;
        int tagm, id;
    };
    __device__ __forceinline__ Item load(int src) const {
        return Item{a.xh[src],   a.vm[src],  a.dv[src], a.comp[src], a.rho[src],
                    a.drho[src], a.vol[src], a.p[src],  a.tagm[src], a.id[src]};
    }
    __device__ __forceinline__ void store(const Item& m, int dst, int c) const {
        b.xh[dst] = m.xh;
        b.vm[dst] = m.vm;
        b.dv[dst] = m.dv;
        b.comp[dst] = m.comp;
        b.rho[dst] = m.rho;
        b.drho[dst] = m.drho;
        b.vol[dst] = m.vol;
        b.p[dst] = m.p;
        b.tagm[dst] = m.tagm;
        b.id[dst] = m.id;
        b.cell[dst] = c;
    }
};

}  // namespace epp
