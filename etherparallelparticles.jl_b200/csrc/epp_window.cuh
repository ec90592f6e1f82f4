// epp_window.cuh -- the default search passes, over per-particle stencil-row windows: in 2D with the
// search action folded in (described here), in 3D lists and counts only (k_win_build3), and with eight
// lanes per particle for small systems (k_win_lanes).
//
// A particle's 3x3 cell stencil is three stencil rows (dy = -1, 0, +1); in each row its
// candidates are one contiguous cell-order range, cells cx-1 .. cx+1 (its "window", about 27
// particles at h = 1.5 dx).  The list search pass (k_build) tests, in lockstep, every candidate of
// the warp's union of stencils against every lane -- about 190 per particle; here each lane tests
// only its own window, 81 candidates.
//
// A warp takes 32 consecutive particles in cell order.  Those of one cell row (without a gap) form a
// part: the union of their windows in a stencil row is one contiguous range, from the first lane's
// window to the last lane's.  The warp stages the three ranges of each part in shared memory, packed one after the other
// -- position and h, the list entry (index and tag) in the unused z lane, and the search action's
// neighbour record -- and every lane reads its own windows from there.  The staging area holds both
// parts of a warp that crosses a cell-row end; what does not fit (a free surface, whose warps span
// many cells over a dense row) is split into passes over fewer lanes, and lanes whose own windows do
// not fit (dense neighbourhoods, h of 2.5 dx and more) all read theirs from global memory at once: 2D
// search at h = 3 dx, 132,518 particles, 195 us, where a pass for each such lane took 2990.  The lane
// builds one acceptance word per stencil row with the reference's IEEE criterion and the active-pair
// matrix, then walks the set bits of the three words in list order, in one loop: it appends the
// neighbour to its list (the lists the momentum, filter and extrapolation passes read; same layout
// and order as k_build's: stencil rows, then cell order, then id order inside a cell) and adds the
// search action's term -- the continuity rate -- from the staged record, so no separate continuity
// pass walks the neighbours again.
//
// What bounds it: instruction issue at large sizes (bulk warps -- one h, one tag, fluid -- take a
// specialised test and walk), and at middle sizes the slowest warp, hence one pass for all parts and
// no dependent global reads in it.
#pragma once
#include "epp_tile.cuh"

namespace epp {

// A bound b on dr2 for the integer test bits(dr2) + accept_bias(b) < 0 <=> dr2 <= b: non-negative
// floats order like their bit patterns.  A NaN bound accepts nothing.
__device__ __forceinline__ int accept_bias(float b) { return b >= 0.0f ? -__float_as_int(b) - 1 : 0; }

struct RowWin {
    int lo, hi;   // candidate range [lo, hi) in cell order
};

// Linear cell row of stencil row r of the cell row rid = y + n1 z, or -1 outside the grid.  2D: r =
// 0, 1, 2 for dy = -1, 0, +1 (z is the instance of a batch, never crossed); 3D: r = 3 (dz + 1) + dy + 1.
template <int D>
__device__ __forceinline__ int stencil_row(const PairArgs& A, int rid, int y, int z, int r) {
    const int yy = y + (D == 3 ? r % 3 : r) - 1, dz = D == 3 ? r / 3 - 1 : 0;
    if (yy < 0 || yy >= A.dom.n[1]) return -1;
    if (D == 3 && (z + dz < 0 || z + dz >= A.dom.n[2])) return -1;
    return rid + yy - y + (D == 3 ? A.dom.n[1] * dz : 0);
}

// Candidates of cells xa .. xb (clamped to the grid) of linear cell row `row` (-1: none).  A range beyond
// either end of the row is empty where the row ends: the ranges of a part's lanes stay in order.
__device__ __forceinline__ RowWin row_range(const PairArgs& A, int row, int xa, int xb) {
    RowWin w{0, 0};
    if (row < 0) return w;
    const int n0 = A.dom.n[0];
    xa = max(xa, 0);
    xb = min(xb, n0 - 1);
    const int l = max(A.start[row * n0 + xa], 0);
    const int h = min(A.start[row * n0 + xb + 1], A.n_max);
    w.lo = l;
    w.hi = max(h, l);
    return w;
}

// What a search pass starts from, read at once rather than after the alive count (i may lie beyond it).
struct WinSelf {
    float4 x;
    int n_alive, tag, cell;
};
__device__ __forceinline__ WinSelf win_self(const PairArgs& A, int i) {
    const int k = min(i, A.n_max - 1);
    return WinSelf{A.s.xh[k], min(A.start[A.dom.n_cells], A.n_max), tag_of(A.s.tagm[k]), A.s.cell[k]};
}

// A warp of more parts than this (spray: few particles to a cell) reads its windows from memory, all lanes
// at once, in place of staging part after part.  Search, us, of particles at random places with the
// rule at 5, 7, 10 and without it: 3D, 0.3 to a cell, 1,505,378 particles 280 / 293 / 364 / 494,
// 209,361 54 / 57 / 71 / 93; 1 to a cell 70 / 70 / 72 / 74; 2D, 1 to a cell, 106,854 particles 20.5 / 18.5
// / 18.5 / 18.5.
constexpr int kPartsMax = 7;

constexpr int kStage2 = 240;   // staged candidates per warp: 7 blocks of 128 threads still fit an SM

template <class Act>
struct Stage2 {
    float4 x[kStage2];                 // (x, y, list entry as bits, h)
    typename Act::Nb nb[kStage2];
};

// Acceptance bits of a lane's window of `len` <= 32 candidates from slot `off`: bit k set when
// candidate k passes the criterion by the reference's IEEE arithmetic.  `one`: every candidate has the
// lane's h (or the default criterion), so one exact bound serves (bias nO); otherwise those of another
// h take its bound, the bias of the last one kept in (ho, no): cells hold their fluid before their
// walls, so along a row h alternates between the lane's own and one other.
__device__ __forceinline__ unsigned window_bits(const float4* sx, int off, int len, float4 xi, bool one, int nO, float& ho,
                                                int& no) {
    // (dx, dy) and (dx^2, dy^2) on the packed f32x2 pipe (each half rounds like __fsub_rn /
    // __fmul_rn), the sum scalar
    const f32x2 XY = f2_pack(xi.x, xi.y);
    unsigned word = 0u;
    if (one) {
#pragma unroll 4
        for (int k = len - 1; k >= 0; --k) {
            const f32x2 d = f2_sub(XY, *reinterpret_cast<const f32x2*>(&sx[off + k]));
            float dx2, dy2;
            f2_unpack(f2_mul(d, d), dx2, dy2);
            word = (word << 1) | ((unsigned)(__float_as_int(__fadd_rn(dx2, dy2)) + nO) >> 31);
        }
        return word;
    }
#pragma unroll 4
    for (int k = len - 1; k >= 0; --k) {
        const float hj = sx[off + k].w;
        const f32x2 d = f2_sub(XY, *reinterpret_cast<const f32x2*>(&sx[off + k]));
        float dx2, dy2;
        f2_unpack(f2_mul(d, d), dx2, dy2);
        if (hj != xi.w && hj != ho) {
            ho = hj;
            no = accept_bias(pair_r2(xi.w, ho));
        }
        word = (word << 1) | ((unsigned)(__float_as_int(__fadd_rn(dx2, dy2)) + (hj == xi.w ? nO : no)) >> 31);
    }
    return word;
}

// What the general per-lane search hands back to the search pass.
struct WinOut {
    int cnt;
    float sx, sy;
};

// Candidates [lo, hi) of one window straight from global memory, 32 at a time: the acceptance bits of
// a word first, its loads in flight together, then one walk over the set bits.  (Candidate by candidate,
// each accepted one evaluated where it was met, a warp ran the term once for nearly every candidate.)
// own: the bound against candidates of the lane's h, or of the default criterion.
template <int D, class Act>
__device__ __forceinline__ void window_from_memory(const PairArgs& A, const Act& act, const typename Act::Self& me,
                                                   const TargetConst& tc, ListWriter<D>& L, int lo, int hi, int i, int ti,
                                                   float4 xi, unsigned amask, float own, OtherBound& other, WinOut& o) {
    const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
#pragma unroll 1
    for (int k0 = lo; k0 < hi; k0 += 32) {
        const int len = min(hi - k0, 32);
        unsigned word = 0u;
#pragma unroll 4
        for (int k = len - 1; k >= 0; --k) {
            const float4 xj = A.s.xh[k0 + k];
            word = (word << 1) | (geometry<D>(xi, xj).dr2 <= other.of(xi.w, xj.w, own, dflt) ? 1u : 0u);
        }
        const int self = i - k0;   // not its own neighbour
        if (self >= 0 && self < 32) word &= ~(1u << self);
        while (word) {
            const int j = k0 + __ffs(word) - 1;
            word &= word - 1u;
            const int tj = tag_of(A.s.tagm[j]);
            if (!(__funnelshift_rc(amask, 0u, (unsigned)(tj - 1)) & 1u)) continue;   // the active-pair matrix
            L.put(o.cnt++, list_entry(j, tj));
            if (Act::NC != 0) {
                const float4 xj = A.s.xh[j];
                const float4 t = act.term(me, act.fetch(j, ti, tj), ti, tj, xj, geometry<D>(xi, xj), tc);
                o.sx = __fadd_rn(o.sx, t.x);
                o.sy = __fadd_rn(o.sy, t.y);
            }
        }
    }
}

// The per-lane search in its general form, from global memory: dense neighbourhoods only (a window
// beyond 64 candidates, or windows beyond the staging area).  Inlined: as an out-of-line call it cost
// the kernel registers (the values live across the call) and 13% of its time.
template <int D, class Act>
__device__ __forceinline__ WinOut win_lane_general(const PairArgs& A, const TileMask& M, const Act& act,
                                                const RowWin (&win)[D == 3 ? 9 : 3], int i, int ti, float4 xi, unsigned amask) {
    const TargetConst tc = target_const<D>(xi.w);
    const typename Act::Self me = act.self(i);
    ListWriter<D> L = list_writer<D>(M, i);
    WinOut o{0, 0.0f, 0.0f};
    OtherBound other{xi.w, 0.0f};
#pragma unroll 1
    for (int r = 0; r < (D == 3 ? 9 : 3); ++r) {
        int lo = 0, hi = 0;
#pragma unroll
        for (int q = 0; q < (D == 3 ? 9 : 3); ++q)
            if (q == r) lo = win[q].lo, hi = win[q].hi;
        window_from_memory<D>(A, act, me, tc, L, lo, hi, i, ti, xi, amask, A.crit == EPP_CRITERION_DEFAULT ? A.dom.gap_square : tc.h2sq,
                              other, o);
    }
    L.flush(o.cnt);
    return o;
}

// The 2D search pass: neighbour lists and nCount, and the search action of `Act` over the accepted
// neighbours in list order (CPCont: continuity + density preview; CPCount: the count only).  A
// particle with more neighbours than a list keeps has only those stored (the pair passes read its
// stencil); its search action still covers all of them.
template <class Act>
__global__ void __launch_bounds__(128, 7) k_win_build(const __grid_constant__ PairArgs A, const __grid_constant__ TileMask M,
                                                   const __grid_constant__ Act act, unsigned long long* pairs) {
    extern __shared__ __align__(16) unsigned char win_smem[];   // a staging area per warp
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    Stage2<Act>& S = reinterpret_cast<Stage2<Act>*>(win_smem)[threadIdx.x >> 5];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int w0 = i - lane;
    const WinSelf me0 = win_self(A, i);
    const int n_alive = me0.n_alive;
    int cnt = 0;
    if (w0 < n_alive) {   // warp-uniform
        const bool on = i < n_alive;
        const int c = __shfl_sync(FULL, me0.cell, min(lane, n_alive - 1 - w0));
        EPP_CHECK(!__any_sync(FULL, c < 0 || c >= A.dom.n_cells), 34, c);
        const int rid = A.dom.by[0].div(max(c, 0)), cx = c - rid * A.dom.n[0];
        const int z = A.dom.by[1].div(rid), y = rid - z * A.dom.n[1];
        const float4 xi = on ? me0.x : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        const int ti = on ? me0.tag : 0;
        const bool valid = on && ti >= 1 && ti <= A.n_tags;
        const unsigned amask = valid ? A.adj[ti - 1] : 0u;   // bits of valid tags only
        const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
        RowWin win[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) win[r] = row_range(A, stencil_row<2>(A, rid, y, z, r), cx - 1, cx + 1);
        // a part ends at the end of a cell row and where the next lane's windows do not meet this one's:
        // what lies between (the floor under a gap of the fluid) is nobody's candidate
        const int rid_p = __shfl_up_sync(FULL, rid, 1), cx_p = __shfl_up_sync(FULL, cx, 1);
        const unsigned starts = __ballot_sync(FULL, lane == 0 || rid != rid_p || cx - cx_p > 3);
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const int l0 = win[0].hi - win[0].lo, l1 = win[1].hi - win[1].lo, l2 = win[2].hi - win[2].lo;
        const int longest = max(l0, max(l1, l2));
        // dense neighbourhoods and spray go straight to memory, all of the warp's at once
        const bool direct = longest > 64 || l0 + l1 + l2 > kStage2 || __popc(starts) > kPartsMax;
        unsigned pending = __ballot_sync(FULL, on && !direct);
        while (pending) {   // warp-uniform: a pass over as many parts as the staging area holds
            const int head = __ffs(pending) - 1;
            const float hw = __shfl_sync(FULL, xi.w, head);   // the pass is plain when every candidate has
            const int tw = __shfl_sync(FULL, ti, head);       // the first lane's h and tag
            bool same_t = true, other = false;
            float hb = hw;   // an h other than hw that this lane staged
            int used = 0, off[3] = {0, 0, 0};
            unsigned taken = 0u;
            __syncwarp();
            while (pending) {
                const int lead = __ffs(pending) - 1;
                const unsigned after = starts & ~((2u << lead) - 1u);   // part starts behind the lead
                int last = min(after ? __ffs(after) - 2 : 31, 31 - __clz(pending));
                int lo[3], len[3], total;
                for (;;) {
                    total = 0;
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        lo[r] = __shfl_sync(FULL, win[r].lo, lead);
                        len[r] = max(__shfl_sync(FULL, win[r].hi, last) - lo[r], 0);
                        total += len[r];
                    }
                    if (total <= kStage2 - used || used > 0 || last == lead) break;
                    last = lead + (last - lead) / 2;
                }
                if (total > kStage2 - used) break;   // next pass (the first part of a pass fits)
                for (int k = lane; k < total; k += 32) {
                    const int j = k < len[0] ? lo[0] + k : k < len[0] + len[1] ? lo[1] + (k - len[0]) : lo[2] + (k - len[0] - len[1]);
                    const float4 xj = A.s.xh[j];
                    const int tj = tag_of(A.s.tagm[j]);
                    const bool bad = tj < 1 || tj > A.n_tags;   // never a neighbour: fails every test (its own lane reports it)
                    S.x[used + k] = make_float4(bad ? __int_as_float(0x7fffffff) : xj.x, xj.y,
                                                __int_as_float(list_entry(j, bad ? 1 : tj)), xj.w);
                    if (Act::NC != 0) S.nb[used + k] = act.fetch(j, 0, tj);
                    if (xj.w != hw) other = true, hb = xj.w;
                    same_t = same_t && tj == tw;
                }
                const unsigned part = ((2u << last) - 1u) & ~((1u << lead) - 1u) & pending;
                if ((part >> lane) & 1u) {
                    off[0] = used + win[0].lo - lo[0];
                    off[1] = used + len[0] + win[1].lo - lo[1];
                    off[2] = used + len[0] + len[1] + win[2].lo - lo[2];
                }
                used += total;
                taken |= part;
                pending &= ~part;
            }
            const unsigned others = __ballot_sync(FULL, other);
            const float h2 = __shfl_sync(FULL, hb, others ? __ffs(others) - 1 : 0);   // another h of the pass, if any
            same_t = __all_sync(FULL, same_t);
            __syncwarp();
            if (!(((taken >> lane) & 1u) && valid)) continue;
            // cells of four particle rows or columns (where the lattice and the cells drift apart) make
            // windows of up to 40: the lanes of the pass then take each row in two words, one after the other
            const bool two = __any_sync(__activemask(), longest > 32);
            const TargetConst tc = target_const<2>(xi.w);
            if (same_t && !((amask >> (tw - 1)) & 1u)) continue;   // nothing the lane may see: walls among walls
            const bool one = dflt || !others;
            const int nO = accept_bias(dflt ? A.dom.gap_square : tc.h2sq);
            // kernel constants and bound with the pass's other h (walls against fluid), so that the walk
            // selects instead of dividing per pair (182 -> 174 us for 64 dam breaks of 1,217,760 particles,
            // step 34.6 -> 33.6 at 22,279); a third h is computed where it is met
            TargetConst to = tc;
            int no = nO;
            if (others) {
                to.h = xi.w == hw ? h2 : hw;
                to.hinv = invharmonic_exact(tc.h, to.h);
                to.kdw = wc2_kdw<2>(to.hinv);
                no = accept_bias(pair_r2(xi.w, to.h));
            }
            float ho = to.h;
            typename Act::Self me = act.self(i);
            ListWriter<2> L = list_writer<2>(M, i);
            const f32x2 XI = f2_pack(xi.x, xi.y);
            bool bulk = false;   // the bulk of the fluid: fluid candidates of the lane's h around a fluid lane
            if constexpr (Act::FAST) bulk = same_t && one && !dflt && tw == act.P.fluid && ti == tw;
            for (int q = 0; q < (two ? 6 : 1); ++q) {
                unsigned a, b = 0u, c2 = 0u;
                int o0 = off[0], o1 = off[1], o2 = off[2];
                if (!two) {
                    // the three words first, then one walk over all of them, so a warp iterates as often as
                    // its busiest lane's neighbour count (not the sum over rows of each row's busiest lane)
                    a = window_bits(S.x, o0, l0, xi, one, nO, ho, no);
                    b = window_bits(S.x, o1, l1, xi, one, nO, ho, no);
                    c2 = window_bits(S.x, o2, l2, xi, one, nO, ho, no);
                    b &= ~(1u << (i - win[1].lo));   // not its own neighbour
                    if (!b) b = c2, o1 = o2, c2 = 0u;   // empty rows last: one word is current, the next follows
                    if (!a) a = b, o0 = o1, b = c2, o1 = o2, c2 = 0u;
                } else {
                    const int r = q >> 1, k0 = (q & 1) * 32;
                    o0 = (r == 0 ? off[0] : r == 1 ? off[1] : off[2]) + k0;
                    a = window_bits(S.x, o0, min((r == 0 ? l0 : r == 1 ? l1 : l2) - k0, 32), xi, one, nO, ho, no);
                    const int self = i - win[1].lo - k0;
                    if (r == 1 && self >= 0 && self < 32) a &= ~(1u << self);
                }
                if (bulk) {
                    if constexpr (Act::FAST) {
                        const f32x2 VI = f2_pack(me.v.x, me.v.y);
                        while (a) {
                            const int slot = o0 + __ffs(a) - 1;
                            a &= a - 1u;
                            if (!a) a = b, o0 = o1, b = c2, o1 = o2, c2 = 0u;
                            const float4 xs = S.x[slot];
                            L.put(cnt++, __float_as_int(xs.z));
                            sum.x = __fadd_rn(sum.x, act.fluid_term(XI, VI, xs, S.nb[slot].v, tc));
                        }
                    }
                } else {
                    while (a) {   // append and run the search action, in list order
                        const int slot = o0 + __ffs(a) - 1;
                        a &= a - 1u;
                        if (!a) a = b, o0 = o1, b = c2, o1 = o2, c2 = 0u;
                        const float4 xs = S.x[slot];
                        const int e = __float_as_int(xs.z);
                        if (!((amask >> (entry_tag(e) - 1)) & 1u)) continue;   // the active-pair matrix
                        L.put(cnt++, e);
                        if (Act::NC != 0) {
                            const int tj = entry_tag(e);
                            const float4 xj = make_float4(xs.x, xs.y, 0.0f, xs.w);
                            TargetConst tq = tc;
                            if (xs.w == to.h) tq.h = to.h, tq.hinv = to.hinv, tq.kdw = to.kdw;
                            const float4 t = act.term(me, S.nb[slot], ti, tj, xj, geometry<2>(xi, xj), tq);
                            sum.x = __fadd_rn(sum.x, t.x);
                            sum.y = __fadd_rn(sum.y, t.y);
                        }
                    }
                }
            }
            L.flush(cnt);
        }
        if (direct && valid) {
            const WinOut o = win_lane_general<2, Act>(A, M, act, win, i, ti, xi, amask);
            cnt = o.cnt;
            sum.x = o.sx;
            sum.y = o.sy;
        }
        if (on) {
            if (!valid) {
                act.end_idle(i, ti);
                atomicOr(A.status, EPP_STATUS_BAD_TAG);
            } else {
                act.end(i, ti, sum, cnt);
            }
        }
    }
    count_pairs(pairs, cnt);
}

// The 3D search pass: neighbour lists and nCount.  Windows as in 2D, nine stencil rows of about 53
// candidates at h = 1.3 dx, one plane (three rows) staged at a time; a particle's 480 candidates are
// tested by its own lane.  It replaces a lockstep search of the warp's whole union of stencils (about
// 700 candidates, 32 at a time, with a divergent append after each chunk): 574 -> 356 us at 955,668
// particles, 182 -> 84 at 165,888.  Issue-bound (80% of the slots, 22.7 of 32 lanes at
// work: the walk over a word's bits is as long as the busiest lane's), which is why a word whose
// candidates have one tag computes its entries and checks the list's capacity once.  Warps near walls stage two h's and take the two bounds by a select.
// When one particle's plane is longer than the staging area (dense neighbourhoods) the stencil goes by
// rows, or by cells, and a cell beyond it is read from global memory by all its lanes at once: 926 us
// at h = 2.5 dx and 165,888 particles, where a pass for each lane with a long row took 12800.
// One warp per cell, its lanes on the candidates
// and ballots in place of the walk, measured 528 us: two POPC per target and chunk, no fewer
// instructions.
// Staged candidates per warp: both parts of a warp that crosses a cell-row end (about 360; with room for
// 320 only, such warps searched a plane in two passes and were the pass's tail: 121 us at 165,888
// particles); 7 blocks of 128 threads fit an SM.
constexpr int kStage3 = 432;

struct Stage3 {
    float4 x[kStage3];          // (x, y, z, h)
    unsigned char t[kStage3];   // tag
};

// Acceptance bits of `len` <= 32 staged candidates from slot `off`, candidate 0 in the top bit; see
// window_bits.  HS = 1: one exact bound (its bias nA) for all; 2: candidates of h == hA take nA, the
// others, all of one other h, nB (fluid and walls); 3: any h, nO for the lane's own, the bias of the
// last other one kept in (ho, no).
template <int HS>
__device__ __forceinline__ unsigned window_bits3(const float4* sx, int off, int len, float4 xi, int nA, float hA, int nB,
                                                 int nO, float& ho, int& no) {
    const f32x2 XY = f2_pack(xi.x, xi.y);
    unsigned word = 0u;
#pragma unroll 4
    for (int k = 0; k < len; ++k) {
        const float4 c = sx[off + k];
        const f32x2 d = f2_sub(XY, f2_pack(c.x, c.y));
        float ex, ey;
        f2_unpack(f2_mul(d, d), ex, ey);
        const float dz = __fsub_rn(xi.z, c.z);
        const float dr2 = __fadd_rn(__fadd_rn(ex, ey), __fmul_rn(dz, dz));
        int n = nA;
        if (HS == 2) n = c.w == hA ? nA : nB;
        if (HS == 3) {
            if (c.w != ho) {
                ho = c.w;
                no = ho == xi.w ? nO : accept_bias(pair_r2(xi.w, ho));
            }
            n = no;
        }
        word = __funnelshift_l((unsigned)(__float_as_int(dr2) + n), word, 1);
    }
    return len < 32 ? word << (32 - len) : word;
}

__global__ void __launch_bounds__(128, 7) k_win_build3(const __grid_constant__ PairArgs A, const __grid_constant__ TileMask M,
                                                       int* ncount, unsigned long long* pairs) {
    extern __shared__ __align__(16) unsigned char win_smem[];   // a staging area per warp
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    Stage3& S = reinterpret_cast<Stage3*>(win_smem)[threadIdx.x >> 5];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int w0 = i - lane;
    const WinSelf me0 = win_self(A, i);
    const int n_alive = me0.n_alive;
    int cnt = 0;
    if (w0 < n_alive) {   // warp-uniform
        const bool on = i < n_alive;
        const int c = __shfl_sync(FULL, me0.cell, min(lane, n_alive - 1 - w0));
        EPP_CHECK(!__any_sync(FULL, c < 0 || c >= A.dom.n_cells), 36, c);
        const int rid = A.dom.by[0].div(max(c, 0)), cx = c - rid * A.dom.n[0];
        const int z = A.dom.by[1].div(rid), y = rid - z * A.dom.n[1];
        const float4 xi = on ? me0.x : make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        const int ti = on ? me0.tag : 0;
        const bool valid = on && ti >= 1 && ti <= A.n_tags;
        const unsigned amask = valid ? A.adj[ti - 1] : 0u;   // bits of valid tags only
        const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
        const float own = dflt ? A.dom.gap_square : target_const<3>(xi.w).h2sq;
        ListWriter<3> L = list_writer<3>(M, min(i, n_alive - 1));
        // parts as in the 2D pass: they end with a cell row and at a gap of it
        const int rid_p = __shfl_up_sync(FULL, rid, 1), cx_p = __shfl_up_sync(FULL, cx, 1);
        const unsigned starts = __ballot_sync(FULL, lane == 0 || rid != rid_p || cx - cx_p > 3);
        const unsigned alive = __ballot_sync(FULL, on);
        // u counts cells of the stencil; a step takes a plane of them, a row or, in dense neighbourhoods, one
        // (spray: a row, its low bits)
        constexpr int SPRAY = 16 + 3;
        int step = __popc(starts) > kPartsMax ? SPRAY : 9;
        for (int u = 0; u < 27; u += step & 15) {   // warp-uniform
            RowWin win[3];
            int mine = 0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int x = step == 1 ? cx - 1 + u % 3 : cx - 1;
                win[q] = q == 0 || step == 9 ? row_range(A, stencil_row<3>(A, rid, y, z, u / 3 + q), x, step == 1 ? x : cx + 1) : RowWin{0, 0};
                mine += win[q].hi - win[q].lo;
            }
            if (step == 9 && __any_sync(FULL, mine > kStage3)) {   // from here on one row at a time
                step = 3;
                win[1] = win[2] = RowWin{0, 0};
                mine = win[0].hi - win[0].lo;
            }
            if (step == 3 && __any_sync(FULL, mine > kStage3)) {   // or one cell
                step = 1;
                win[0] = row_range(A, stencil_row<3>(A, rid, y, z, u / 3), cx - 1, cx - 1);
                mine = win[0].hi - win[0].lo;
            }
            const bool direct = mine > kStage3 || step == SPRAY;   // from memory, all such lanes at once
            if (direct && valid) {
                OtherBound other{xi.w, 0.0f};
                WinOut o{cnt, 0.0f, 0.0f};
                window_from_memory<3>(A, CPCount<3>{ncount}, CPCount<3>::Self{}, TargetConst{}, L, win[0].lo, win[0].hi, i, ti, xi,
                                      amask, own, other, o);
                cnt = o.cnt;
            }
            unsigned pending = alive & ~__ballot_sync(FULL, direct);
            while (pending) {   // warp-uniform: a pass over as many parts as the staging area holds
                const int head = __ffs(pending) - 1;
                const float hw = __shfl_sync(FULL, xi.w, head);
                const int tw = __shfl_sync(FULL, ti, head);
                bool same_t = true;
                bool other = false, two_h = true;   // an h other than hw was staged by this lane; one such h only
                float hb = hw;
                int used = 0, off[3] = {0, 0, 0};
                unsigned taken = 0u;
                __syncwarp();
                while (pending) {
                    const int lead = __ffs(pending) - 1;
                    const unsigned after = starts & ~((2u << lead) - 1u);   // part starts behind the lead
                    int last = min(after ? __ffs(after) - 2 : 31, 31 - __clz(pending));
                    int lo[3], len[3], total;
                    for (;;) {
                        total = 0;
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            lo[q] = __shfl_sync(FULL, win[q].lo, lead);
                            len[q] = max(__shfl_sync(FULL, win[q].hi, last) - lo[q], 0);
                            total += len[q];
                        }
                        if (total <= kStage3 - used || used > 0 || last == lead) break;
                        last = lead + (last - lead) / 2;
                    }
                    if (total > kStage3 - used) break;   // next pass (the first part of a pass fits)
#pragma unroll 4   // their loads in flight together (2% at 955,668 particles, 4% at 165,888; the 2D pass lost 3%)
                    for (int k = lane; k < total; k += 32) {
                        const int j = k < len[0] ? lo[0] + k
                                                 : k < len[0] + len[1] ? lo[1] + (k - len[0]) : lo[2] + (k - len[0] - len[1]);
                        float4 xj = A.s.xh[j];
                        const int tj = tag_of(A.s.tagm[j]);
                        const bool bad = tj < 1 || tj > A.n_tags;   // never a neighbour: fails every test
                        if (bad) xj.x = __int_as_float(0x7fffffff);
                        S.x[used + k] = xj;
                        S.t[used + k] = (unsigned char)(bad ? 1 : tj);
                        if (xj.w != hw) {
                            two_h = two_h && (!other || hb == xj.w);
                            other = true;
                            hb = xj.w;
                        }
                        same_t = same_t && tj == tw;
                    }
                    const unsigned part = ((2u << last) - 1u) & ~((1u << lead) - 1u) & pending;
                    if ((part >> lane) & 1u) {
                        off[0] = used + win[0].lo - lo[0];
                        off[1] = used + len[0] + win[1].lo - lo[1];
                        off[2] = used + len[0] + len[1] + win[2].lo - lo[2];
                    }
                    used += total;
                    taken |= part;
                    pending &= ~part;
                }
                const unsigned others = __ballot_sync(FULL, other);
                const float h2 = __shfl_sync(FULL, hb, others ? __ffs(others) - 1 : 0);   // the other h, if any
                two_h = __all_sync(FULL, two_h && (!other || hb == h2));
                same_t = __all_sync(FULL, same_t);
                __syncwarp();
                if (!(((taken >> lane) & 1u) && valid)) continue;
                if (same_t && !((amask >> (tw - 1)) & 1u)) continue;   // walls among walls
                // exact bounds of this lane against hw and the other h, as window_bits3 takes them
                const int hs = dflt || !others ? 1 : two_h ? 2 : 3;   // warp-uniform
                const int nO = accept_bias(own);
                const int nA = dflt || xi.w == hw ? nO : accept_bias(pair_r2(xi.w, hw));
                const int nB = hs == 1 || xi.w == h2 ? nO : accept_bias(pair_r2(xi.w, h2));
                float ho = xi.w;
                int no = nO;
#pragma unroll 1
                for (int q = 0; q < (step == 9 ? 3 : 1); ++q) {
                    const int lo = q == 0 ? win[0].lo : q == 1 ? win[1].lo : win[2].lo;
                    const int n = (q == 0 ? win[0].hi : q == 1 ? win[1].hi : win[2].hi) - lo;
                    const int o = q == 0 ? off[0] : q == 1 ? off[1] : off[2];
                    const int self = u / 3 + q == 4 ? i - lo : -1;   // not its own neighbour
                    for (int k0 = 0; k0 < n; k0 += 32) {
                        const int len = min(n - k0, 32);
                        unsigned word = hs == 1   ? window_bits3<1>(S.x, o + k0, len, xi, nA, hw, nB, nO, ho, no)
                                        : hs == 2 ? window_bits3<2>(S.x, o + k0, len, xi, nA, hw, nB, nO, ho, no)
                                                  : window_bits3<3>(S.x, o + k0, len, xi, nA, hw, nB, nO, ho, no);
                        if ((self >> 5) == (k0 >> 5)) word &= ~(0x80000000u >> (self & 31));
                        if (same_t && cnt >= ListConf<3>::LCAP) {   // no list to keep
                            cnt += __popc(word);
                            continue;
                        }
                        if (same_t && cnt + 32 <= ListConf<3>::LCAP) {   // entries from their index, room for all
                            const int e0 = list_entry(lo + k0, tw);
                            while (word) {
                                const int b = __clz(word);
                                word ^= 0x80000000u >> b;
                                L.put_room(cnt++, e0 + b);
                            }
                            continue;
                        }
                        while (word) {
                            const int b = __clz(word);
                            word ^= 0x80000000u >> b;
                            const int tj = S.t[o + k0 + b];
                            if ((amask >> (tj - 1)) & 1u) L.put(cnt++, list_entry(lo + k0 + b, tj));   // the active-pair matrix
                        }
                    }
                }
            }
        }
        L.flush(cnt);
        if (on) ncount[i] = cnt;
        if (on && !valid) atomicOr(A.status, EPP_STATUS_BAD_TAG);
    }
    count_pairs(pairs, cnt);
}

// The same pass for small systems: L lanes per particle, candidates straight from global memory, so a
// particle's walk is L times shorter.  Lane g tests candidates g, g + L, ... of each window (four loads
// in flight); a ballot of the group gives each accepted one its place in the list, kept in shared
// memory; then lane g writes entries g, g + L, ... out and evaluates the action's terms for them, and
// the first lane adds the terms in list order: lists, counts and sums have the bits of k_win_build.  With
// more neighbours than a list keeps, a search without terms is done (the first ones are stored: 3D, h =
// 2.5 dx, 20,340 particles, 157 us against 588 with a second search), one with terms goes through the
// general per-lane search.  It issues four times k_win_build's instructions per particle (383 against
// 93) but a fifth of them one after the other: 12 us against 25 at 1,418 particles, 22 each at 22,279;
// 3D 52 against 88 at 33,123.
template <int D, class Act, int L>
__global__ void __launch_bounds__(128) k_win_lanes(const __grid_constant__ PairArgs A, const __grid_constant__ TileMask M,
                                                   const __grid_constant__ Act act, unsigned long long* pairs) {
    constexpr int P = 128 / L, CAP = ListConf<D>::LCAP, NR = D == 3 ? 9 : 3;
    __shared__ int s_e[P][CAP + 1];                           // accepted entries (odd rows: no bank conflicts)
    __shared__ float s_t[Act::NC != 0 ? P : 1][CAP + 1];      // their terms
    const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / L);
    const WinSelf me0 = win_self(A, i);
    const int g = threadIdx.x % L, p = threadIdx.x / L;
    const int first = (int)(threadIdx.x & 31u & ~(unsigned)(L - 1));
    const unsigned group = ((1u << L) - 1u) << first;
    int cnt = 0;
    if (i < me0.n_alive) {
        const float4 xi = me0.x;
        const int ti = me0.tag, c = me0.cell;
        if (ti < 1 || ti > A.n_tags) {
            if (g == 0) {
                act.end_idle(i, ti);
                atomicOr(A.status, EPP_STATUS_BAD_TAG);
            }
        } else {
            EPP_CHECK(c >= 0 && c < A.dom.n_cells, 35, c);
            const int rid = A.dom.by[0].div(c), cx = c - rid * A.dom.n[0];
            const int z = A.dom.by[1].div(rid), y = rid - z * A.dom.n[1];
            RowWin win[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) win[r] = row_range(A, stencil_row<D>(A, rid, y, z, r), cx - 1, cx + 1);
            const unsigned amask = A.adj[ti - 1];   // bits of valid tags only
            const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
            const TargetConst tc = target_const<D>(xi.w);
            const float r2own = dflt ? A.dom.gap_square : tc.h2sq;
            const f32x2 XI = f2_pack(xi.x, xi.y);
            float ho = xi.w, ro = r2own;   // the bound of the last h_j seen
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                for (int j0 = win[r].lo; j0 < win[r].hi; j0 += 4 * L) {
                    float4 xj[4];
                    int tm[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int j = j0 + q * L + g;
                        xj[q] = make_float4(0.0f, 0.0f, 0.0f, xi.w);
                        tm[q] = 0;
                        if (j < win[r].hi && j != i) {
                            xj[q] = A.s.xh[j];
                            tm[q] = tag_of(A.s.tagm[j]);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (j0 + q * L >= win[r].hi) break;   // uniform in the group
                        // the reference's IEEE criterion and the active-pair matrix (tag 0: none)
                        float ex, ey;
                        const f32x2 d = f2_sub(XI, f2_pack(xj[q].x, xj[q].y));
                        f2_unpack(f2_mul(d, d), ex, ey);
                        float dr2 = __fadd_rn(ex, ey);
                        if (D == 3) {
                            const float dz = __fsub_rn(xi.z, xj[q].z);
                            dr2 = __fadd_rn(dr2, __fmul_rn(dz, dz));
                        }
                        if (xj[q].w != ho) {
                            ho = xj[q].w;
                            ro = dflt || ho == xi.w ? r2own : pair_r2(xi.w, ho);
                        }
                        const bool ok = dr2 <= ro && (__funnelshift_rc(amask, 0u, (unsigned)(tm[q] - 1)) & 1u);
                        const unsigned hits = (__ballot_sync(group, ok) >> first) & ((1u << L) - 1u);
                        const int at = cnt + __popc(hits & ((1u << g) - 1u));
                        if (ok && at < CAP) s_e[p][at] = list_entry(j0 + q * L + g, tm[q]);
                        cnt += __popc(hits);
                    }
                }
            }
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (Act::NC != 0 && cnt > CAP) {
                if (g == 0) {
                    const WinOut o = win_lane_general<D, Act>(A, M, act, win, i, ti, xi, amask);
                    sum.x = o.sx;
                    sum.y = o.sy;
                }
            } else {
                __syncwarp(group);
                const typename Act::Self me = act.self(i);
#pragma unroll 2
                for (int k = g; k < min(cnt, CAP); k += L) {
                    const int e = s_e[p][k], j = entry_index(e), tj = entry_tag(e);
                    if (D == 3) M.list[(size_t)i * CAP + k] = e;
                    else M.list[(size_t)k * M.cap + i] = e;
                    if constexpr (Act::NC != 0) {
                        const float4 xj = A.s.xh[j];
                        const typename Act::Nb nb = act.fetch(j, ti, tj);
                        s_t[p][k] = act.term(me, nb, ti, tj, xj, geometry<D>(xi, xj), tc).x;
                    }
                }
                if constexpr (Act::NC != 0) {
                    __syncwarp(group);
                    if (g == 0) {
#pragma unroll 4
                        for (int k = 0; k < cnt; ++k) sum.x = __fadd_rn(sum.x, s_t[p][k]);
                    }
                }
            }
            if (g == 0) act.end(i, ti, sum, cnt);
        }
    }
    count_pairs(pairs, g == 0 ? cnt : 0);
}

}  // namespace epp
