// epp_tile.cuh -- neighbour lists: the pair passes over them (k_list), and the 2D lockstep search of
// EPP_TUNING_LISTS that builds them (k_build; the default searches are in epp_window.cuh).
//
// k_list (continuity, momentum, filter, extrapolation, the count actions) walks each particle's list
// with one or four lanes a particle, so every lane runs its own neighbours without waiting for the
// others' candidates; a particle with more neighbours than a list keeps takes its stencil instead.
//
// k_build takes 32 consecutive particles in cell order a warp.  When their cells lie in one cell row (x
// from xa to xb at fixed y) the union of their stencils is, for each of the three stencil rows, the
// cells xa-1 .. xb+1 -- contiguous in cell order, so three particle ranges shared by the whole warp.  A
// warp that crosses a row end (about 2% of them) uses each lane's own stencil instead.  Each chunk of
// 32 candidates is staged in shared memory with one coalesced load per lane; every lane tests all of
// them against its own particle -- all lanes in lockstep -- by the reference's IEEE criterion and the
// active-pair matrix, and appends its accepted neighbours (sorted index and tag, candidate order).
//
// Summation order per particle = stencil rows (z, y offset), then cell order, then id order inside a
// cell: deterministic, a rounding-level reordering of the reference's list order (3D momentum adds four
// interleaved partial sums of it).
#pragma once
#include "epp_cellpair.cuh"

namespace epp {

// (2 harmonic(h_i, h_j))^2 with IEEE operations; kept out of line (rare: h_j != cached h_j).
__device__ __noinline__ float pair_r2(float hi, float hj) {
    const float h2 = harmonic2_exact(hi, hj);
    return __fmul_rn(h2, h2);
}

// The bound on dr2 against candidates of another h than the particle's own, kept from one candidate to
// the next: along a row h alternates between the particle's own and one other (fluid and walls).
struct OtherBound {
    float h, r2;
    // the bound for a candidate of h_j; own: against the particle's h, or of the default criterion
    __device__ __forceinline__ float of(float hi, float hj, float own, bool dflt) {
        if (hj == hi || dflt) return own;
        if (hj != h) {
            h = hj;
            r2 = pair_r2(hi, hj);
        }
        return r2;
    }
};

// Candidate filter: the reference's criterion (IEEE, exact) and the active-pair matrix.
template <int D>
__device__ __forceinline__ bool accept(const PairArgs& A, int i, float4 xi, unsigned amask, float h2sq,
                                       int j, float4 xj, unsigned& st) {
    if (j == i) return false;
    const float dx = __fsub_rn(xi.x, xj.x);
    const float dy = __fsub_rn(xi.y, xj.y);
    float dr2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    if (D == 3) {
        const float dz = __fsub_rn(xi.z, xj.z);
        dr2 = __fadd_rn(dr2, __fmul_rn(dz, dz));
    }
    bool ok;
    if (A.crit == EPP_CRITERION_DEFAULT) {
        ok = dr2 <= A.dom.gap_square;
    } else if (xj.w == xi.w) {
        ok = dr2 <= h2sq;
    } else {
        const float h2 = harmonic2_exact(xi.w, xj.w);
        ok = dr2 <= __fmul_rn(h2, h2);
    }
    if (!ok) return false;
    const int tj = tag_of(A.s.tagm[j]);
    if (tj < 1 || tj > A.n_tags) {
        st |= EPP_STATUS_BAD_TAG;
        return false;
    }
    return (amask >> (tj - 1)) & 1u;
}

template <int D>
__device__ __forceinline__ PairGeo geometry(float4 xi, float4 xj) {
    PairGeo g;
    g.dx = __fsub_rn(xi.x, xj.x);
    g.dy = __fsub_rn(xi.y, xj.y);
    g.dz = D == 3 ? __fsub_rn(xi.z, xj.z) : 0.0f;
    g.dr2 = __fadd_rn(__fmul_rn(g.dx, g.dx), __fmul_rn(g.dy, g.dy));
    if (D == 3) g.dr2 = __fadd_rn(g.dr2, __fmul_rn(g.dz, g.dz));
    return g;
}

template <int D>
struct TileConf {
    static constexpr int NRMAX = D == 2 ? 3 : 9;   // stencil rows: ranges of a tile or of one particle
};

// A neighbour-list entry carries the neighbour's sorted index in its low 28 bits and its tag - 1
// in the top 4 (tags are 1..EPP_MAX_TAGS = 16), so the list passes get the tag with the index
// instead of gathering it.  Contexts hold at most 2^28 particles.
constexpr int kEntryBits = 28;
__device__ __forceinline__ int list_entry(int j, int tag) { return j | ((tag - 1) << kEntryBits); }
__device__ __forceinline__ int entry_index(int e) { return e & ((1 << kEntryBits) - 1); }
__device__ __forceinline__ int entry_tag(int e) { return (int)((unsigned)e >> kEntryBits) + 1; }

struct TileMask {
    int cap;
    int* list;   // [cap * LCAP]: row i holds the neighbours (sorted indices) of particle i in order
};

template <int D>
struct ListConf {
    static constexpr int LCAP = D == 2 ? 64 : 160;   // neighbours kept per particle (multiple of 4)
    // 3D: row-major, a particle's entries contiguous (written and read 16 bytes at a time);
    // 2D: column-major, entry k of particle i at k * cap + i (a warp's reads coalesce).
    static constexpr bool ROW = D == 3;
};

// Appends a lane's neighbours to its list; entries past LCAP are counted but not stored.
// Row-major lists take one int4 store per four neighbours.
template <int D>
struct ListWriter {
    int* base;   // row of the particle (row-major) or its column origin (column-major)
    int cap;
    int b0, b1, b2;
    __device__ __forceinline__ void put(int cnt, int j) {
        if (cnt < ListConf<D>::LCAP) put_room(cnt, j);
    }
    __device__ __forceinline__ void put_room(int cnt, int j) {   // cnt < LCAP
        if (!ListConf<D>::ROW) {   // column-major: base advances one column per entry
            *base = j;
            base += cap;
            return;
        }
        // row-major: the last three entries wait in b0..b2 (oldest first); every fourth entry
        // stores the group and the row pointer moves on
        if ((cnt & 3) == 3) {
            *reinterpret_cast<int4*>(base) = make_int4(b0, b1, b2, j);
            base += 4;
        }
        b0 = b1;
        b1 = b2;
        b2 = j;
    }
    // the last partial group of a row (its unused slots are never read)
    __device__ __forceinline__ void flush(int cnt) {
        if (!ListConf<D>::ROW || cnt >= ListConf<D>::LCAP) return;
        const int r = cnt & 3;   // entries waiting: the newest r of b0..b2
        if (r == 1) *reinterpret_cast<int4*>(base) = make_int4(b2, 0, 0, 0);
        else if (r == 2) *reinterpret_cast<int4*>(base) = make_int4(b1, b2, 0, 0);
        else if (r == 3) *reinterpret_cast<int4*>(base) = make_int4(b0, b1, b2, 0);
    }
};

template <int D>
__device__ __forceinline__ ListWriter<D> list_writer(const TileMask& M, int i) {
    return ListWriter<D>{ListConf<D>::ROW ? M.list + (size_t)i * ListConf<D>::LCAP : M.list + i, M.cap, 0, 0, 0};
}

// Candidate ranges (contiguous particle index ranges) of a warp tile or of one particle.
template <int D>
struct TileRanges {
    int lo[TileConf<D>::NRMAX], len[TileConf<D>::NRMAX], cum[TileConf<D>::NRMAX];   // cum: first candidate index
    int n, total;

    __device__ __forceinline__ void add(const PairArgs& A, int row, int xa, int xb) {
        // cells xa..xb (clamped) of linear cell row `row`
        const int n0 = A.dom.n[0];
        xa = max(xa, 0);
        xb = min(xb, n0 - 1);
        int l = 0, h = 0;
        if (xa <= xb) {
            l = max(A.start[row * n0 + xa], 0);
            h = min(A.start[row * n0 + xb + 1], A.n_max);
            h = max(h, l);
        }
        lo[n] = l;
        len[n] = h - l;
        cum[n] = total;
        total += h - l;
        ++n;
    }
    // The stencil of the cells [xa, xb] of cell row (y, z): rows (y+dy, z+dz), x in [xa-1, xb+1].
    __device__ __forceinline__ void stencil(const PairArgs& A, int y, int z, int xa, int xb) {
        const int n1 = A.dom.n[1];
#pragma unroll
        for (int dz = (D == 3 ? -1 : 0); dz <= (D == 3 ? 1 : 0); ++dz) {
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                const int yy = y + dy, zz = z + dz;
                const bool in = yy >= 0 && yy < n1 && (D == 2 || (zz >= 0 && zz < A.dom.n[2]));
                if (in) add(A, yy + n1 * zz, xa - 1, xb + 1);
                else add(A, 0, 1, 0);   // empty range keeps the row slots aligned
            }
        }
    }
    // candidate index k (0 <= k < total) -> particle index: the last range starting at or before k
    // holds it (empty ranges share their successor's start, which comes after them)
    __device__ __forceinline__ int at(int k) const {
        int b = lo[0];
#pragma unroll
        for (int r = 1; r < TileConf<D>::NRMAX; ++r)
            if (r < n && k >= cum[r]) b = lo[r] - cum[r];
        return k + b;
    }
};

// Neighbour list of one lane from its own stencil (warps that cross a cell-row end): candidates
// in order, each filtered with the reference's criterion and the active-pair matrix.
template <int D>
__device__ __forceinline__ int lane_stencil_list(const PairArgs& A, ListWriter<D>& L, const TileRanges<D>& R,
                                                 int i, float4 xi, int ti, float h2sq, unsigned& st) {
    const unsigned amask = A.adj[ti - 1];
    int cnt = 0;
    for (int r = 0; r < R.n; ++r) {
        for (int j = R.lo[r]; j < R.lo[r] + R.len[r]; ++j) {
            EPP_CHECK(j >= 0 && j < A.n_max, 14, j);
            if (!accept<D>(A, i, xi, amask, h2sq, j, A.s.xh[j], st)) continue;
            L.put(cnt++, list_entry(j, tag_of(A.s.tagm[j])));
        }
    }
    return cnt;
}

// The 2D search pass of EPP_TUNING_LISTS: neighbour lists and nCount.  Each chunk of 32 candidates of the warp's union
// is staged in shared memory (position and index, one coalesced load per lane; the next chunk's
// loads are issued before the current chunk is tested); every lane tests all 32 against its own
// particle in lockstep with the reference's IEEE criterion.  A chunk whose candidates share one
// h (all of them away from material interfaces) is tested against one exact bound per lane;
// other chunks look the bound up per candidate.  One ballot per tag gives the chunk's candidates
// of each tag, so a lane keeps only the pairs its row of the active-pair matrix allows, then
// appends them to its list in candidate order.
__global__ void __launch_bounds__(128, 8)
    k_build(const __grid_constant__ PairArgs A, const __grid_constant__ TileMask M, int* ncount,
            unsigned long long* pairs) {
    __shared__ __align__(16) float s_p[4][3][32];   // staged x, y, h of a chunk (per warp)
    __shared__ int s_j[4][32];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int n_alive = min(A.start[A.dom.n_cells], A.n_max);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int w0 = i - lane;
    int cnt = 0;
    if (w0 < n_alive) {   // warp-uniform
        const bool on = i < n_alive;
        const int c_first = A.s.cell[w0];
        const int c_last = A.s.cell[min(w0 + 31, n_alive - 1)];
        EPP_CHECK(c_first >= 0 && c_first < A.dom.n_cells && c_last >= c_first && c_last < A.dom.n_cells, 11, c_last);
        const int n0 = A.dom.n[0];
        const int r0 = c_first / n0, r1 = c_last / n0;
        // tile mode: the warp's cells lie in one cell row (all but the ~2% of warps that cross
        // a row end); otherwise every lane uses its own stencil
        const bool tiled = r1 == r0;
        TileRanges<2> R;
        R.n = 0;
        R.total = 0;
        if (tiled) {
            R.stencil(A, r0 % A.dom.n[1], r0 / A.dom.n[1], c_first - r0 * n0, c_last - r0 * n0);
        } else {
            const int c = A.s.cell[min(i, n_alive - 1)];
            R.stencil(A, (c / n0) % A.dom.n[1], (c / n0) / A.dom.n[1], c % n0, c % n0);
        }
        const float4 xi = on ? A.s.xh[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const int ti = on ? tag_of(A.s.tagm[i]) : 0;
        const bool valid = on && ti >= 1 && ti <= A.n_tags;
        unsigned st = 0;
        if (on && !valid) st |= EPP_STATUS_BAD_TAG;
        const TargetConst tc = target_const<2>(on ? xi.w : 1.0f);
        const unsigned amask = valid ? A.adj[ti - 1] : 0u;
        ListWriter<2> L = list_writer<2>(M, min(i, n_alive - 1));
        if (!tiled) {
            if (valid) cnt = lane_stencil_list<2>(A, L, R, i, xi, ti, tc.h2sq, st);
        } else {
            const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
            float hc_h = xi.w;   // exact bound of the last h_j seen
            float hc_r2 = dflt ? A.dom.gap_square : tc.h2sq;
            const int nchunk = (R.total + 31) >> 5;
            // this lane's own particle in the union: the middle stencil row holds it
            constexpr int RMID = 1;
            const int k_self = on ? R.cum[RMID] + (i - R.lo[RMID]) : -1;
            // chunk 0 in flight
            bool real = lane < R.total;
            int jn = real ? R.at(lane) : 0;
            float4 xn = real ? A.s.xh[jn] : make_float4(1e30f, 1e30f, 1e30f, 0.0f);
            int tn = real ? tag_of(A.s.tagm[jn]) : 0;
            for (int ch = 0; ch < nchunk; ++ch) {
                EPP_CHECK(jn >= 0 && jn < A.n_max, 12, jn);
                // padding past the last candidate is far away: it fails every test
                s_p[wib][0][lane] = xn.x;
                s_p[wib][1][lane] = xn.y;
                s_p[wib][2][lane] = xn.w;
                s_j[wib][lane] = list_entry(jn, tn);   // appended as is (a real, allowed tag)
                const int tj = tn;
                const bool real_c = real;
                if (__ballot_sync(0xffffffffu, real_c && (tj < 1 || tj > A.n_tags))) st |= EPP_STATUS_BAD_TAG;
                // candidates whose tag this lane's row of the active-pair matrix accepts
                unsigned allowed = 0u;
                for (int t = 1; t <= A.n_tags; ++t) {
                    const unsigned of_t = __ballot_sync(0xffffffffu, real_c && tj == t);
                    if ((amask >> (t - 1)) & 1u) allowed |= of_t;
                }
                // one h for every real candidate of the chunk?
                const float h0 = __shfl_sync(0xffffffffu, xn.w, 0);
                const bool one_h = __all_sync(0xffffffffu, !real_c || xn.w == h0);
                __syncwarp();
                // next chunk's loads, in flight while this one is tested
                if (ch + 1 < nchunk) {
                    const int k = ((ch + 1) << 5) + lane;
                    real = k < R.total;
                    jn = real ? R.at(k) : 0;
                    xn = real ? A.s.xh[jn] : make_float4(1e30f, 1e30f, 1e30f, 0.0f);
                    tn = real ? tag_of(A.s.tagm[jn]) : 0;
                }
                unsigned word = 0u;
                if (one_h) {
                    if (h0 != hc_h) {
                        hc_h = h0;
                        hc_r2 = dflt ? A.dom.gap_square : h0 == xi.w ? tc.h2sq : pair_r2(xi.w, h0);
                    }
                    // dr2 <= R2 as integers: non-negative floats order like their bit patterns, so
                    // bits(dr2) - bits(R2) - 1 is negative exactly for the accepted candidates, and
                    // a funnel shift moves that sign bit into the chunk's word (candidate 0 ends in
                    // the top bit, where the append loop below starts)
                    const int nR2 = -__float_as_int(hc_r2) - 1;
                    // two candidates per packed sub / mul; dr2 = dx dx + dy dy, IEEE
                    const f32x2 XI = f2_pack(xi.x, xi.x), YI = f2_pack(xi.y, xi.y);
                    const f32x2* px = reinterpret_cast<const f32x2*>(s_p[wib][0]);
                    const f32x2* py = reinterpret_cast<const f32x2*>(s_p[wib][1]);
#pragma unroll
                    for (int b = 0; b < 16; ++b) {
                        const f32x2 dx = f2_sub(XI, px[b]);
                        const f32x2 dy = f2_sub(YI, py[b]);
                        float x0, x1, y0, y1;
                        f2_unpack(f2_mul(dx, dx), x0, x1);
                        f2_unpack(f2_mul(dy, dy), y0, y1);
                        float d0 = __fadd_rn(x0, y0), d1 = __fadd_rn(x1, y1);
                        word = __funnelshift_l((unsigned)(__float_as_int(d0) + nR2), word, 1);
                        word = __funnelshift_l((unsigned)(__float_as_int(d1) + nR2), word, 1);
                    }
                } else {
#pragma unroll 8
                    for (int b = 0; b < 32; ++b) {
                        const float4 xj = make_float4(s_p[wib][0][b], s_p[wib][1][b], 0.0f, s_p[wib][2][b]);
                        const float dx = __fsub_rn(xi.x, xj.x);
                        const float dy = __fsub_rn(xi.y, xj.y);
                        float dr2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
                        if (xj.w != hc_h) {
                            hc_h = xj.w;
                            hc_r2 = dflt ? A.dom.gap_square : xj.w == xi.w ? tc.h2sq : pair_r2(xi.w, xj.w);
                        }
                        word |= (unsigned)(dr2 <= hc_r2) << (31 - b);
                    }
                }
                // candidate b at bit 31 - b: walked from the top with count-leading-zeros
                word &= __brev(allowed);
                if ((k_self >> 5) == ch) word &= ~(0x80000000u >> (k_self & 31));   // not its own neighbour
                // this lane's neighbours among the chunk, in candidate order
                while (word) {
                    const int b = __clz(word);
                    word ^= 0x80000000u >> b;
                    L.put(cnt++, s_j[wib][b]);
                }
                __syncwarp();
            }
        }
        L.flush(cnt);
        if (st) atomicOr(A.status, st);
        if (on) ncount[i] = cnt;
    }
    count_pairs(pairs, cnt);
}

// Neighbours of particle i from its own stencil, filtered inline (used when the list of the last
// search overflowed); same order as the search pass.  Returns the sum with the count in w.
template <int D, class Act>
__device__ __noinline__ float4 neighbours_by_stencil(const PairArgs& A, int i, float4 xi, int ti,
                                                     const TargetConst& tc, const Act& act) {
    const int c = A.s.cell[i];
    const int n0 = A.dom.n[0];
    TileRanges<D> R;
    R.n = 0;
    R.total = 0;
    R.stencil(A, (c / n0) % A.dom.n[1], (c / n0) / A.dom.n[1], c % n0, c % n0);
    const unsigned amask = A.adj[ti - 1];
    unsigned st = 0;
    const typename Act::Self me = act.self(i);
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int cnt = 0;
    for (int r = 0; r < R.n; ++r)
        for (int j = R.lo[r]; j < R.lo[r] + R.len[r]; ++j) {
            const float4 xj = A.s.xh[j];
            if (!accept<D>(A, i, xi, amask, tc.h2sq, j, xj, st)) continue;
            const int tj = tag_of(A.s.tagm[j]);
            const float4 t = act.term(me, act.fetch(j, ti, tj), ti, tj, xj, geometry<D>(xi, xj), tc);
            sum.x += t.x;
            sum.y += t.y;
            sum.z += t.z;
            ++cnt;
        }
    if (st) atomicOr(A.status, st);
    sum.w = (float)cnt;
    return sum;
}

// What a list pass gathers of a neighbour (Rec), the pair's term (Term) and the sum of the terms (Acc),
// by action.  By default position and the action's own fields, the term from Act::term, each component
// added with its own rounding.  `from` is a term as lane `src` of the group holds it.
template <int D, class Act>
struct ListTerm {
    struct Me {
        float4 x;
        typename Act::Self s;
        TargetConst tc;
        int tag;
    };
    struct Rec {
        float4 x;
        typename Act::Nb nb;
    };
    struct Term {
        float x, y, z;
    };
    using Acc = Term;
    static __device__ __forceinline__ Me me(const Act& act, int i, float4 xi, int ti) {
        return Me{xi, act.self(i), target_const<D>(xi.w), ti};
    }
    static __device__ __forceinline__ Rec load(const PairArgs& A, const Act& act, const Me& m, int j, int tj) {
        return Rec{__ldg(&A.s.xh[j]), act.fetch(j, m.tag, tj)};
    }
    static __device__ __forceinline__ Term term(const Act& act, const Me& m, const Rec& r, int tj) {
        const float4 t = act.term(m.s, r.nb, m.tag, tj, r.x, geometry<D>(m.x, r.x), m.tc);
        return Term{t.x, t.y, t.z};
    }
    static __device__ __forceinline__ Term from(unsigned group, const Term& t, int src) {
        return Term{__shfl_sync(group, t.x, src), Act::NC > 1 ? __shfl_sync(group, t.y, src) : 0.0f,
                    Act::NC > 2 && D == 3 ? __shfl_sync(group, t.z, src) : 0.0f};
    }
    static __device__ __forceinline__ void add(Acc& a, const Term& t) {
        a.x = __fadd_rn(a.x, t.x);
        if (Act::NC > 1) a.y = __fadd_rn(a.y, t.y);
        if (Act::NC > 2 && D == 3) a.z = __fadd_rn(a.z, t.z);
    }
};

// The benchmark physics' momentum: du += f d as fused multiply-adds.  2D: all of a neighbour from its
// 32-byte record, one load in place of three 16-byte gathers; x and y through the packed f32x2 pipe.
template <int D, bool FUSED>
struct ListTerm<D, CPMom<D, FUSED, false>> {
    using Act = CPMom<D, FUSED, false>;
    struct Me {
        f32x2 x, v;
        float z, vz;
        typename Act::Self s;
        TargetConst tc;
    };
    struct Rec3 {
        float4 x, v;
        float2 rz;
    };
    using Rec = typename std::conditional<D == 2, Rec8, Rec3>::type;
    struct Term {
        float f, dx, dy, dz;
    };
    struct Acc {
        float x, y, z;
    };
    static __device__ __forceinline__ Me me(const Act& act, int i, float4 xi, int) {
        const typename Act::Self s = act.self(i);
        return Me{f2_pack(xi.x, xi.y), f2_pack(s.v.x, s.v.y), xi.z, s.v.z, s, target_const<D>(xi.w)};
    }
    static __device__ __forceinline__ Rec load(const PairArgs& A, const Act&, const Me&, int j, int) {
        if constexpr (D == 2) return load_rec(A.s.rec, j);
        else return Rec{__ldg(&A.s.xh[j]), __ldg(&A.s.vm[j]), __ldg(reinterpret_cast<const float2*>(A.s.rec) + j)};
    }
    static __device__ __forceinline__ Term term(const Act& act, const Me& m, const Rec& r, int tj) {
        float px, py, ux, uy;   // the neighbour's position and velocity
        if constexpr (D == 2) {
            px = r.a.x, py = r.a.y, ux = r.a.z, uy = r.a.w;
        } else {
            px = r.x.x, py = r.x.y, ux = r.v.x, uy = r.v.y;
        }
        Term t;
        const f32x2 d = f2_sub(m.x, f2_pack(px, py));
        float ex, ey, vx, vy;
        f2_unpack(d, t.dx, t.dy);
        f2_unpack(f2_mul(d, d), ex, ey);
        f2_unpack(f2_sub(m.v, f2_pack(ux, uy)), vx, vy);
        float dr2 = __fadd_rn(ex, ey);
        float vdx = __fmaf_rn(t.dy, vy, __fmul_rn(t.dx, vx));
        if constexpr (D == 2) {
            t.dz = 0.0f;
            t.f = act.pair_force(m.s, tj, r.b.x, r.b.y, r.b.z, r.b.w, dr2, vdx, m.tc);
        } else {
            t.dz = __fsub_rn(m.z, r.x.z);
            dr2 = __fadd_rn(dr2, __fmul_rn(t.dz, t.dz));
            vdx = __fmaf_rn(t.dz, __fsub_rn(m.vz, r.v.z), vdx);
            t.f = act.pair_force(m.s, tj, r.x.w, r.v.w, r.rz.x, r.rz.y, dr2, vdx, m.tc);
        }
        return t;
    }
    static __device__ __forceinline__ Term from(unsigned group, const Term& t, int src) {
        return Term{__shfl_sync(group, t.f, src), __shfl_sync(group, t.dx, src), __shfl_sync(group, t.dy, src),
                    D == 3 ? __shfl_sync(group, t.dz, src) : 0.0f};
    }
    static __device__ __forceinline__ void add(Acc& a, const Term& t) {
        a.x = __fmaf_rn(t.f, t.dx, a.x);
        a.y = __fmaf_rn(t.f, t.dy, a.y);
        if (D == 3) a.z = __fmaf_rn(t.f, t.dz, a.z);
    }
};

// 3D momentum sums four interleaved partials (every size takes the same form: there are no 3D batches).
template <int D, class Act>
constexpr bool kListInter = D == 3 && Act::NC == 3;

// sum += t with compensated (Kahan) summation.
__device__ __forceinline__ void add_compensated(float& sum, float& low, float t) {
    const float y = __fsub_rn(t, low);
    const float s = __fadd_rn(sum, y);
    low = __fsub_rn(__fsub_rn(s, sum), y);
    sum = s;
}

// neighbours_by_stencil by a group of four lanes, lanes first .. first + 3 of the warp, for the 3D list
// passes: a word of acceptance bits of every fourth candidate a lane, then a walk over the set ones.
// Where the sum is four partials each lane adds its own; an ordered one has the lanes' words
// interleaved and takes the accepted candidates four at a time, as k_list takes a list, and adds them
// with compensation: its hundreds of terms nearly cancel (largest relative error of the continuity sum
// against 64 bits at h = 2 dx over that of a plain FP32 sum, eight states: 0.3 to 0.9, and 1.1 to 9.7
// without; 561 -> 578 us at 165,888 particles).  One lane at
// work while the others of its group waited made those passes twice as long as one thread per particle
// where lists overflow (h = 2 dx, 165,888 particles: momentum 891 us with one thread, 1687 with one lane
// of four, 444 with all four; continuity 849, 1560, 578).
template <int D, class Act>
__device__ __noinline__ float4 neighbours_by_group(const PairArgs& A, int i, float4 xi, int ti, float h2sq, const Act& act,
                                                   int g, int first) {
    using T = ListTerm<D, Act>;
    constexpr bool INTER = kListInter<D, Act>;
    constexpr int N = INTER ? 32 : 8;   // candidates of a lane's word
    const unsigned group = 15u << first;
    const int c = A.s.cell[i];
    const int n0 = A.dom.n[0];
    TileRanges<D> R;
    R.n = 0;
    R.total = 0;
    R.stencil(A, (c / n0) % A.dom.n[1], (c / n0) / A.dom.n[1], c % n0, c % n0);
    const unsigned amask = A.adj[ti - 1];
    const bool dflt = A.crit == EPP_CRITERION_DEFAULT;
    const float own = dflt ? A.dom.gap_square : h2sq;
    OtherBound other{xi.w, own};
    const typename T::Me me = T::me(act, i, xi, ti);
    typename T::Acc acc{}, low{};
    int cnt = 0;
#pragma unroll 1
    for (int r = 0; r < R.n; ++r) {
        const int end = R.lo[r] + R.len[r];
#pragma unroll 1
        for (int j0 = R.lo[r]; j0 < end; j0 += 4 * N) {   // uniform in the group
            unsigned word = 0u;   // bit k: candidate j0 + g + 4 k
#pragma unroll 4
            for (int k = min((end - j0 - g + 3) >> 2, N) - 1; k >= 0; --k) {
                const float4 xj = A.s.xh[j0 + g + 4 * k];
                word = (word << 1) | (geometry<D>(xi, xj).dr2 <= other.of(xi.w, xj.w, own, dflt) ? 1u : 0u);
            }
            if constexpr (INTER) {
                while (word) {
                    const int j = j0 + g + 4 * (__ffs(word) - 1), tj = tag_of(A.s.tagm[j]);
                    word &= word - 1u;
                    if (j == i || !(__funnelshift_rc(amask, 0u, (unsigned)(tj - 1)) & 1u)) continue;
                    T::add(acc, T::term(act, me, T::load(A, act, me, j, tj), tj));
                    ++cnt;
                }
            } else {
                word = (word | word << 12) & 0x000f000fu;   // bit k to bit 4 k
                word = (word | word << 6) & 0x03030303u;
                word = (word | word << 3) & 0x11111111u;
                unsigned mask = __reduce_or_sync(group, word << g);   // bit k: candidate j0 + k
                if (i >= j0 && i < j0 + 32) mask &= ~(1u << (i - j0));
                while (mask) {   // uniform in the group
                    unsigned m = mask;   // lane g takes the g-th accepted one
                    if (g > 0) m &= m - 1u;
                    if (g > 1) m &= m - 1u;
                    if (g > 2) m &= m - 1u;
                    typename T::Term t{};
                    bool ok = false;
                    if (m) {
                        const int j = j0 + __ffs(m) - 1, tj = tag_of(A.s.tagm[j]);
                        ok = __funnelshift_rc(amask, 0u, (unsigned)(tj - 1)) & 1u;
                        if (ok) t = T::term(act, me, T::load(A, act, me, j, tj), tj);
                    }
                    const unsigned hits = __ballot_sync(group, ok) >> first;
                    cnt += __popc(hits & 15u);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const typename T::Term tu = T::from(group, t, first + u);
                        if ((hits >> u) & 1u) {
                            add_compensated(acc.x, low.x, tu.x);
                            if (Act::NC > 1) add_compensated(acc.y, low.y, tu.y);
                        }
                        mask &= mask - 1u;
                    }
                }
            }
        }
    }
    if constexpr (INTER) {
        cnt = __reduce_add_sync(group, cnt);
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            acc.x = __fadd_rn(acc.x, __shfl_xor_sync(group, acc.x, o));
            acc.y = __fadd_rn(acc.y, __shfl_xor_sync(group, acc.y, o));
            acc.z = __fadd_rn(acc.z, __shfl_xor_sync(group, acc.z, o));
        }
    }
    return make_float4(acc.x, acc.y, acc.z, (float)cnt);
}

// Blocks an SM of a list pass: 2D with one thread per particle 9 (56 registers; they beat 7, 8 and 10); in
// 3D with four lanes what the loop over a list takes, the overflow path being longer (momentum of the
// benchmark physics 64 registers, 1915 us at 6,207,228 particles, 2101 with 7 blocks; continuity 56, 41 us
// at 165,888, 46 with 7).
template <int D, class Act, int L>
constexpr int kListBlocks = L == 1 ? (D == 2 ? 9 : 4) : D == 2 ? 6 : kListInter<D, Act> ? 7 : 9;
template <bool FUSED>
constexpr int kListBlocks<3, CPMom<3, FUSED, false>, 4> = 8;

// A pair action over the neighbour lists written by the last search pass (same positions, cells and
// criterion).  L lanes share a particle, lane g takes entries k = g mod L.
//   L = 1        one thread per particle, terms added in list order
//   L = 4        every lane of the group adds a round's four terms in list order: the bits of L = 1
//                (a 2D batch and its instances alone may differ in L)
//   L = 4 INTER  (3D momentum) four partial sums, one a lane, folded as (0 + 1) + (2 + 3)
// What bounds it: the wavefronts its neighbour gathers take in the L1 (84-91% of peak in 3D) and, with
// few warps in flight, one thread's serial walk.  Lanes that share a particle gather consecutive
// entries, whose records share cache lines: 3D momentum, 955,668 particles, 308 us with L = 1 and 271
// with L = 4 (three 16-byte gathers each way; one 32-byte record for x, v made it no faster, as half as
// many particles share a line); 259 with (rho, p/rho^2) in 8 bytes as the third gather, 1968 -> 1870 at
// 6,207,228, where L = 2, 8 and 16 took 2270, 2420 and 3500.  3D continuity there: 1443 with L = 1, 1553
// with four partial sums in L = 4.  In 2D a neighbour's record fits one 32-byte load: momentum 79 -> 68 us
// at 515,018 particles.
// EPI: fused momentum step (integrate + bin for every particle, dead bin included).
template <int D, class Act, bool EPI, int L>
__global__ void __launch_bounds__(128, kListBlocks<D, Act, L>)
    k_list(const __grid_constant__ PairArgs A, const __grid_constant__ TileMask M, const int* ncount,
           const __grid_constant__ Act act) {
    using T = ListTerm<D, Act>;
    constexpr bool ROW = ListConf<D>::ROW;
    constexpr bool INTER = kListInter<D, Act> && L > 1;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(tid / L), g = (int)(tid % L);
    // what the pass starts from, read at once: one after the other (alive count, then tag, nCount, first
    // entry) these cost four latencies (2D momentum 254 -> 243 us at 2,030,018 particles with the epilogue's
    // loads before its stores, 3D 261 -> 250 at 955,668)
    const int ic = min(i, A.n_max - 1);
    const int n_alive = min(A.start[A.dom.n_cells], A.n_max);
    const float4 xi = A.s.xh[ic];
    const int ti = tag_of(A.s.tagm[ic]), cnt = ncount[ic];
    const int* const first_entry = ROW ? M.list + (size_t)ic * ListConf<D>::LCAP + g : M.list + ic + (size_t)g * M.cap;
    int en = 0;
    if constexpr (!(L == 1 && ROW)) en = ROW ? *first_entry : __ldcs(first_entry);   // stale where the list is empty
    if (i < n_alive) {
        if (ti < 1 || ti > A.n_tags || !act.wants(ti)) {
            if (g == 0) act.end_idle(i, ti);
            return;
        }
        if (cnt > ListConf<D>::LCAP) {   // more neighbours than the list keeps
            // (2D: one lane, the bits of one thread per particle whatever the physics; no slower there)
            if (D == 3 || g == 0) {
                const TargetConst tc = target_const<D>(xi.w);
                float4 sum;
                if constexpr (D == 3 && L > 1)
                    sum = neighbours_by_group<D, Act>(A, i, xi, ti, tc.h2sq, act, g, (int)(threadIdx.x & 31u & ~(unsigned)(L - 1)));
                else
                    sum = neighbours_by_stencil<D>(A, i, xi, ti, tc, act);
                const int got = (int)sum.w;
                sum.w = 0.0f;
                if (g == 0) act.end(i, ti, sum, got);
            }
            return;
        }
        const typename T::Me me = T::me(act, i, xi, ti);
        typename T::Acc acc{};
        if constexpr (L == 1 && ROW) {
            // software pipeline, neighbour k + 1's loads in flight while k's term runs; the row is
            // read four entries (16 bytes) at a time, two groups ahead (ordinary loads: a row's next
            // group shares its line), inside a group the entry is picked at compile time
            const int4* row = reinterpret_cast<const int4*>(M.list + (size_t)i * ListConf<D>::LCAP);
            int4 q = cnt > 0 ? row[0] : make_int4(0, 0, 0, 0);
            int4 qn = cnt > 4 ? row[1] : make_int4(0, 0, 0, 0);
            en = cnt > 0 ? q.x : list_entry(0, 1);
            EPP_CHECK(entry_index(en) < A.n_max, 16, entry_index(en));
            typename T::Rec rn = T::load(A, act, me, entry_index(en), entry_tag(en));
            for (int k0 = 0; k0 < cnt; k0 += 4) {
                const int4 q2 = k0 + 8 < cnt ? row[(k0 >> 2) + 2] : make_int4(0, 0, 0, 0);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = k0 + u;
                    if (k >= cnt) break;
                    const int tj = entry_tag(en);
                    const typename T::Rec r = rn;
                    if (k + 1 < cnt) {
                        en = u == 0 ? q.y : u == 1 ? q.z : u == 2 ? q.w : qn.x;
                        EPP_CHECK(entry_index(en) < A.n_max, 16, entry_index(en));
                        rn = T::load(A, act, me, entry_index(en), entry_tag(en));
                    }
                    T::add(acc, T::term(act, me, r, tj));
                }
                q = qn;
                qn = q2;
            }
        } else {
            // the lane's next entry is read ahead.  2D lists are column-major and read once each:
            // streaming loads keep the L1 for the records.
            const int* list = first_entry;
            const size_t stride = ROW ? L : (size_t)L * M.cap;
            const int first = (int)(threadIdx.x & 31u & ~(unsigned)(L - 1));
            const unsigned group = L == 1 ? 0u : ((1u << L) - 1u) << first;
            auto read = [&]() { return ROW ? *list : __ldcs(list); };
            // 2D, four lanes: the next record in flight too (step 22.5 -> 21.1 us at 1,418 particles); 3D loses to
            // the registers it takes (momentum 250 -> 300 us at 955,668)
            constexpr bool PIPE = L > 1 && D == 2;
            typename T::Rec rn;
            int tn = 1;
            if (PIPE && g < cnt) {
                EPP_CHECK(entry_index(en) < A.n_max, 16, entry_index(en));
                tn = entry_tag(en);
                rn = T::load(A, act, me, entry_index(en), tn);
                if (L + g < cnt) {
                    list += stride;
                    en = read();
                }
            }
            for (int k0 = 0; k0 < cnt; k0 += L) {
                typename T::Term t{};
                if (k0 + g < cnt) {
                    typename T::Rec r;
                    int tj;
                    if (PIPE) {
                        r = rn;
                        tj = tn;
                        if (k0 + L + g < cnt) {
                            EPP_CHECK(entry_index(en) < A.n_max, 16, entry_index(en));
                            tn = entry_tag(en);
                            rn = T::load(A, act, me, entry_index(en), tn);
                            if (k0 + 2 * L + g < cnt) {
                                list += stride;
                                en = read();
                            }
                        }
                    } else {
                        const int j = entry_index(en);
                        tj = entry_tag(en);
                        EPP_CHECK(j < A.n_max, 16, j);
                        r = T::load(A, act, me, j, tj);
                        if (k0 + L + g < cnt) {
                            list += stride;
                            en = read();
                        }
                    }
                    t = T::term(act, me, r, tj);
                    if (L == 1 || INTER) T::add(acc, t);
                }
                if constexpr (L > 1 && !INTER) {
#pragma unroll
                    for (int u = 0; u < L; ++u) {
                        const typename T::Term tu = T::from(group, t, first + u);
                        if (k0 + u < cnt) T::add(acc, tu);
                    }
                }
            }
            if constexpr (INTER) {
#pragma unroll
                for (int o = 1; o < L; o <<= 1) {
                    acc.x = __fadd_rn(acc.x, __shfl_xor_sync(group, acc.x, o));
                    if (Act::NC > 1) acc.y = __fadd_rn(acc.y, __shfl_xor_sync(group, acc.y, o));
                    if (Act::NC > 2) acc.z = __fadd_rn(acc.z, __shfl_xor_sync(group, acc.z, o));
                }
            }
        }
        if (g == 0) act.end(i, ti, make_float4(acc.x, acc.y, acc.z, 0.0f), cnt);
    } else if (EPI && i < A.n_max && g == 0) {
        act.end_idle(i, ti);
    }
}

}  // namespace epp
