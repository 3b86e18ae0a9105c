// cycles.cuh -- conflicted 3/4/5-cycle search on the CSR of attractive edges
// (src/conflicted_cycles_cuda.cu:13-343).  Each conflicted cycle is emitted
// as triangles.  Expansions (a rep edge; a rep edge and a neighbour; a rep
// edge and two neighbours) are taken in canonical order in chunks of 2^24,
// each emitting its triangles in the reference's order; a chunk whose
// emissions exceed the room left in the budget keeps them round-robin: the
// first K emissions of every expansion (K as large as fits) and one more for
// the first expansions that have one, until the budget is full.  Computed by
// count -> K -> scan -> write.
//
// What bounds the search: dependent loads.  The lists of a vertex are a
// handful to a few tens of entries anywhere in memory, so intersecting two of
// them by a merge is a chain of as many loads as they have entries; lists
// without repeated entries are compared eight by eight entries at a time
// instead (count_common_blocks), whose loads are independent.  On the 1M-point
// k-NN graph in D mode (13 attractive neighbours a vertex) the searches took 54.1 ms
// with merges and 43.5 with blocks.
#pragma once
#include "graph.cuh"

namespace rama {

struct TriBuf {
    int32_t *t1, *t2, *t3;  // capacity budget + 1
    int64_t budget;
    int64_t count;  // the reference's triangle counter (budget+1 once overflowed)
    int64_t num;    // valid entries: min(count, budget)
    int none;       // no repulsive edge has an attractive edge at both ends: no cycle of any length
    int closed;     // every side of every triangle is an edge of the graph (3-cycles only)
    int distinct;   // no triangle appears twice and none is degenerate (3-cycles of a graph without parallel edges)
};

__device__ __forceinline__ int count_common(const int32_t *adj, int32_t a0, int32_t a1, int32_t b0, int32_t b1)
{
    int c = 0;
    while (a0 < a1 && b0 < b1) {
        int32_t x = adj[a0], y = adj[b0];
        c += (x == y);
        a0 += (x <= y);
        b0 += (y <= x);
    }
    return c;
}

// calls f(mid) for the common neighbours in ascending order while f returns true
template <class F>
__device__ __forceinline__ void for_common(const int32_t *adj, int32_t a0, int32_t a1, int32_t b0, int32_t b1, F f)
{
    while (a0 < a1 && b0 < b1) {
        int32_t x = adj[a0], y = adj[b0];
        if (x == y && !f(x)) return;
        a0 += (x <= y);
        b0 += (y <= x);
    }
}

// The same for two ascending lists without repeated entries, CB entries of
// each at a time: all pairs of a block are compared (CB^2 compares, no
// dependent loads), then the block with the smaller last entry moves on, both
// when they are equal.  A common entry lies in exactly one pair of blocks that
// meet, and blocks meet in ascending order.  hit(mask, base) gets the matches
// of one pair of blocks as bits over the first list's block at `base` and
// returns whether to go on.
//
// A list's blocks start at the 16-byte boundary at or before its first entry
// (adj is 256-byte aligned and padded to 256 bytes) and are read
// by 128-bit loads; what lies outside the list is replaced by values that
// match nothing.  The lanes of a warp read different lists, so a load
// instruction costs a line per lane whatever its width.
constexpr int CB = 8;

__device__ __forceinline__ void list_block(const int32_t *adj, int32_t p, int32_t s, int32_t e, int32_t below,
                                           int32_t above, int32_t (&v)[CB])
{
    const int4 x = *reinterpret_cast<const int4 *>(adj + p);
    int4 y = make_int4(above, above, above, above);
    if (p + 4 < e) y = *reinterpret_cast<const int4 *>(adj + p + 4);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (p + k < s) v[k] = below;
#pragma unroll
    for (int k = 0; k < CB; ++k)
        if (p + k >= e) v[k] = above;
}

template <class Hit>
__device__ __forceinline__ void common_blocks(const int32_t *adj, int32_t as, int32_t a1, int32_t bs, int32_t b1,
                                              Hit hit)
{
    if (as >= a1 || bs >= b1) return;
    int32_t a[CB], b[CB];
    int32_t a0 = as & ~3, b0 = bs & ~3;
    list_block(adj, a0, as, a1, -1, 0x7fffffff, a);
    list_block(adj, b0, bs, b1, -2, 0x7ffffffe, b);
    for (;;) {
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < CB; ++k) {
            bool any = false;
#pragma unroll
            for (int q = 0; q < CB; ++q) any |= a[k] == b[q];
            m |= any ? 1u << k : 0u;
        }
        if (m && !hit(m, a0)) return;
        // a padded block is its list's last: it has no entry left behind
        const int32_t la = a0 + CB < a1 ? a[CB - 1] : 0x7fffffff;
        const int32_t lb = b0 + CB < b1 ? b[CB - 1] : 0x7fffffff;
        if (la <= lb) {
            a0 += CB;
            if (a0 >= a1) return;
            list_block(adj, a0, as, a1, -1, 0x7fffffff, a);
        }
        if (lb <= la) {
            b0 += CB;
            if (b0 >= b1) return;
            list_block(adj, b0, bs, b1, -2, 0x7ffffffe, b);
        }
    }
}

// both forms; `uniq`: the lists have no repeated entries
__device__ __forceinline__ int common_count(bool uniq, const int32_t *adj, int32_t a0, int32_t a1, int32_t b0,
                                            int32_t b1)
{
    if (!uniq) return count_common(adj, a0, a1, b0, b1);
    int c = 0;
    common_blocks(adj, a0, a1, b0, b1, [&](unsigned m, int32_t) {
        c += __popc(m);
        return true;
    });
    return c;
}

template <class F>
__device__ __forceinline__ void common_each(bool uniq, const int32_t *adj, int32_t a0, int32_t a1, int32_t b0,
                                            int32_t b1, F f)
{
    if (!uniq) {
        for_common(adj, a0, a1, b0, b1, f);
        return;
    }
    common_blocks(adj, a0, a1, b0, b1, [&](unsigned m, int32_t base) {
        for (; m; m &= m - 1)
            if (!f(adj[base + __ffs(m) - 1])) return false;
        return true;
    });
}

__device__ __forceinline__ void write_tri(const TriBuf &tb, int64_t pos, int32_t a, int32_t b, int32_t c)
{
    if (pos >= tb.budget) return;
    int32_t lo = min(a, min(b, c)), hi = max(a, max(b, c));
    int32_t md = max(min(a, b), min(max(a, b), c));
    tb.t1[pos] = lo;
    tb.t2[pos] = md;
    tb.t3[pos] = hi;
}

// Remove degenerate triangles, sort lexicographically, unique (the first n
// entries of the buffer); returns the new count.  By buckets of the smallest
// vertex, degenerate triangles in none: a triangle travels as a record (middle
// vertex, largest vertex, -, smallest vertex) and the tile pass orders the
// buckets in shared memory and writes the triangles in order.  (With every
// triangle ranked against its bucket in global memory and written to its place
// from there, the triangles of the 1M-point k-NN graph in D mode took 24.4 ms.)
// With tb.distinct the sorted triangles go to new arrays that take the
// buffer's place; otherwise a scan drops repetitions on the way back.
template <class Team>
__device__ __noinline__ int64_t tri_normalize(const Team &t, Scratch &sc, char *, TriBuf &tb, int64_t n, int32_t nmax)
{
    if (n == 0) return 0;
    char *sm = team_smem();
    const int nb = bits_for((uint64_t)(nmax > 0 ? nmax : 1));
    int32_t *t1 = tb.t1, *t2 = tb.t2, *t3 = tb.t3;
    const bool distinct = tb.distinct != 0;
    const uint64_t m0 = sc.arena.mark();
    int32_t *o1 = sc.arena.take<int32_t>(n + 1), *o2 = sc.arena.take<int32_t>(n + 1),
            *o3 = sc.arena.take<int32_t>(n + 1);
    const uint64_t m1 = sc.arena.mark();
    const int32_t nbk = nmax + 1;
    Records R;
    R.rec = sc.arena.take<int4>(n + 1);
    R.start = sc.arena.take<int32_t>((int64_t)nbk + 1);
    R.slot = sc.arena.take<int32_t>(n + 1);
    R.lohi = nullptr;
    BucketLists L = bucket_lists(sc, n);
    if (!sc.arena.ok()) return 0;
    int4 *rec = R.rec;
    int32_t *start = R.start, *slot = R.slot;
    const uint64_t mask = (nb == 0) ? 0 : ((uint64_t(1) << nb) - 1);
    struct Tri {
        int32_t lo, md, hi;
        __device__ bool ok() const { return lo != md && md != hi; }
    };
    auto tri = [=](int64_t k) {
        const int32_t a = t1[k], b = t2[k], c = t3[k];
        Tri r;
        r.lo = min(a, min(b, c));
        r.hi = max(a, max(b, c));
        r.md = max(min(a, b), min(max(a, b), c));
        return r;
    };
    for (int64_t v = t.rank(); v <= nbk; v += t.size()) start[v] = 0;
    if (t.rank() < 4) L.n[t.rank()] = 0;
    t.sync();
    {
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        for (int64_t base = (int64_t)t.rank() - lane_id(); base < n; base += S * U) {
            int32_t b[U], s[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int64_t q = base + k * S + lane_id();
                const Tri r = tri(q < n ? q : n - 1);
                b[k] = q < n && r.ok() ? r.lo : -1;
            }
            bucket_slots<U>(start, b, s);
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (base + k * S + lane_id() < n) slot[base + k * S + lane_id()] = s[k];
        }
    }
    t.sync();
    const int64_t w = team_bucket_starts(t, sc, sm, nbk, start, L, [](int64_t, int32_t, int32_t) {});
    if (!L.has_big()) {
        team_for_batched(
            t, n,
            [=](int64_t k) {
                const Tri r = tri(k);
                return make_int4(r.md, r.hi, r.ok() ? start[r.lo] + slot[k] : -1, r.lo);
            },
            [=](int64_t, int4 v) {
                if (v.z >= 0) rec[v.z] = v;
            });
        t.sync();
        team_sort_long_records(t, sm, R, L);
        team_record_tiles<true>(t, sm, R, w,
                                [&](const RecTile<int4> &T, int base, const int4 (&)[4], const bool (&mine)[4]) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k)
                                        if (mine[k]) {
                                            const int4 r = T.win[base + 32 * k];
                                            const int64_t p = T.p0 + base + 32 * k;
                                            o1[p] = r.w;
                                            o2[p] = r.x;
                                            o3[p] = r.y;
                                        }
                                });
        t.sync();
    } else {
        // a vertex with more than BUCKET_MAX triangles: LSD radix, stable sort
        // by hi carrying (lo, md), then by (lo, md) carrying hi
        uint64_t *k1 = sc.arena.take<uint64_t>(n + 1), *k2 = sc.arena.take<uint64_t>(n + 1);
        uint64_t *u1 = reinterpret_cast<uint64_t *>(rec), *u2 = u1 + (n + 1);  // (the records are not used here)
        if (!sc.arena.ok()) return 0;
        team_compact(
            t, sc, sm, n, [=](int64_t k) { return tri(k).ok(); },
            [=](int64_t k, int64_t p) {
                const Tri r = tri(k);
                k1[p] = (uint64_t)(uint32_t)r.hi;
                u1[p] = pack_key(r.lo, r.md, nb);
            });
        team_sort_pairs(t, sc, sm, k1, u1, k2, u2, w, nb);
        for (int64_t k = t.rank(); k < w; k += t.size()) {
            uint64_t tmp = u1[k];
            u1[k] = k1[k];  // hi becomes the value
            k1[k] = tmp;
        }
        t.sync();
        team_sort_pairs(t, sc, sm, k1, u1, k2, u2, w, 2 * nb);
        for (int64_t k = t.rank(); k < w; k += t.size()) {
            o1[k] = (int32_t)(k1[k] >> nb);
            o2[k] = (int32_t)(k1[k] & mask);
            o3[k] = (int32_t)u1[k];
        }
        t.sync();
    }
    if (distinct) {
        tb.t1 = o1;
        tb.t2 = o2;
        tb.t3 = o3;
        sc.arena.release(m1);
        return w;
    }
    const int64_t u = team_compact(
        t, sc, sm, w,
        [=](int64_t k) { return k == 0 || o1[k] != o1[k - 1] || o2[k] != o2[k - 1] || o3[k] != o3[k - 1]; },
        [=](int64_t k, int64_t p) {
            t1[p] = o1[k];
            t2[p] = o2[k];
            t3[p] = o3[k];
        });
    sc.arena.release(m0);
    return u;
}

// The lists of attractive neighbours (cost > pos_tol), ascending: vertex v's
// are adj[off[v], off[v + 1]).  By buckets of the vertex, each edge in two, as
// records (neighbour, vertex) that the tile pass orders in shared memory.
// Every edge's ends are loaded along with its cost: about half of the edges
// are attractive, so nearly every sector is needed.  With loads behind the
// cost's branch and each entry ranked in global memory by one thread, the
// lists of the 1M-point k-NN graph in D mode took 16.1 ms.
// `off` holds nrows + 1 zeros.  Returns false, with off used up, when a vertex
// has more than BUCKET_MAX neighbours.
template <class Team>
__device__ __noinline__ bool attractive_lists(const Team &t, Scratch &sc, char *, const Graph &graph, int32_t nrows,
                                              float pos_tol, int32_t *off, int32_t *&adj_out, int64_t &m2)
{
    char *sm = team_smem();
    const Graph A = graph;  // its pointers in registers
    int32_t *adj = sc.arena.take<int32_t>(2 * A.n + 1);
    adj_out = adj;
    const uint64_t m = sc.arena.mark();
    RecordArray<int2> R;
    R.rec = sc.arena.take<int2>(2 * A.n + 1);
    R.start = off;
    int2 *rec = R.rec;
    int2 *slot = sc.arena.take<int2>(A.n + 1);
    BucketLists L = bucket_lists(sc, 2 * A.n);
    m2 = 0;
    if (!sc.arena.ok()) return true;
    if (t.rank() < 4) L.n[t.rank()] = 0;
    {
        // SORT_BATCH strides of a warp at a time: the edges, then the atomics
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        for (int64_t base = (int64_t)t.rank() - lane_id(); base < A.n; base += S * U) {
            int32_t r[U], c[U], sr[U], sc2[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int64_t e = base + k * S + lane_id(), x = e < A.n ? e : A.n - 1;
                const float w = A.cost[x];
                r[k] = A.row[x];
                c[k] = A.col[x];
                if (!(e < A.n && w > pos_tol)) r[k] = -1;
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                sc2[k] = 0;
                if (r[k] >= 0) sc2[k] = atomicAdd(&off[c[k]], 1);
            }
            bucket_slots<U>(off, r, sr);
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (r[k] >= 0) slot[base + k * S + lane_id()] = make_int2(sr[k], sc2[k]);
        }
    }
    t.sync();
    m2 = team_bucket_starts(t, sc, sm, nrows, off, L, [](int64_t, int32_t, int32_t) {});
    if (L.has_big()) {
        // every thread has seen it before the caller, which writes to this
        // memory next, goes on
        t.sync();
        sc.arena.release(m);
        return false;
    }
    struct Ends {
        int32_t r, c, pr, pc;  // r: -1 if not attractive
    };
    team_for_batched(
        t, A.n,
        [=](int64_t e) {
            const float w = A.cost[e];
            const int2 s = slot[e];  // (not set where it is not used)
            Ends x;
            x.r = A.row[e];
            x.c = A.col[e];
            const bool pos = w > pos_tol;
            x.pr = off[pos ? x.r : 0] + s.x;
            x.pc = off[pos ? x.c : 0] + s.y;
            if (!pos) x.r = -1;
            return x;
        },
        [=](int64_t, Ends x) {
            if (x.r < 0) return;
            rec[x.pr] = make_int2(x.c, x.r);
            rec[x.pc] = make_int2(x.r, x.c);
        });
    t.sync();
    if (L.has_long()) {
        team_sort_long_buckets<uint32_t>(
            t, sm, L, off, [=](int32_t p) { return (uint32_t)rec[p].x; },
            [=](int32_t v, int32_t p, uint32_t key) { rec[p] = make_int2((int32_t)key, v); });
        t.sync();
    }
    team_record_tiles<true>(t, sm, R, m2, [&](const RecTile<int2> &T, int base, const int2 (&)[4], const bool (&mine)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (mine[k]) adj[T.p0 + base + 32 * k] = T.win[base + 32 * k].x;
    });
    t.sync();
    sc.arena.release(m);
    return true;
}

// Expansion stage over X expansions (X given as an exclusive scan xo[R+1]
// over rep edges; xo == nullptr means one expansion per rep edge).  For each
// expansion: count(x) emissions, then write them at `count + prefix`.
// Processed in chunks so that a filled budget stops the work early.
__device__ __forceinline__ int64_t expansion_owner(const int64_t *xo, int64_t R, int64_t x)
{
    if (!xo) return x;
    int64_t lo = 0, hi = R;  // largest r with xo[r] <= x
    while (lo < hi) {
        int64_t mid = (lo + hi + 1) >> 1;
        if (xo[mid] <= x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// The owners of a run of consecutive expansions, taken by a warp 32 at a
// time: one search (a probe per lane) for the first, then every lane steps
// forward from the last owner of the 32 before it.  Runs of up to EXP_RUN
// times 32, shorter where that would leave warps without work, and 1 where an
// expansion is a rep edge and needs no search.
constexpr int EXP_RUN = 8;

struct OwnerWalk {
    int64_t r0;
    __device__ __forceinline__ void start(const int64_t *xo, int64_t R, int64_t x)
    {
        if (!xo) return;
        int64_t lo = 0, hi = R;  // largest r in [lo, hi] with xo[r] <= x
        while (hi - lo > 0) {
            const int64_t step = (hi - lo + 31) / 32;
            const int64_t probe = lo + (lane_id() + 1) * step;
            const unsigned m = __ballot_sync(FULL, probe <= hi && xo[probe] <= x);
            const int k = __popc(m);  // probes that hold are a prefix
            lo += k * step;
            hi = k == 32 ? hi : min(hi, lo + step - 1);
        }
        r0 = lo;
    }
    // the owner of expansion x (x ascends by 32 per call, one per lane)
    __device__ __forceinline__ int64_t next(const int64_t *xo, int64_t R, int64_t x, bool valid)
    {
        if (!xo) return x;
        int64_t r = r0;
        if (valid) {
            int steps = 0;  // long runs of rep edges without expansions: search instead
            while (r < R && xo[r + 1] <= x && ++steps <= 64) ++r;
            if (steps > 64) r = expansion_owner(xo, R, x);
        }
        const unsigned v = __ballot_sync(FULL, valid);
        if (v) r0 = __shfl_sync(FULL, r, 31 - __clz(v));
        return r;
    }
};

// Bins of the histogram of emissions per expansion (the last one: all larger).
constexpr int EXP_BINS = 1024;

// emit(r, loc, pos, keep) writes the first `keep` emissions of an expansion
// at pos, pos + 1, ...
template <class Team, class Count, class Emit>
__device__ __forceinline__ void expansion_stage(const Team &t, Scratch &sc, char *sm, TriBuf &tb, const int64_t *xo,
                                                int64_t R, int64_t X, Count cnt, Emit emit)
{
    const int64_t CH = int64_t(1) << 24;
    const int64_t KALL = int64_t(1) << 40;  // no truncation: every emission is kept
    uint64_t m = sc.arena.mark();
    int32_t *ccount = sc.arena.take<int32_t>(CH < X ? CH : X + 1);
    int32_t *cbase = sc.arena.take<int32_t>((CH < X ? CH : X) + 1);
    int32_t *hist = sc.arena.take<int32_t>(EXP_BINS);
    if (!sc.arena.ok()) return;
    int64_t count = tb.count;
    const int64_t budget = tb.budget;
    for (int64_t x0 = 0; x0 < X && count <= budget; x0 += CH) {
        const int64_t xn = (X - x0) < CH ? (X - x0) : CH;
        const int64_t share = xn / (32 * (int64_t)team_nwarps(t));
        const int run = !xo || share < 1 ? 1 : (share > EXP_RUN ? EXP_RUN : (int)share);
        // count
        int64_t mine = 0;
        for (int64_t qb = (int64_t)team_warp(t) * (32 * run); qb < xn; qb += (int64_t)team_nwarps(t) * (32 * run)) {
            OwnerWalk ow;
            ow.start(xo, R, x0 + qb);
            for (int k = 0; k < run; ++k) {
                const int64_t q = qb + 32 * k + lane_id();
                const bool valid = q < xn;
                const int64_t x = x0 + q, r = ow.next(xo, R, x, valid);
                if (!valid) continue;
                const int32_t c = cnt(r, xo ? x - xo[r] : 0);
                ccount[q] = c;
                mine += c;
            }
        }
        for (int64_t b = t.rank(); b < EXP_BINS; b += t.size()) hist[b] = 0;
        const int64_t tot = team_total<Team, int64_t>(t, sc, sm, mine);
        const int64_t start = count;
        const int64_t rem = budget - start;
        if (tot > rem && rem == 0) {
            // No room for any of them.  The histogram must not be read here:
            // nothing would sync between that and the caller's next writes to
            // this stage's workspace.
            count = budget + 1;
            break;
        }
        // round-robin when the chunk does not fit: the largest K with
        // sum_q min(count_q, K) <= rem, and `extra` expansions keep one more.
        // K from a histogram of the counts; by bisection over sums where it
        // lies beyond the histogram.
        int64_t K = KALL, extra = 0;
        if (tot > rem) {
            int32_t *lh = reinterpret_cast<int32_t *>(sm);
            for (int b = threadIdx.x; b < EXP_BINS; b += blockDim.x) lh[b] = 0;
            __syncthreads();
            for (int64_t q = t.rank(); q < xn; q += t.size()) {
                const int32_t c = ccount[q];
                if (c > 0) atomicAdd(&lh[c < EXP_BINS - 1 ? c : EXP_BINS - 1], 1);
            }
            __syncthreads();
            for (int b = threadIdx.x; b < EXP_BINS; b += blockDim.x)
                if (lh[b]) atomicAdd(&hist[b], lh[b]);
            t.sync();
            // The CTA takes the bins to shared memory and one warp finds K:
            // lane l holds bins 32 l .. 32 l + 31.  (With every warp of the
            // grid reading the bins from L2 a truncation took 0.35 ms.)
            for (int b = threadIdx.x; b < EXP_BINS; b += blockDim.x) lh[b] = __ldcg(hist + b);
            __shared__ int64_t best[2];
            __syncthreads();
            if (warp_in_block() == 0) {
                constexpr int PER = EXP_BINS / 32;
                int64_t n_l = 0, s_l = 0;  // expansions and emissions of the lane's bins
                for (int k = 0; k < PER; ++k) {
                    const int b = lane_id() * PER + k;
                    n_l += lh[b];
                    s_l += (int64_t)lh[b] * b;
                }
                // expansions in higher bins, and emissions in lower ones
                const int64_t n_all = warp_sum(n_l);
                int64_t above = n_all - (warp_incl_scan(n_l) - n_l);  // counts >= the lane's first bin
                int64_t below = warp_incl_scan(s_l) - s_l;
                // S(k) = below(k) + k * (counts >= k), for k up to EXP_BINS - 1
                int64_t bestk = -1, bests = 0;
                for (int k = 0; k < PER; ++k) {
                    const int64_t b = lane_id() * PER + k;
                    const int64_t S = below + b * above;
                    if (S <= rem) {
                        bestk = b;
                        bests = S;
                    }
                    below += (int64_t)lh[b] * b;
                    above -= lh[b];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const int64_t ok = __shfl_xor_sync(FULL, bestk, o), os = __shfl_xor_sync(FULL, bests, o);
                    if (ok > bestk) {
                        bestk = ok;
                        bests = os;
                    }
                }
                if (lane_id() == 0) {
                    best[0] = bestk;
                    best[1] = bests;
                }
            }
            __syncthreads();
            const int64_t bestk = best[0], bests = best[1];
            int64_t lo = bestk, slo = bests;  // S(0) = 0 always fits
            if (lo == EXP_BINS - 1) {
                const int32_t mx = team_max<Team, int32_t>(t, sc, sm, xn, 0, [=](int64_t q) { return ccount[q]; });
                int64_t hi = mx;
                for (int guard = 0; lo < hi && guard < 40; ++guard) {
                    const int64_t k = (lo + hi + 1) >> 1;
                    const int64_t s = team_sum<Team, int64_t>(t, sc, sm, xn, [=](int64_t q) -> int64_t {
                        const int64_t c = ccount[q];
                        return c < k ? c : k;
                    });
                    if (s <= rem) {
                        lo = k;
                        slo = s;
                    } else {
                        hi = k - 1;
                    }
                }
            }
            K = lo;
            extra = rem - slo;
            __syncthreads();
        }
        if (tot > 0) {  // (and rem > 0)
            // positions: one scan of (kept below K) << 25 | (has more than K);
            // count_q is replaced by the number it keeps
            team_scan<Team, int64_t>(
                t, sc, sm, xn,
                [=](int64_t q) -> int64_t {
                    const int64_t c = ccount[q];
                    return ((c < K ? c : K) << 25) | (c > K ? 1 : 0);
                },
                [=](int64_t q, int64_t pre, int64_t v) {
                    const int64_t pmin = pre >> 25, pbig = pre & ((int64_t(1) << 25) - 1);
                    cbase[q] = (int32_t)(pmin + (pbig < extra ? pbig : extra));
                    ccount[q] = (int32_t)((v >> 25) + ((v & 1) && pbig < extra ? 1 : 0));
                });
            for (int64_t qb = (int64_t)team_warp(t) * (32 * run); qb < xn;
                 qb += (int64_t)team_nwarps(t) * (32 * run)) {
                OwnerWalk ow;
                ow.start(xo, R, x0 + qb);
                for (int k = 0; k < run; ++k) {
                    const int64_t q = qb + 32 * k + lane_id();
                    const bool valid = q < xn;
                    const int64_t x = x0 + q, r = ow.next(xo, R, x, valid);
                    if (!valid || ccount[q] == 0) continue;
                    emit(r, xo ? x - xo[r] : 0, start + cbase[q], (int64_t)ccount[q]);
                }
            }
            t.sync();
        }
        count = tot <= rem ? start + tot : budget + 1;
    }
    tb.count = count;
    sc.arena.release(m);
}

// conflicted_cycles_cuda (:222-343).  Triangles land in tb (allocated here
// in the temporaries); tb.count is the reference's counter.  `ordered` keeps
// the order of the reference's buffer, which sorts the triangles between the
// cycle lengths; the dual sorts them once at the end, so it sorts in between
// only where repetitions have to go (their number decides what fits the
// budget).
template <class Team>
__device__ __noinline__ void conflicted_cycles(const Team &t, Scratch &sc, char *, const Graph &graph, int max_len,
                                               float tri_factor, float tol, bool ordered, TriBuf &tb)
{
    char *sm = team_smem();
    const Graph A = graph;  // its pointers in registers
    tb.count = 0;
    tb.num = 0;
    tb.budget = 0;
    tb.none = 0;
    tb.closed = 1;
    const bool uniq = A.uniq != 0;
    tb.distinct = uniq;
    tb.t1 = tb.t2 = tb.t3 = nullptr;
    if (max_len < 3 || A.n == 0) return;
    // the smallest cost: known from the pass that built the graph, or one pass
    const float mn = A.cmin == A.cmin
                         ? A.cmin
                         : team_min<Team, float>(t, sc, sm, A.n, 3.4e38f, [=](int64_t e) { return A.cost[e]; });
    const float thresh = mn * tol;          // determine_threshold (:170-174)
    const float pos_tol = -1.0f * thresh;   // create_matrices (:176-220)
    const int32_t N = A.max_dim();
    // Every conflicted cycle closes a repulsive edge (u, v) with a path of
    // attractive edges, so both u and v have an attractive edge.  Repulsive
    // edges without one at either end emit nothing: they are left out of the
    // search (the emission order of the others, and so the budget's
    // truncation, is unchanged), and a graph with none left needs no lists.
    int2 *rep = sc.arena.take<int2>(A.n + 1);  // the kept repulsive edges' ends
    int8_t *haspos = sc.arena.take<int8_t>((int64_t)N + 1);
    int32_t *off = sc.arena.take<int32_t>((int64_t)N + 2);
    if (!sc.arena.ok()) return;
    for (int64_t v = t.rank(); v < N; v += t.size()) haspos[v] = 0;
    for (int64_t v = t.rank(); v <= N; v += t.size()) off[v] = 0;
    t.sync();
    // (all three arrays loaded at once: about half of the edges are attractive,
    // so nearly every sector is needed, and no load waits for another)
    team_for_batched(
        t, A.n, [=](int64_t e) { return make_int3(A.row[e], A.col[e], __float_as_int(A.cost[e])); },
        [=](int64_t, int3 v) {
            if (__int_as_float(v.z) > pos_tol) {
                haspos[v.x] = 1;
                haspos[v.y] = 1;
            }
        });
    t.sync();
    // one pass counts both: the low 32 bits count every repulsive edge (the
    // budget counts them all, :247), the high bits the kept ones; the kept
    // ones are compacted only when there are any
    // (the loads of several edges in flight together: none is skipped, an edge
    // that is not repulsive looks at vertex 0)
    auto rep_code = [=](int64_t e) -> int64_t {
        const bool rep = A.cost[e] < thresh;
        const int32_t r = A.row[e], c = A.col[e];
        const int8_t a = haspos[rep ? r : 0], b = haspos[rep ? c : 0];
        return rep ? ((a & b) != 0 ? (int64_t(1) << 32) + 1 : 1) : 0;
    };
    const int64_t packed = team_scan_while<Team, int64_t>(
        t, sc, sm, A.n, rep_code, [](int64_t total) { return (total >> 32) != 0; },
        [=](int64_t e, int64_t pre, int64_t v) {
            if (v >> 32) rep[pre >> 32] = make_int2(A.row[e], A.col[e]);
        });
    const int64_t Rall = packed & 0xffffffffll;
    const int64_t R = packed >> 32;
    sc.alg_bytes += 12.0 * (double)A.n;
    if (R == 0) {
        tb.none = 1;
        prof_mark(t, sc, PH_CYCLES);
        return;
    }
    prof_mark(t, sc, PH_CYCLES);
    int32_t *adj = nullptr;
    int64_t m2 = 0;
    if (A.n >= (int64_t(1) << 30) || !attractive_lists(t, sc, sm, A, N, pos_tol, off, adj, m2)) {
        Csr C = build_symmetric_csr(t, sc, sm, A, N, [=](int64_t e) { return A.cost[e] > pos_tol; });
        off = C.off;
        adj = C.adj;
        m2 = C.m2;
    }
    prof_mark(t, sc, PH_CSR);
    const int64_t budget = (int64_t)(int32_t)(tri_factor * (float)Rall);  // (:247)
    tb.budget = budget < 0 ? 0 : budget;
    tb.t1 = sc.arena.take<int32_t>(tb.budget + 1);
    tb.t2 = sc.arena.take<int32_t>(tb.budget + 1);
    tb.t3 = sc.arena.take<int32_t>(tb.budget + 1);
    int64_t *xo = max_len >= 4 ? sc.arena.take<int64_t>(R + 2) : nullptr;
    if (!sc.arena.ok()) return;
    auto stage_normalize = [&]() {
        const int distinct = tb.distinct;
        if (distinct && !ordered) return;
        tb.distinct = 0;  // sorted in place
        tb.count = tri_normalize(t, sc, sm, tb, tb.count, N);
        tb.distinct = distinct;
    };
    // ---- 3-cycles: find_triangles_parallel (:31-61)
    {
        const TriBuf T = tb;
        expansion_stage(
            t, sc, sm, tb, nullptr, R, R,
            [=](int64_t r, int64_t) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                return common_count(uniq, adj, off[v1], off[v1 + 1], off[v2], off[v2 + 1]);
            },
            [=](int64_t r, int64_t, int64_t pos, int64_t keep) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                int64_t e = 0;
                common_each(uniq, adj, off[v1], off[v1 + 1], off[v2], off[v2 + 1], [&](int32_t mid) {
                    write_tri(T, pos + e, v1, v2, mid);
                    return ++e < keep;
                });
            });
    }
    // ---- 4-cycles: find_quadrangles_parallel (:63-101)
    if (max_len >= 4 && tb.count < tb.budget) {
        stage_normalize();
        const int64_t X = team_scan<Team, int64_t>(
            t, sc, sm, R, [=](int64_t r) -> int64_t { const int32_t v1 = rep[r].x; return off[v1 + 1] - off[v1]; },
            [=](int64_t r, int64_t pre, int64_t) { xo[r] = pre; });
        if (t.rank() == 0) xo[R] = X;
        t.sync();
        const TriBuf T = tb;
        const int64_t before = tb.count;
        expansion_stage(
            t, sc, sm, tb, xo, R, X,
            [=](int64_t r, int64_t loc) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                int32_t n1 = adj[off[v1] + loc];
                return 2 * common_count(uniq, adj, off[n1], off[n1 + 1], off[v2], off[v2 + 1]);
            },
            [=](int64_t r, int64_t loc, int64_t pos, int64_t keep) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                int32_t n1 = adj[off[v1] + loc];
                int64_t e = 0;
                common_each(uniq, adj, off[n1], off[n1 + 1], off[v2], off[v2 + 1], [&](int32_t mid) {
                    write_tri(T, pos + e, v1, v2, n1);
                    if (++e >= keep) return false;
                    write_tri(T, pos + e, v2, n1, mid);
                    return ++e < keep;
                });
            });
        if (tb.count != before) tb.closed = tb.distinct = 0;
    }
    // ---- 5-cycles: find_pentagons_parallel (:103-148)
    if (max_len >= 5 && tb.count < tb.budget) {
        stage_normalize();
        const int64_t X = team_scan<Team, int64_t>(
            t, sc, sm, R,
            [=](int64_t r) -> int64_t {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                return (int64_t)(off[v1 + 1] - off[v1]) * (int64_t)(off[v2 + 1] - off[v2]);
            },
            [=](int64_t r, int64_t pre, int64_t) { xo[r] = pre; });
        if (t.rank() == 0) xo[R] = X;
        t.sync();
        const TriBuf T = tb;
        const int64_t before = tb.count;
        expansion_stage(
            t, sc, sm, tb, xo, R, X,
            [=](int64_t r, int64_t loc) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                const uint32_t d1 = (uint32_t)(off[v1 + 1] - off[v1]);
                // (loc < d1 * d2, which fits 32 bits unless both lists are long)
                const bool small = loc < (int64_t(1) << 32);
                const int32_t q2 = small ? (int32_t)((uint32_t)loc / d1) : (int32_t)(loc / d1);
                const int32_t q1 = (int32_t)(loc - (int64_t)q2 * d1);
                const int32_t n1 = adj[off[v1] + q1];
                const int32_t n2 = adj[off[v2] + q2];
                if (n1 == n2) return 0;
                return 3 * common_count(uniq, adj, off[n1], off[n1 + 1], off[n2], off[n2 + 1]);
            },
            [=](int64_t r, int64_t loc, int64_t pos, int64_t keep) {
                const int32_t v1 = rep[r].x, v2 = rep[r].y;
                const uint32_t d1 = (uint32_t)(off[v1 + 1] - off[v1]);
                // (loc < d1 * d2, which fits 32 bits unless both lists are long)
                const bool small = loc < (int64_t(1) << 32);
                const int32_t q2 = small ? (int32_t)((uint32_t)loc / d1) : (int32_t)(loc / d1);
                const int32_t q1 = (int32_t)(loc - (int64_t)q2 * d1);
                const int32_t n1 = adj[off[v1] + q1];
                const int32_t n2 = adj[off[v2] + q2];
                if (n1 == n2) return;
                int64_t e = 0;
                common_each(uniq, adj, off[n1], off[n1 + 1], off[n2], off[n2 + 1], [&](int32_t mid) {
                    write_tri(T, pos + e, v1, v2, n1);
                    if (++e >= keep) return false;
                    write_tri(T, pos + e, v2, n1, mid);
                    if (++e >= keep) return false;
                    write_tri(T, pos + e, v2, mid, n2);
                    return ++e < keep;
                });
            });
        if (tb.count != before) tb.closed = tb.distinct = 0;
    }
    tb.num = tb.count < tb.budget ? tb.count : tb.budget;
    sc.alg_bytes += 8.0 * (double)R + 4.0 * (double)m2 + 12.0 * (double)tb.num;
}

}  // namespace rama
