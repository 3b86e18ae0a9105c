// graph.cuh -- the device graph store (directed COO, row<col, sorted by
// (row,col)) and its coarsening.  Restates dCOO (include/dCOO.h:13-121,
// src/dCOO.cu:14-172) with one radix sort of packed (row,col) keys per
// coarsening and a deterministic segmented sum of parallel edges.
#pragma once
#include "prims.cuh"

namespace rama {

struct Graph {
    int32_t *row, *col;
    float *cost;
    int64_t n;
    int32_t rows, cols;  // dCOO::rows_ / cols_
    float cmin;          // smallest cost of an edge with row != col (NaN: not known)
    int32_t ecols;       // largest column of an edge + 1 (rows / cols keep dims from before the diagonal went)
    int uniq;            // no two edges share both ends and none is a self-loop (0: not known)
    __device__ __forceinline__ int32_t max_dim() const { return rows > cols ? rows : cols; }
};

__device__ __forceinline__ float unknown_cost() { return __int_as_float(0x7fc00000); }

// Scratch arrays of a new graph, allocated in the temporaries.
template <class Team>
__device__ Graph graph_alloc(const Team &t, Scratch &sc, int64_t n)
{
    Graph g;
    g.row = sc.arena.take<int32_t>(n + 1);
    g.col = sc.arena.take<int32_t>(n + 1);
    g.cost = sc.arena.take<float>(n + 1);
    g.n = n;
    g.rows = g.cols = 0;
    g.cmin = unknown_cost();
    g.ecols = 0;
    g.uniq = 0;
    return g;
}

// Move a graph built in the temporaries into the top slot of the arena
// (the slot ends at the arena's end; the old graph there is dead).  Fails
// (team-uniformly) if the slot would overlap live temporaries.
template <class Team>
__device__ Graph graph_commit(const Team &t, Scratch &sc, const Graph &src)
{
    Arena &a = sc.arena;
    uint64_t bytes = (uint64_t)(src.n + 1) * 12 + 3 * 256;
    uint64_t top = (a.cap - bytes) & ~uint64_t(255);
    Graph g = src;
    if (a.failed || bytes > a.cap || top < a.lo) {
        a.failed = 1;
        return src;
    }
    g.row = reinterpret_cast<int32_t *>(a.base + top);
    g.col = reinterpret_cast<int32_t *>(a.base + top + ((uint64_t)(src.n + 1) * 4 + 255) / 256 * 256);
    g.cost = reinterpret_cast<float *>(a.base + top + 2 * (((uint64_t)(src.n + 1) * 4 + 255) / 256 * 256));
    // source lies in the temporaries, strictly below `top`: no overlap
    for (int64_t e = t.rank(); e < src.n; e += t.size()) {
        g.row[e] = src.row[e];
        g.col[e] = src.col[e];
        g.cost[e] = src.cost[e];
    }
    a.top = top;
    t.sync();
    return g;
}

// dims as in dCOO::init (src/dCOO.cu:47-51): rows = last row + 1,
// cols = max col + 1 (0 for an empty graph); in the same pass, the smallest
// cost of an edge that is not a self-loop (dCOO::min of the graph once its
// diagonal is removed; the cycle search's threshold, src/conflicted_cycles_cuda.cu:170-174)
template <class Team>
__device__ void graph_set_dims(const Team &t, Scratch &sc, char *sm, Graph &g)
{
    if (g.n == 0) {
        g.rows = g.cols = g.ecols = 0;
        g.cmin = unknown_cost();
        return;
    }
    int32_t mc = -1;
    float mn = 3.4e38f;
    team_maxi_minf(
        t, sc, sm, g.n, -1, 3.4e38f, [=](int64_t e) { return g.col[e]; },
        [=](int64_t e) { return g.row[e] != g.col[e] ? g.cost[e] : 3.4e38f; }, mc, mn);
    g.cols = g.ecols = mc + 1;
    g.rows = uread(&g.row[g.n - 1]) + 1;
    g.cmin = mn;
}

// whether no two neighbours of the sorted edge list share both ends, and no
// edge is a self-loop (which stands twice in its vertex's list of neighbours)
template <class Team>
__device__ bool graph_is_simple(const Team &t, Scratch &sc, char *sm, const Graph &g)
{
    const int32_t *row = g.row, *col = g.col;
    return team_sum<Team, int64_t>(t, sc, sm, g.n, [=](int64_t e) -> int64_t {
               return row[e] == col[e] || (e > 0 && row[e] == row[e - 1] && col[e] == col[e - 1]);
           }) == 0;
}

__device__ __forceinline__ uint64_t pack_key(int32_t a, int32_t b, int nbits)
{
    return ((uint64_t)(uint32_t)a << nbits) | (uint32_t)b;
}

// ---------------------------------------------------------------------------
// Edges ordered by (lo, hi, edge index), for the initial sort and for every
// contraction.
//
// An edge travels as one 16-byte record (hi, edge index, cost bits, lo): the
// slot pass maps the endpoints and takes a slot in bucket lo by an atomic, a
// scan gives the bucket starts, and one 128-bit store per edge scatters the
// record.  Buckets of up to BUCKET_SMALL records stay unordered: the tile pass
// that reads them next orders them in shared memory.  Longer ones are sorted
// where they lie (a warp each up to 256, a CTA up to BUCKET_MAX), those beyond
// BUCKET_MAX by a stable radix sort of (lo, hi) over their edges in input
// order.  Bound by the scatter (a 32-byte sector per 16-byte record) and by
// the latency of the gathers and atomics of the slot pass.
//
// The form before this one scattered key, payload and bucket to three arrays,
// ranked every edge against its bucket in global memory, wrote three sorted
// arrays and read them twice more for the run heads and once for the sums:
// 15.9 ms for the initial sort and the seven contractions of the 24.8 M
// edge volume, against 10.6 this way.
// ---------------------------------------------------------------------------
template <class Rec>
struct RecordArray {
    Rec *rec;
    int32_t *start;  // nbk + 1
};

struct Records : RecordArray<int4> {  // n: x = hi, y = edge, z = cost bits, w = lo
    int2 *lohi;      // n: ends in edge order (free after the sort)
    int32_t *slot;   // n: (free after the sort)
};

// a record's key within its bucket, its bucket, and a record that is in none
__device__ __forceinline__ uint64_t rec_key(const int4 &r) { return ((uint64_t)(uint32_t)r.x << 32) | (uint32_t)r.y; }
__device__ __forceinline__ uint32_t rec_key(const int2 &r) { return (uint32_t)r.x; }
__device__ __forceinline__ int32_t rec_bucket(const int4 &r) { return r.w; }
__device__ __forceinline__ int32_t rec_bucket(const int2 &r) { return r.y; }
__device__ __forceinline__ void rec_none(int4 &r) { r = make_int4(-1, -1, 0, -1); }
__device__ __forceinline__ void rec_none(int2 &r) { r = make_int2(-1, -1); }

// Orders the listed buckets of records where they lie: 65..256 records by a
// warp, up to BUCKET_MAX by a CTA.  Ends in a team sync if there are any.
template <class Team>
__device__ __forceinline__ void team_sort_long_records(const Team &t, char *sm, const Records &R, BucketLists L)
{
    if (!L.has_long()) return;
    const int NW = blockDim.x >> 5;
    {
        uint64_t *wk = reinterpret_cast<uint64_t *>(sm) + warp_in_block() * 256;
        int32_t *wi = reinterpret_cast<int32_t *>(sm + NW * 256 * 8) + warp_in_block() * 256;
        const int32_t nw = uread(&L.n[0]);
        for (int64_t q = team_warp(t); q < nw; q += team_nwarps(t)) {
            const int32_t b = L.warp[q], s = R.start[b], m = R.start[b + 1] - s;
            int P = 128;
            while (P < m) P <<= 1;
            for (int x = lane_id(); x < m; x += 32) {
                const int4 r = R.rec[s + x];
                wk[x] = rec_key(r);
                wi[x] = r.z;
            }
            __syncwarp();
            smem_bitonic(wk, wi, m, P, lane_id(), 32, [] { __syncwarp(); });
            for (int x = lane_id(); x < m; x += 32)
                R.rec[s + x] = make_int4((int32_t)(wk[x] >> 32), (int32_t)(uint32_t)wk[x], wi[x], b);
            __syncwarp();
        }
    }
    __syncthreads();
    {
        uint64_t *ck = reinterpret_cast<uint64_t *>(sm);
        int32_t *ci = reinterpret_cast<int32_t *>(sm + BUCKET_MAX * 8);
        const int32_t nc = uread(&L.n[1]);
        for (int64_t q = t.block(); q < nc; q += t.nblocks()) {
            const int32_t b = L.cta[q], s = R.start[b], m = R.start[b + 1] - s;
            int P = 512;
            while (P < m) P <<= 1;
            for (int x = threadIdx.x; x < m; x += blockDim.x) {
                const int4 r = R.rec[s + x];
                ck[x] = rec_key(r);
                ci[x] = r.z;
            }
            __syncthreads();
            smem_bitonic(ck, ci, m, P, threadIdx.x, blockDim.x, [] { __syncthreads(); });
            for (int x = threadIdx.x; x < m; x += blockDim.x)
                R.rec[s + x] = make_int4((int32_t)(ck[x] >> 32), (int32_t)(uint32_t)ck[x], ci[x], b);
            __syncthreads();
        }
    }
    t.sync();
}

// ends(e): (lo, hi) of edge e, loads only; nbh: bits of a node id; PHASES: the
// steps are timed as the contraction's (the initial sort is one phase)
template <bool PHASES, class Team, class Ends>
__device__ __forceinline__ bool team_sort_records(const Team &t, Scratch &sc, char *sm, int64_t n, int32_t nbk,
                                                  int nbh, const float *cost, Ends ends, Records &R)
{
    R.rec = sc.arena.take<int4>(n + 1);
    R.start = sc.arena.take<int32_t>((int64_t)nbk + 2);
    R.lohi = sc.arena.take<int2>(n + 1);
    R.slot = sc.arena.take<int32_t>(n + 1);
    BucketLists L = bucket_lists(sc, n);
    if (!sc.arena.ok()) return false;
    int4 *rec = R.rec;
    int32_t *start = R.start, *slot = R.slot;
    int2 *lohi = R.lohi;
    for (int64_t b = t.rank(); b <= nbk; b += t.size()) start[b] = 0;
    if (t.rank() < 4) L.n[t.rank()] = 0;
    t.sync();
    {
        // SORT_BATCH strides of a warp at a time: the ends, then the atomics,
        // then the stores
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        int64_t base = (int64_t)t.rank() - lane_id();
        for (; base + (U - 1) * S + 31 < n; base += S * U) {
            int2 w[U];
            int32_t b[U], s[U];
#pragma unroll
            for (int k = 0; k < U; ++k) w[k] = ends(base + k * S + lane_id());
#pragma unroll
            for (int k = 0; k < U; ++k) b[k] = w[k].x;
            bucket_slots<U>(start, b, s);
#pragma unroll
            for (int k = 0; k < U; ++k) {
                lohi[base + k * S + lane_id()] = w[k];
                slot[base + k * S + lane_id()] = s[k];
            }
        }
        for (; base < n; base += S) {
            const int64_t e = base + lane_id();
            const int2 w = e < n ? ends(e) : make_int2(-1, -1);
            const int32_t s = bucket_slot(start, w.x);
            if (e < n) {
                lohi[e] = w;
                slot[e] = s;
            }
        }
    }
    t.sync();
    if (PHASES) prof_mark(t, sc, PH_CSORT_SLOT);
    team_bucket_starts(t, sc, sm, nbk, start, L, [](int64_t, int32_t, int32_t) {});
    struct Item {
        int4 r;
        int32_t p;
    };
    team_for_batched(
        t, n,
        [=](int64_t e) {
            const int2 w = lohi[e];
            Item x;
            x.r = make_int4(w.y, (int32_t)e, __float_as_int(cost[e]), w.x);
            x.p = start[w.x] + slot[e];
            return x;
        },
        [=](int64_t, Item x) { rec[x.p] = x.r; });
    t.sync();
    if (PHASES) prof_mark(t, sc, PH_CSORT_SCATTER);
    team_sort_long_records(t, sm, R, L);
    if (PHASES) prof_mark(t, sc, PH_CSORT_RANK);
    if (L.has_big()) {
        // the buckets beyond BUCKET_MAX: their edges in input order, a stable
        // radix sort of (lo, hi), then each into its bucket's range
        auto is_big = [=](int64_t e) {
            const int32_t b = lohi[e].x;
            return start[b + 1] - start[b] > BUCKET_MAX;
        };
        uint64_t bm = sc.arena.mark();
        const int64_t nbig = team_sum<Team, int64_t>(t, sc, sm, n, [=](int64_t e) -> int64_t { return is_big(e) ? 1 : 0; });
        uint64_t *bk1 = sc.arena.take<uint64_t>(nbig + 1), *bk2 = sc.arena.take<uint64_t>(nbig + 1);
        int32_t *bv1 = sc.arena.take<int32_t>(nbig + 1), *bv2 = sc.arena.take<int32_t>(nbig + 1);
        int32_t *kfirst = sc.arena.take<int32_t>((int64_t)nbk + 1);
        if (!sc.arena.ok()) return false;
        team_compact(t, sc, sm, n, is_big, [=](int64_t e, int64_t k) {
            const int2 w = lohi[e];
            bk1[k] = ((uint64_t)(uint32_t)w.x << nbh) | (uint32_t)w.y;
            bv1[k] = (int32_t)e;
        });
        team_sort_pairs(t, sc, sm, bk1, bv1, bk2, bv2, nbig, 2 * nbh);
        for (int64_t k = t.rank(); k < nbig; k += t.size()) {
            const int32_t b = (int32_t)(bk1[k] >> nbh);
            if (k == 0 || (int32_t)(bk1[k - 1] >> nbh) != b) kfirst[b] = (int32_t)k;
        }
        t.sync();
        const uint64_t mask = (uint64_t(1) << nbh) - 1;
        for (int64_t k = t.rank(); k < nbig; k += t.size()) {
            const int32_t b = (int32_t)(bk1[k] >> nbh), e = bv1[k];
            rec[start[b] + (k - kfirst[b])] = make_int4((int32_t)(bk1[k] & mask), e, __float_as_int(cost[e]), b);
        }
        t.sync();
        sc.arena.release(bm);
        if (PHASES) prof_mark(t, sc, PH_CSORT_BIG);
    }
    return true;
}

// Walks the ordered records of this CTA's share in tiles held in shared
// memory.  A tile is a window of kk * blockDim records less BUCKET_SMALL, kk = 4
// for large lists and 1 or 2 where that many tiles still find a CTA each: the
// CTA that holds a small bucket's first record has all of it in its window,
// and orders it there (every record goes to the number of smaller keys in its
// bucket; the records pass through registers).  Records of longer buckets are
// in order already and belong to the tile that holds them.
//
// visit(T, base, prev, mine) is called by every thread of the CTA once per
// tile, for its records win[base + 32 k] (k < 4; position order over (k, lane)
// within a warp's 32 kk; those from kk on are nobody's): prev[k] is the record before, mine[k] whether the
// position belongs to this CTA.  Two windows in turn, so that a tile's records
// are read while slower warps still visit the last one's.
template <class Rec>
struct RecTile {
    const Rec *win;  // the window, win[0] at position p0
    int64_t p0;
    int64_t begin;    // this CTA's records of the tile: [begin, end)
    int64_t end;
};

// first position at or after p that no earlier tile owns
template <class Rec>
__device__ __forceinline__ int64_t rec_owned_from(const RecordArray<Rec> &R, int64_t p, int64_t n)
{
    if (p >= n) return n;
    const int32_t lo = rec_bucket(R.rec[p]);
    const int32_t s = R.start[lo], e = R.start[lo + 1];
    return e - s > BUCKET_SMALL || s == p ? p : e;
}

//
// TIES: records of a bucket may have equal keys (they keep their order).
template <bool TIES = false, class Team, class Rec, class Visit>
__device__ __forceinline__ void team_record_tiles(const Team &t, char *sm, const RecordArray<Rec> &R, int64_t n,
                                                  Visit visit)
{
    constexpr int K = 4;
    // records a thread of this walk
    const int kk = n <= t.nblocks() * (int64_t)(blockDim.x - BUCKET_SMALL)       ? 1
                   : n <= t.nblocks() * (int64_t)(2 * blockDim.x - BUCKET_SMALL) ? 2
                                                                                 : K;
    const int W = kk * blockDim.x, TILE = W - BUCKET_SMALL;
    const int64_t ntiles = (n + TILE - 1) / TILE;
    const int64_t per = (ntiles + t.nblocks() - 1) / t.nblocks();
    const int64_t t0 = (int64_t)t.block() * per;
    const int64_t t1 = t0 + per < ntiles ? t0 + per : ntiles;
    const int base = warp_in_block() * 32 * kk + lane_id();
    int64_t a = t0 < t1 ? rec_owned_from(R, t0 * TILE, n) : n;
    int flip = 0;
    for (int64_t tile = t0; tile < t1; ++tile, flip ^= 1) {
        Rec *win = reinterpret_cast<Rec *>(sm) + flip * W;
        const int64_t p0 = tile * TILE;
        const int64_t b = rec_owned_from(R, p0 + TILE, n);
        Rec r[K];
        int32_t s[K], e[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int64_t p = p0 + base + 32 * k;
            r[k] = R.rec[p < n ? p : n - 1];
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            s[k] = R.start[rec_bucket(r[k])];
            e[k] = R.start[rec_bucket(r[k]) + 1];
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (k < kk) win[base + 32 * k] = r[k];
        // the next tile's records on their way to L2 (a line per 128 bytes)
        if (tile + 1 < t1 && lane_id() % (128 / (int)sizeof(Rec)) == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int64_t p = p0 + TILE + base + 32 * k;
                if (k < kk && p < n) asm volatile("prefetch.L2 [%0];" ::"l"(R.rec + p));
            }
        }
        __syncthreads();
        int dst[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = base + 32 * k;
            const int64_t p = p0 + i;
            dst[k] = i;
            if (k < kk && p >= a && p < b && e[k] - s[k] <= BUCKET_SMALL) {
                const auto key = rec_key(r[k]);
                const int f = (int)(s[k] - p0), l = (int)(e[k] - p0);
                int rank = 0;
                for (int x = f; x < l; ++x) {
                    const auto o = rec_key(win[x]);
                    rank += o < key || (TIES && o == key && x < i);
                }
                dst[k] = f + rank;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int64_t p = p0 + base + 32 * k;
            if (k < kk && p >= a && p < b) win[dst[k]] = r[k];
        }
        __syncthreads();
        RecTile<Rec> T;
        T.win = win;
        T.p0 = p0;
        T.begin = a;
        T.end = b;
        Rec none, prev[K];
        rec_none(none);
        bool mine[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = base + 32 * k;
            const int64_t p = p0 + i;
            mine[k] = k < kk && p >= a && p < b;
            prev[k] = !mine[k] ? none : (p > a ? win[i - 1] : (p > 0 ? R.rec[p - 1] : none));
        }
        visit(T, base, prev, mine);
        a = b;
    }
    __syncthreads();  // the windows are free again
}

// shared memory of two windows of a CTA of `threads` threads
__host__ __device__ constexpr int record_smem_bytes(int threads) { return 2 * 4 * threads * 16; }

// the graph slot at the top of the arena, for n edges (team-uniform; fails
// when it would overlap live temporaries)
__device__ __forceinline__ bool graph_slot(Scratch &sc, int64_t n, Graph &g, uint64_t &top)
{
    Arena &ar = sc.arena;
    const uint64_t bytes = (uint64_t)(n + 1) * 12 + 3 * 256;
    top = (ar.cap - bytes) & ~uint64_t(255);
    if (ar.failed || bytes > ar.cap || top < ar.lo) {
        ar.failed = 1;
        return false;
    }
    const uint64_t words = ((uint64_t)(n + 1) * 4 + 255) / 256 * 256;
    g.row = reinterpret_cast<int32_t *>(ar.base + top);
    g.col = reinterpret_cast<int32_t *>(ar.base + top + words);
    g.cost = reinterpret_cast<float *>(ar.base + top + 2 * words);
    return true;
}

// dCOO ctor with unsorted input (src/dCOO.cu:38-45): endpoints ordered,
// sorted by (row,col), stable.  Inputs are (i, j, c) of length n.  The sorted
// edges go straight from the tile pass into the graph slot; edge lists of
// 2^31 or more take graph_from_edges_sorted (one radix sort of every edge's
// keys).
template <class Team>
__device__ __noinline__ Graph graph_from_edges_sorted(const Team &t, Scratch &sc, char *, const int32_t *i, const int32_t *j,
                                         const float *c, int64_t n);

template <class Team>
__device__ __noinline__ Graph graph_from_edges(const Team &t, Scratch &sc, char *, const int32_t *i, const int32_t *j,
                                  const float *c, int64_t n)
{
    char *sm = team_smem();
    if (n == 0 || n >= (int64_t(1) << 31)) return graph_from_edges_sorted(t, sc, sm, i, j, c, n);
    Graph g;
    g.n = n;
    g.rows = g.cols = g.ecols = 0;
    g.uniq = 0;
    g.cmin = unknown_cost();
    const int32_t mx = team_max<Team, int32_t>(t, sc, sm, n, 0, [=](int64_t e) { return i[e] > j[e] ? i[e] : j[e]; });
    const int nbh = bits_for((uint64_t)(mx > 0 ? mx : 1));
    uint64_t m = sc.arena.mark();
    Records R;
    if (!team_sort_records<false>(
            t, sc, sm, n, mx + 1, nbh, c,
            [=](int64_t e) {
                const int32_t a = i[e], b = j[e];
                return a < b ? make_int2(a, b) : make_int2(b, a);
            },
            R))
        return g;
    uint64_t top;
    if (!graph_slot(sc, n, g, top)) return g;
    int32_t dup = 0;
    float mn = 3.4e38f;
    team_record_tiles(t, sm, R, n, [&](const RecTile<int4> &T, int base, const int4 (&prev)[4], const bool (&mine)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (mine[k]) {
                const int4 r = T.win[base + 32 * k];
                const int64_t p = T.p0 + base + 32 * k;
                g.row[p] = r.w;
                g.col[p] = r.x;
                g.cost[p] = __int_as_float(r.z);
                if (r.w != r.x) mn = fminf(mn, __int_as_float(r.z));
                dup |= prev[k].w == r.w && prev[k].x == r.x;
            }
    });
    // dims as in dCOO::init (src/dCOO.cu:47-51); the largest endpoint is a
    // column.  The last record is read before the fold's team sync: the caller
    // hands its memory on with no sync of its own (the tile pass leaves the
    // records of R as they are).
    g.cols = g.ecols = mx + 1;
    g.rows = uread(&R.rec[n - 1].w) + 1;
    team_fold_maxi_minf(t, sc, sm, dup, mn);
    g.cmin = mn;
    g.uniq = dup == 0;
    sc.arena.top = top;
    sc.arena.release(m);
    sc.alg_bytes += 24.0 * (double)n;
    return g;
}

template <class Team>
__device__ __noinline__ Graph graph_from_edges_sorted(const Team &t, Scratch &sc, char *, const int32_t *i, const int32_t *j,
                                         const float *c, int64_t n)
{
    char *sm = team_smem();
    Graph out;
    out.n = n;
    out.rows = out.cols = out.ecols = 0;
    out.uniq = 0;
    int32_t mx = team_max<Team, int32_t>(t, sc, sm, n, 0, [=](int64_t e) { return i[e] > j[e] ? i[e] : j[e]; });
    const int nb = bits_for((uint64_t)mx);
    uint64_t m = sc.arena.mark();
    uint64_t *k1 = sc.arena.take<uint64_t>(n + 1), *k2 = sc.arena.take<uint64_t>(n + 1);
    float *v1 = sc.arena.take<float>(n + 1), *v2 = sc.arena.take<float>(n + 1);
    Graph g = graph_alloc(t, sc, n);
    if (!sc.arena.ok()) return out;
    for (int64_t e = t.rank(); e < n; e += t.size()) {
        int32_t a = i[e], b = j[e];
        k1[e] = pack_key(a < b ? a : b, a < b ? b : a, nb);
        v1[e] = c[e];
    }
    t.sync();
    team_sort_pairs(t, sc, sm, k1, v1, k2, v2, n, 2 * nb);
    const uint64_t mask = (nb == 0) ? 0 : ((uint64_t(1) << nb) - 1);
    for (int64_t e = t.rank(); e < n; e += t.size()) {
        g.row[e] = (int32_t)(k1[e] >> nb);
        g.col[e] = (int32_t)(k1[e] & mask);
        g.cost[e] = v1[e];
    }
    t.sync();
    graph_set_dims(t, sc, sm, g);
    Graph r = graph_commit(t, sc, g);
    sc.arena.release(m);
    sc.alg_bytes += 24.0 * (double)n;
    return r;
}

// dCOO::contract_cuda (src/dCOO.cu:57-95) followed by has_bad_contractions
// (src/rama_cuda.cu:18-30) and remove_diagonal (src/dCOO.cu:106-116).
// Parallel edges are summed in sorted (stable) order with RSUM.
// Returns the new graph (committed to the top slot); *bad is set if a
// self-loop of negative cost appeared.  Dims are taken before the diagonal
// is removed, as the reference does.
// The edges keyed by their contracted endpoints, sorted: k1[p] = (lo, hi)
// packed with nb bits each, v1[p] = the edge's cost, in (lo, hi) order and,
// for equal keys, in edge order (the order a stable sort leaves; it fixes the
// summation order of parallel edges).  The edges are bucketed by their new
// row lo and each row is ordered by (hi, edge index); rows of more than
// BUCKET_MAX edges send the whole list through the LSD radix sort instead.
// k1/v1 (and the spare k2/v2) hold n + 1 entries; the result ends in k1/v1.
template <class Team>
__device__ __noinline__ void contract_sorted_keys(const Team &t, Scratch &sc, char *, const Graph &A, const int32_t *map,
                                     int32_t map_max, int nb, uint64_t *&k1, float *&v1, uint64_t *&k2, float *&v2)
{
    char *sm = team_smem();
    const int64_t n = A.n;
    bool done = false;
    uint64_t m = sc.arena.mark();
    int32_t *bst = sc.arena.take<int32_t>((int64_t)map_max + 2);
    int32_t *bidx = sc.arena.take<int32_t>(n + 1);
    if (sc.arena.ok() && n < (int64_t(1) << 31)) {
        done = team_bucket_sort(
            t, sc, sm, n, map_max + 1,
            [=](int64_t e) {
                const int32_t a = map[A.row[e]], b = map[A.col[e]];
                return a < b ? a : b;
            },
            [=](int64_t e) -> uint64_t {
                const int32_t a = map[A.row[e]], b = map[A.col[e]];
                return ((uint64_t)(uint32_t)(a < b ? b : a) << 32) | (uint64_t)e;
            },
            k2, bidx, bst);
        if (done) {
            for (int64_t b = t.rank(); b <= map_max; b += t.size())
                for (int32_t p = bst[b]; p < bst[b + 1]; ++p) k1[p] = pack_key((int32_t)b, (int32_t)(k2[p] >> 32), nb);
            for (int64_t p = t.rank(); p < n; p += t.size()) v1[p] = A.cost[bidx[p]];
            t.sync();
        }
    }
    sc.arena.release(m);
    if (done) return;
    for (int64_t e = t.rank(); e < n; e += t.size()) {
        int32_t a = map[A.row[e]], b = map[A.col[e]];
        k1[e] = pack_key(a < b ? a : b, a < b ? b : a, nb);
        v1[e] = A.cost[e];
    }
    t.sync();
    team_sort_pairs(t, sc, sm, k1, v1, k2, v2, n, 2 * nb);
}

template <class Team>
__device__ __noinline__ Graph graph_contract_sorted(const Team &t, Scratch &sc, char *, const Graph &A, const int32_t *map,
                                       int32_t map_max, int *bad)
{
    char *sm = team_smem();
    const int64_t n = A.n;
    const int nb = bits_for((uint64_t)(map_max > 0 ? map_max : 0));
    uint64_t m = sc.arena.mark();
    uint64_t *k1 = sc.arena.take<uint64_t>(n + 1), *k2 = sc.arena.take<uint64_t>(n + 1);
    float *v1 = sc.arena.take<float>(n + 1), *v2 = sc.arena.take<float>(n + 1);
    int64_t *runpos = sc.arena.take<int64_t>(n + 2);
    int32_t *badflag = sc.arena.take<int32_t>(2);
    Graph out = A;
    if (!sc.arena.ok()) return out;
    if (t.rank() == 0) badflag[0] = 0;
    contract_sorted_keys(t, sc, sm, A, map, map_max, nb, k1, v1, k2, v2);
    // run heads -> run index
    const int64_t nruns = team_compact(
        t, sc, sm, n, [=](int64_t k) { return k == 0 || k1[k] != k1[k - 1]; },
        [=](int64_t k, int64_t r) { runpos[r] = k; });
    if (t.rank() == 0) runpos[nruns] = n;
    t.sync();
    Graph g = graph_alloc(t, sc, nruns);
    int32_t *longq = sc.arena.take<int32_t>(nruns + 1);
    int32_t *nlong = sc.arena.take<int32_t>(2);
    if (!sc.arena.ok()) return out;
    const uint64_t mask = (nb == 0) ? 0 : ((uint64_t(1) << nb) - 1);
    if (t.rank() == 0) nlong[0] = 0;
    t.sync();
    for (int64_t r = t.rank(); r < nruns; r += t.size()) {
        int64_t s = runpos[r], e = runpos[r + 1];
        uint64_t key = k1[s];
        g.row[r] = (int32_t)(key >> nb);
        g.col[r] = (int32_t)(key & mask);
        if (e - s <= 32) {
            g.cost[r] = rsum_serial((int)(e - s), [=](int k) { return v1[s + k]; });
        } else {
            int q = atomicAdd(nlong, 1);
            longq[q] = (int32_t)r;
        }
    }
    t.sync();
    const int32_t nl = uread(nlong);
    for (int64_t q = team_warp(t); q < nl; q += team_nwarps(t)) {
        int64_t r = longq[q];
        int64_t s = runpos[r], e = runpos[r + 1];
        float v = rsum_warp(e - s, [=](int64_t k) { return v1[s + k]; });
        if (lane_id() == 0) g.cost[r] = v;
    }
    t.sync();
    g.n = nruns;
    graph_set_dims(t, sc, sm, g);
    // bad contractions + stable removal of the diagonal
    for (int64_t r = t.rank(); r < nruns; r += t.size())
        if (g.row[r] == g.col[r] && g.cost[r] < 0.0f) badflag[0] = 1;
    Graph h = graph_alloc(t, sc, nruns);
    if (!sc.arena.ok()) return out;
    const int64_t nk = team_compact(
        t, sc, sm, nruns, [=](int64_t r) { return g.row[r] != g.col[r]; },
        [=](int64_t r, int64_t p) {
            h.row[p] = g.row[r];
            h.col[p] = g.col[r];
            h.cost[p] = g.cost[r];
        });
    *bad = uread(badflag);
    h.n = nk;
    h.rows = g.rows;
    h.cols = g.cols;
    h.cmin = g.cmin;
    h.ecols = 0;
    if (nk > 0) h.ecols = 1 + team_max<Team, int32_t>(t, sc, sm, nk, -1, [=](int64_t e) { return h.col[e]; });
    h.uniq = 1;
    Graph res = graph_commit(t, sc, h);
    sc.arena.release(m);
    sc.alg_bytes += 20.0 * (double)n + 12.0 * (double)nruns;
    return res;
}

// The contraction (dCOO::contract_cuda + has_bad_contractions +
// remove_diagonal) by buckets of the new row:
//   1. the edges are ordered by their contracted ends (team_sort_records);
//   2. a tile pass finds the heads of the runs of equal (lo, hi); a head's
//      thread sums its run in edge order (RSUM) out of the tile and appends
//      the edge to its CTA's part of the output, or checks a self-loop's sum
//      for a bad contraction; runs of more than 32 records of long buckets go
//      to warps afterwards, runs of more than RSUM_CHUNK by chunks to many;
//   3. the CTAs' parts are joined in the graph slot at the top of the arena
//      (the old graph there is dead by then), with the largest column and the
//      smallest cost on the way; a single CTA writes there directly.  The
//      rows are the last bucket + 1 (dims are taken before the diagonal goes,
//      as the reference does).
// graph_contract_sorted (one radix sort of every edge's packed keys) remains
// for edge lists of 2^31 edges or more.  Both give the same graph bit for bit.
template <class Team>
__device__ __noinline__ Graph graph_contract(const Team &t, Scratch &sc, char *, const Graph &graph,
                                             const int32_t *map, int32_t map_max, int *bad)
{
    char *sm = team_smem();
    const Graph A = graph;  // its pointers in registers
    const int64_t n = A.n;
    Graph out = A;
    if (n == 0 || n >= (int64_t(1) << 31)) return graph_contract_sorted(t, sc, sm, A, map, map_max, bad);
    const int nbh = bits_for((uint64_t)(map_max > 0 ? map_max : 1));
    uint64_t m = sc.arena.mark();
    // [0] bad, [1] long runs, [2] largest self-loop column
    int32_t *fl = sc.arena.take<int32_t>(8);
    int4 *longq = sc.arena.take<int4>(n / 33 + 2);  // long runs: first and last position, output (-1: self-loop)
    if (!sc.arena.ok()) return out;
    if (t.rank() == 0) {
        fl[0] = 0;
        fl[1] = 0;
        fl[2] = -1;
    }
    Records R;
    if (!team_sort_records<true>(
            t, sc, sm, n, map_max + 1, nbh, A.cost,
            [=](int64_t e) {
                const int32_t a = map[A.row[e]], b = map[A.col[e]];
                return a < b ? make_int2(a, b) : make_int2(b, a);
            },
            R))
        return out;
    // the new graph's slot, sized for at most n edges; it ends at the arena's
    // end, so it lies within the old graph's slot (n is the old edge count)
    Graph h;
    uint64_t top;
    if (!graph_slot(sc, n, h, top)) return out;
    // temporaries taken from here on stay below the new slot (when the old
    // graph does not live in the slot, as in a single step, the arena's top
    // is its end)
    if (top < sc.arena.top) sc.arena.top = top;
    // where a CTA's edges go first: its own records' positions in two arrays
    // that the sort no longer needs, or the slot itself
    const bool direct = t.nblocks() == 1;
    int2 *tends = R.lohi;
    float *tcost = reinterpret_cast<float *>(R.slot);
    __shared__ int32_t wtot[2][32];
    int64_t first = -1;  // this CTA's first record
    int64_t kept = 0;    // edges it has written
    int parity = 0;
    int32_t dloc = -1;  // largest self-loop column
    auto finish = [=](int64_t k, float sum) {
        if (k >= 0) {
            if (direct)
                h.cost[k] = sum;
            else
                tcost[k] = sum;
        } else if (sum < 0.0f) {
            fl[0] = 1;
        }
    };
    // RSUM of a run of n records in the tile.  Most edges are merged with no
    // other (of the 24.8 M edge volume's, 92 % in the first contraction): one value is its
    // own sum (+0.0 for -0.0), and two floats added in 64 bits and rounded are
    // their 32-bit sum.
    auto run_sum = [](const int4 *v, int n) {
        const float a = __fadd_rn(0.0f, __int_as_float(v[0].z));
        if (n == 1) return a;
        if (n == 2) return __fadd_rn(a, __int_as_float(v[1].z));
        return rsum_upto64(n, [=](int q) { return __int_as_float(v[q].z); });
    };
    team_record_tiles(t, sm, R, n, [&](const RecTile<int4> &T, int base, const int4 (&prev)[4], const bool (&mine)[4]) {
        int4 r[4];
        bool head[4];
        unsigned keep[4];
        int wsum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r[k] = T.win[base + 32 * k];
            head[k] = mine[k] && (prev[k].w != r[k].w || prev[k].x != r[k].x);
            keep[k] = __ballot_sync(FULL, head[k] && r[k].w != r[k].x);
            wsum += __popc(keep[k]);
        }
        if (lane_id() == 0) wtot[parity][warp_in_block()] = wsum;
        __syncthreads();
        const int nw = blockDim.x >> 5;
        const int wt = lane_id() < nw ? wtot[parity][lane_id()] : 0;
        const int incl = warp_incl_scan(wt);
        parity ^= 1;
        if (first < 0) first = T.begin;  // (its edges are no more than its records)
        int64_t k0 = (direct ? 0 : first) + kept +
                     (warp_in_block() > 0 ? __shfl_sync(FULL, incl, warp_in_block() - 1) : 0);
        kept += __shfl_sync(FULL, incl, 31);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t mk = k0 + __popc(keep[k] & lanemask_lt());
            k0 += __popc(keep[k]);
            if (!head[k]) continue;
            const bool loop = r[k].w == r[k].x;
            const int64_t o = loop ? -1 : mk;
            if (loop) {
                dloc = max(dloc, r[k].x);
            } else if (direct) {
                h.row[o] = r[k].w;
                h.col[o] = r[k].x;
            } else {
                tends[o] = make_int2(r[k].w, r[k].x);
            }
            // the run's end: within the tile, or anywhere in a long bucket
            const int i = base + 32 * k;
            const int lim = (int)(T.end - T.p0 < i + 33 ? T.end - T.p0 : i + 33);
            int x = i + 1;
            while (x < lim && T.win[x].x == r[k].x && T.win[x].w == r[k].w) ++x;
            if (x == lim) {
                const int32_t s = R.start[r[k].w], e = R.start[r[k].w + 1];
                if (e - s > BUCKET_SMALL) {
                    // first record of the bucket with a larger hi
                    int64_t lo = T.p0 + x, hi = e;
                    while (lo < hi) {
                        const int64_t mid = (lo + hi) >> 1;
                        if (R.rec[mid].x <= r[k].x)
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                    const int64_t p = T.p0 + i;
                    if (lo - p > 32)
                        longq[atomicAdd(&fl[1], 1)] = make_int4((int32_t)p, (int32_t)lo, (int32_t)o, 0);
                    else
                        finish(o, rsum_upto64((int)(lo - p), [=](int q) { return __int_as_float(R.rec[p + q].z); }));
                    continue;
                }
                const int l = (int)(e - T.p0);
                while (x < l && T.win[x].x == r[k].x) ++x;
            }
            finish(o, run_sum(T.win + i, x - i));
        }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dloc = max(dloc, __shfl_xor_sync(FULL, dloc, o));
    if (lane_id() == 0 && dloc >= 0) atomicMax(&fl[2], dloc);
    int64_t obase = 0, nk = kept;
    if (!direct) {
        int64_t *part = reinterpret_cast<int64_t *>(sc.next_part());
        if (threadIdx.x == 0) part[t.block()] = kept;
        t.sync();
        cta_prefix_parts(t, sc, part, obase, nk);
    } else {
        t.sync();
    }
    // runs of 33..RSUM_CHUNK edges: a warp each.  Longer runs (a cluster's
    // self-loop run can hold a large part of the graph): their chunks of
    // RSUM_CHUNK edges are shared out over every warp of the team, then a warp
    // per run sums its chunk sums -- the same sum as rsum_warp.
    const int32_t nl = uread(&fl[1]);
    if (nl > 0) {
        const int4 *rec = R.rec;
        int32_t *coff = sc.arena.take<int32_t>((int64_t)nl + 1);
        if (!sc.arena.ok()) return out;
        const int64_t nchunks = team_scan<Team, int64_t>(
            t, sc, sm, nl,
            [=](int64_t q) -> int64_t {
                const int64_t len = longq[q].y - longq[q].x;
                return len > RSUM_CHUNK ? (len + RSUM_CHUNK - 1) / RSUM_CHUNK : 0;
            },
            [=](int64_t q, int64_t pre, int64_t) { coff[q] = (int32_t)pre; });
        double *chunk_sum = sc.arena.take<double>(nchunks + 1);
        if (!sc.arena.ok()) return out;
        for (int64_t w = team_warp(t); w < nl + nchunks; w += team_nwarps(t)) {
            if (w < nl) {
                const int4 L = longq[w];
                if (L.y - L.x <= RSUM_CHUNK) {
                    const float v =
                        (float)rsum_chunk_warp(L.y - L.x, [=](int64_t x) { return __int_as_float(rec[L.x + x].z); });
                    if (lane_id() == 0) finish(L.z, v);
                }
            } else {
                // chunk g belongs to the last run q with coff[q] <= g
                const int64_t g = w - nl;
                int32_t lo = 0, hi = nl - 1;
                while (lo < hi) {
                    const int32_t mid = (lo + hi + 1) >> 1;
                    if (coff[mid] <= g)
                        lo = mid;
                    else
                        hi = mid - 1;
                }
                const int4 L = longq[lo];
                const int64_t cb = L.x + (g - coff[lo]) * RSUM_CHUNK;
                const int64_t len = L.y - cb < RSUM_CHUNK ? L.y - cb : RSUM_CHUNK;
                const double d = rsum_chunk_warp(len, [=](int64_t x) { return __int_as_float(rec[cb + x].z); });
                if (lane_id() == 0) chunk_sum[g] = d;
            }
        }
        t.sync();
        if (nchunks > 0) {
            for (int64_t w = team_warp(t); w < nl; w += team_nwarps(t)) {
                const int4 L = longq[w];
                const int64_t len = L.y - L.x;
                if (len <= RSUM_CHUNK) continue;
                const int64_t c0 = coff[w], nc = (len + RSUM_CHUNK - 1) / RSUM_CHUNK;
                double acc = 0.0;  // lane l: chunks l, l + 32, ... in order
                for (int64_t c = lane_id(); c < nc; c += 32) acc = __dadd_rn(acc, chunk_sum[c0 + c]);
                const float v = (float)rsum_lane_tree(acc);
                if (lane_id() == 0) finish(L.z, v);
            }
            t.sync();
        }
    }
    *bad = uread(&fl[0]);
    const int32_t dmax = uread(&fl[2]);
    // 3. the edges to their places; dims and the smallest cost (every new
    //    edge has row < col)
    int32_t mc = -1;
    float mn = 3.4e38f;
    if (direct) {
        for (int64_t k = t.rank(); k < nk; k += t.size()) {
            mc = max(mc, h.col[k]);
            mn = fminf(mn, h.cost[k]);
        }
    } else {
        constexpr int U = 4;
        const int S = blockDim.x;
        int64_t k = threadIdx.x;
        auto put = [&](int64_t q, int2 w, float c) {
            h.row[obase + q] = w.x;
            h.col[obase + q] = w.y;
            h.cost[obase + q] = c;
            mc = max(mc, w.y);
            mn = fminf(mn, c);
        };
        for (; k + (U - 1) * S < kept; k += U * S) {
            int2 w[U];
            float c[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                w[q] = tends[first + k + q * S];
                c[q] = tcost[first + k + q * S];
            }
#pragma unroll
            for (int q = 0; q < U; ++q) put(k + q * S, w[q], c[q]);
        }
        for (; k < kept; k += S) put(k, tends[first + k], tcost[first + k]);
    }
    h.rows = uread(&R.rec[n - 1].w) + 1;  // before the fold's team sync, after which the records' memory is handed on
    team_fold_maxi_minf(t, sc, sm, mc, mn);
    prof_mark(t, sc, PH_CONTRACT_RUNS);
    h.n = nk;
    h.cols = (mc > dmax ? mc : dmax) + 1;
    h.cmin = nk > 0 ? mn : unknown_cost();
    h.ecols = mc + 1;
    h.uniq = 1;
    sc.arena.top = top;
    sc.arena.release(m);
    sc.alg_bytes += 20.0 * (double)n + 12.0 * (double)nk;
    return h;
}

// compute_sanitized_graph (include/rama_utils.h:429-466): drop duplicate
// edges (the first occurrence in stable (min,max) order survives), then
// renumber the nodes that have edges to 0..k-1.  Outputs live in the
// temporaries; idmap (size = max id + 1) maps original ids to new ones.
template <class Team>
__device__ __noinline__ int64_t sanitize_edges(const Team &t, Scratch &sc, char *, const int32_t *I, const int32_t *J,
                                  const float *Cc, int64_t n, int32_t *&si, int32_t *&sj, float *&sw, int32_t *&idmap,
                                  int32_t &idsize)
{
    char *sm = team_smem();
    int32_t mx = team_max<Team, int32_t>(t, sc, sm, n, 0, [=](int64_t e) { return I[e] > J[e] ? I[e] : J[e]; });
    idsize = mx + 1;
    const int nb = bits_for((uint64_t)mx);
    si = sc.arena.take<int32_t>(n + 1);
    sj = sc.arena.take<int32_t>(n + 1);
    sw = sc.arena.take<float>(n + 1);
    idmap = sc.arena.take<int32_t>((int64_t)idsize + 1);
    uint64_t m = sc.arena.mark();
    uint64_t *k1 = sc.arena.take<uint64_t>(n + 1), *k2 = sc.arena.take<uint64_t>(n + 1);
    float *v1 = sc.arena.take<float>(n + 1), *v2 = sc.arena.take<float>(n + 1);
    if (!sc.arena.ok()) return 0;
    for (int64_t e = t.rank(); e < n; e += t.size()) {
        int32_t a = I[e], b = J[e];
        k1[e] = pack_key(a < b ? a : b, a < b ? b : a, nb);
        v1[e] = Cc[e];
    }
    for (int64_t v = t.rank(); v < idsize; v += t.size()) idmap[v] = 0;
    t.sync();
    team_sort_pairs(t, sc, sm, k1, v1, k2, v2, n, 2 * nb);
    const uint64_t mask = (nb == 0) ? 0 : ((uint64_t(1) << nb) - 1);
    const int64_t u = team_compact(
        t, sc, sm, n, [=](int64_t k) { return k == 0 || k1[k] != k1[k - 1]; },
        [=](int64_t k, int64_t p) {
            int32_t a = (int32_t)(k1[k] >> nb), b = (int32_t)(k1[k] & mask);
            si[p] = a;
            sj[p] = b;
            sw[p] = v1[k];
            idmap[a] = 1;
            idmap[b] = 1;
        });
    team_scan<Team, int64_t>(
        t, sc, sm, idsize, [=](int64_t v) -> int64_t { return idmap[v]; },
        [=](int64_t v, int64_t pre, int64_t) { idmap[v] = (int32_t)pre; });
    for (int64_t e = t.rank(); e < u; e += t.size()) {
        si[e] = idmap[si[e]];
        sj[e] = idmap[sj[e]];
    }
    t.sync();
    sc.arena.release(m);
    return u;
}

// Stable contraction WITHOUT diagonal removal (the raw contract_cuda result,
// for parity tests); result lives in the temporaries.
template <class Team>
__device__ Graph graph_contract_raw(const Team &t, Scratch &sc, char *sm, const Graph &A, const int32_t *map,
                                    int32_t map_max)
{
    const int64_t n = A.n;
    const int nb = bits_for((uint64_t)(map_max > 0 ? map_max : 0));
    uint64_t *k1 = sc.arena.take<uint64_t>(n + 1), *k2 = sc.arena.take<uint64_t>(n + 1);
    float *v1 = sc.arena.take<float>(n + 1), *v2 = sc.arena.take<float>(n + 1);
    int64_t *runpos = sc.arena.take<int64_t>(n + 2);
    Graph out = A;
    if (!sc.arena.ok()) return out;
    contract_sorted_keys(t, sc, sm, A, map, map_max, nb, k1, v1, k2, v2);
    const int64_t nruns = team_compact(
        t, sc, sm, n, [=](int64_t k) { return k == 0 || k1[k] != k1[k - 1]; },
        [=](int64_t k, int64_t r) { runpos[r] = k; });
    if (t.rank() == 0) runpos[nruns] = n;
    t.sync();
    Graph g = graph_alloc(t, sc, nruns);
    if (!sc.arena.ok()) return out;
    const uint64_t mask = (nb == 0) ? 0 : ((uint64_t(1) << nb) - 1);
    for (int64_t r = t.rank(); r < nruns; r += t.size()) {
        int64_t s = runpos[r], e = runpos[r + 1];
        uint64_t key = k1[s];
        g.row[r] = (int32_t)(key >> nb);
        g.col[r] = (int32_t)(key & mask);
        g.cost[r] = (e - s <= 32) ? rsum_serial((int)(e - s), [=](int k) { return v1[s + k]; }) : 0.0f;
    }
    t.sync();
    for (int64_t r = team_warp(t); r < nruns; r += team_nwarps(t)) {
        int64_t s = runpos[r], e = runpos[r + 1];
        if (e - s <= 32) continue;
        float v = rsum_warp(e - s, [=](int64_t k) { return v1[s + k]; });
        if (lane_id() == 0) g.cost[r] = v;
    }
    t.sync();
    g.n = nruns;
    graph_set_dims(t, sc, sm, g);
    return g;
}

// ---------------------------------------------------------------------------
// Symmetric CSR of a (row,col)-sorted directed edge list restricted to the
// edges where keep(e) holds: row v lists its neighbours u<v (increasing u)
// then w>v (increasing w) -- the (row,col) order of the doubled list
// (to_undirected + coo_sorting, include/rama_utils.h:107-131, 287-294).
// Built with one stable radix sort of the kept edges by column.
// ---------------------------------------------------------------------------
struct Csr {
    int32_t nrows;
    int32_t *off;  // nrows + 1
    int32_t *adj;  // 2m
    float *w;      // 2m
    int64_t m2;
};

template <class Team, class Keep>
__device__ __noinline__ Csr build_symmetric_csr(const Team &t, Scratch &sc, char *, const Graph &A, int32_t nrows,
                                                Keep keep)
{
    char *sm = team_smem();
    Csr C;
    C.nrows = nrows;
    C.m2 = 0;
    // 1. compact kept edges (their order stays (row,col)-sorted)
    int64_t *kidx = sc.arena.take<int64_t>(A.n + 1);
    int32_t *deg = sc.arena.take<int32_t>((int64_t)nrows + 1);
    C.off = sc.arena.take<int32_t>((int64_t)nrows + 2);
    if (!sc.arena.ok()) return C;
    for (int64_t v = t.rank(); v <= nrows; v += t.size()) deg[v] = 0;
    const int64_t m = team_compact(t, sc, sm, A.n, keep, [=](int64_t e, int64_t p) { kidx[p] = e; });
    C.m2 = 2 * m;
    C.adj = sc.arena.take<int32_t>(2 * m + 1);
    C.w = sc.arena.take<float>(2 * m + 1);
    uint64_t mk = sc.arena.mark();
    uint64_t *k1 = sc.arena.take<uint64_t>(m + 1), *k2 = sc.arena.take<uint64_t>(m + 1);
    int32_t *v1 = sc.arena.take<int32_t>(m + 1), *v2 = sc.arena.take<int32_t>(m + 1);
    int32_t *infill = sc.arena.take<int32_t>((int64_t)nrows + 1);
    int32_t *colstart = sc.arena.take<int32_t>((int64_t)nrows + 1);
    int32_t *rowstart = sc.arena.take<int32_t>((int64_t)nrows + 1);
    if (!sc.arena.ok()) return C;
    // 2. degrees (in + out) and in-degrees (number of u<v entries per row)
    for (int64_t v = t.rank(); v <= nrows; v += t.size()) infill[v] = 0;
    t.sync();
    for (int64_t p = t.rank(); p < m; p += t.size()) {
        int64_t e = kidx[p];
        atomicAdd(&deg[A.row[e]], 1);
        atomicAdd(&deg[A.col[e]], 1);
        atomicAdd(&infill[A.col[e]], 1);
        k1[p] = (uint64_t)(uint32_t)A.col[e];
        v1[p] = (int32_t)p;
    }
    t.sync();
    team_scan<Team, int64_t>(
        t, sc, sm, (int64_t)nrows, [=](int64_t v) -> int64_t { return deg[v]; },
        [=](int64_t v, int64_t pre, int64_t) { C.off[v] = (int32_t)pre; });
    // first position of each column among the column-sorted kept edges, and
    // of each row among the (row-sorted) kept edges
    team_scan<Team, int64_t>(
        t, sc, sm, (int64_t)nrows, [=](int64_t v) -> int64_t { return infill[v]; },
        [=](int64_t v, int64_t pre, int64_t) { colstart[v] = (int32_t)pre; });
    team_scan<Team, int64_t>(
        t, sc, sm, (int64_t)nrows, [=](int64_t v) -> int64_t { return deg[v] - infill[v]; },
        [=](int64_t v, int64_t pre, int64_t) { rowstart[v] = (int32_t)pre; });
    if (t.rank() == 0) C.off[nrows] = (int32_t)(2 * m);
    t.sync();
    // 3. kept edges in column order, rows increasing within a column (a
    //    bucket sort by column of the kept positions, which are in row order;
    //    columns of more than BUCKET_MAX entries: a stable radix sort) ->
    //    the reverse entries
    int32_t *bst = sc.arena.take<int32_t>((int64_t)nrows + 2);
    if (sc.arena.ok() && m < (int64_t(1) << 31) &&
        team_bucket_sort(
            t, sc, sm, m, nrows, [=](int64_t p) { return A.col[kidx[p]]; }, [=](int64_t p) { return (uint64_t)p; },
            k2, v2, bst)) {
        for (int64_t q = t.rank(); q < m; q += t.size()) {
            const int64_t p = (int64_t)k2[q];
            const int64_t e = kidx[p];
            const int32_t c = A.col[e];
            const int64_t dst = (int64_t)C.off[c] + (q - bst[c]);
            C.adj[dst] = A.row[e];
            C.w[dst] = A.cost[e];
        }
    } else {
        team_sort_pairs(t, sc, sm, k1, v1, k2, v2, m, bits_for((uint64_t)(nrows > 0 ? nrows : 1)));
        for (int64_t q = t.rank(); q < m; q += t.size()) {
            int32_t c = (int32_t)k1[q];
            int64_t p = v1[q];
            int64_t e = kidx[p];
            int64_t dst = (int64_t)C.off[c] + (q - colstart[c]);
            C.adj[dst] = A.row[e];
            C.w[dst] = A.cost[e];
        }
    }
    // forward entries: the kept edges of row r are contiguous in kidx order
    for (int64_t p = t.rank(); p < m; p += t.size()) {
        int64_t e = kidx[p];
        int32_t r = A.row[e];
        int64_t dst = (int64_t)C.off[r] + infill[r] + (p - rowstart[r]);
        C.adj[dst] = A.col[e];
        C.w[dst] = A.cost[e];
    }
    t.sync();
    sc.arena.release(mk);
    return C;
}

// lower bound of the directed graph: sum of min(0, c) (get_lb,
// include/rama_utils.h:179-190), CSUM
template <class Team>
__device__ __noinline__ double graph_lb(const Team &t, Scratch &sc, const Graph &A)
{
    return team_csum(t, sc, A.n, [=](int64_t e) -> float {
        const float c = A.cost[e];
        return c < 0.0f ? c : 0.0f;
    });
}

// compress_label_sequence (include/rama_utils.h:160-177)
template <class Team>
__device__ __noinline__ void compress_labels(const Team &t, Scratch &sc, char *, const int32_t *data, int64_t n,
                                int32_t max_label, int32_t *out)
{
    char *sm = team_smem();
    uint64_t m = sc.arena.mark();
    int32_t *mask = sc.arena.take<int32_t>((int64_t)max_label + 2);
    if (!sc.arena.ok()) return;
    for (int64_t l = t.rank(); l <= max_label; l += t.size()) mask[l] = 0;
    t.sync();
    for (int64_t k = t.rank(); k < n; k += t.size()) mask[data[k]] = 1;
    t.sync();
    team_scan<Team, int64_t>(
        t, sc, sm, (int64_t)max_label + 1, [=](int64_t l) -> int64_t { return mask[l]; },
        [=](int64_t l, int64_t pre, int64_t) { mask[l] = (int32_t)pre; });
    for (int64_t k = t.rank(); k < n; k += t.size()) out[k] = mask[data[k]];
    t.sync();
    sc.arena.release(m);
}

}  // namespace rama
