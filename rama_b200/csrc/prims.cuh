// prims.cuh -- team-generic parallel primitives (scan, canonical sums,
// stable compaction, LSD radix sort, CSR offsets, connected components).
//
// All results are independent of the team size: order-sensitive primitives
// split the input into one contiguous chunk per CTA, and the floating-point
// sums either follow a fixed reduction tree defined by element index only
// (RSUM) or carry enough bits that the order does not show (CSUM).
#pragma once
#include <cstdint>
#include <type_traits>

#include "team.cuh"

namespace rama {

constexpr unsigned FULL = 0xffffffffu;

// ---------------------------------------------------------------------------
// per-team scratch: double-buffered block partials (a primitive that writes a
// partial array always uses the buffer its predecessor did not use, so a CTA
// that runs ahead never overwrites partials another CTA is still reading),
// plus the arena.
// ---------------------------------------------------------------------------
struct Scratch {
    Arena arena;
    char *part[2];  // each >= 48 * (nblocks + 2) bytes
    int32_t *err;   // set when a bounded wait gave up (zeroed at the start of a solve)
    int parity;
    double alg_bytes;  // algorithmic bytes of the work done (team-uniform tally)
    int64_t *prof;     // optional: per-phase nanoseconds [0, PH_COUNT), then per-phase
                       // algorithmic bytes [PH_COUNT, 2 PH_COUNT) (leader only)
    uint64_t tlast;
    double alg_last;   // alg_bytes at the last phase mark
    __device__ __forceinline__ char *next_part()
    {
        parity ^= 1;
        return part[parity];
    }
};

// A workspace of `bytes` bytes at `base` (256-byte aligned) holds the two
// partial buffers, the error word and then the arena.
constexpr uint64_t SCRATCH_PART_BYTES = 16 * 4096;  // >= 48 * (max CTAs + 2)

__device__ __forceinline__ Scratch scratch_over(char *base, uint64_t bytes)
{
    Scratch sc;
    sc.part[0] = base;
    sc.part[1] = base + SCRATCH_PART_BYTES;
    sc.err = reinterpret_cast<int32_t *>(base + 2 * SCRATCH_PART_BYTES);
    sc.parity = 0;
    sc.alg_bytes = 0.0;
    sc.prof = nullptr;
    sc.tlast = 0;
    sc.alg_last = 0.0;
    sc.arena.base = base;
    sc.arena.cap = bytes - 256;
    sc.arena.lo = 2 * SCRATCH_PART_BYTES + 256;
    sc.arena.top = sc.arena.cap;
    sc.arena.peak = sc.arena.lo;
    sc.arena.want = 0;
    sc.arena.failed = 0;
    return sc;
}

// Phase timing: the team leader charges the time since the last mark, and
// the algorithmic bytes tallied since then, to `phase`.  Marks sit right
// after team syncs, so a phase's time is the span in which the whole team
// worked on it.
enum Phase : int {
    PH_INIT = 0,
    PH_CYCLES = 1,
    PH_MP_BUILD = 2,
    PH_MP_ITER = 3,
    PH_DUAL_COMMIT = 4,
    PH_MATCHING = 5,
    PH_WOC = 6,
    PH_CONTRACT = 7,
    PH_OTHER = 8,
    PH_MATCH_ITER = 9,    // the offer / match iterations of a matching round
    PH_CSORT_BIG = 10,    // contraction sort: the buckets of more than BUCKET_MAX edges
    PH_CSR = 11,          // symmetric CSR builds (cycle search, forest)
    PH_CSORT_SLOT = 12,   // contraction sort: endpoints and bucket slots
    PH_CSORT_SCATTER = 13,  // ... bucket starts and the scatter
    PH_CSORT_RANK = 14,   // ... ordering within the buckets
    PH_CONTRACT_RUNS = 15,  // contraction: run heads, sums, the new edges
    PH_MATCH_LABELS = 16,   // matching: labels of the contraction map
    PH_MATCH_FIRST = 17,    // matching: the first offer / match iteration (reads every edge)
    PH_WOC_MSF = 18,        // forest: attractive edges and their maximum spanning forest
    PH_WOC_CSR = 19,        // forest: the forest's symmetric lists
    PH_WOC_CHECKS = 20,     // forest: components, cycle checks, thresholds
    PH_WOC_ROOT = 21,       // forest: rooting (level-synchronous BFS)
    PH_WOC_PATHS = 22,      // forest: path lengths and bottleneck cuts
    PH_CYC_SEARCH = 23,     // cycle search: the expansions after the CSR
    PH_MP_NORM = 24,        // message passing: triangle normalisation
    PH_MP_CHORDS = 25,      // message passing: chords and the merged edge list
    PH_MP_INCID = 26,       // message passing: triangle-edge correspondence, incidence order
    PH_COUNT = 27
};

__device__ __forceinline__ uint64_t prof_now()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <class Team>
__device__ __forceinline__ void prof_mark(const Team &t, Scratch &sc, int phase)
{
    if (sc.prof && t.leader()) {
        uint64_t now = prof_now();
        sc.prof[phase] += (int64_t)(now - sc.tlast);
        sc.prof[PH_COUNT + phase] += (int64_t)(sc.alg_bytes - sc.alg_last);
        sc.tlast = now;
    }
    sc.alg_last = sc.alg_bytes;
}

// ---------------------------------------------------------------------------
// block-level helpers (all threads of the CTA must call)
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T warp_incl_scan(T v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T n = __shfl_up_sync(FULL, v, o);
        if (lane_id() >= o) v += n;
    }
    return v;
}

template <class T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// exclusive scan over the CTA; `sm` needs 34 * sizeof(T) bytes
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T *sm, T &total)
{
    const int w = warp_in_block(), nw = blockDim.x >> 5;
    T inc = warp_incl_scan(v);
    if (lane_id() == 31) sm[w] = inc;
    __syncthreads();
    if (w == 0) {
        T x = lane_id() < nw ? sm[lane_id()] : T(0);
        T xi = warp_incl_scan(x);
        sm[lane_id()] = xi - x;
        if (lane_id() == 31) sm[32] = xi;
    }
    __syncthreads();
    T r = sm[w] + inc - v;
    total = sm[32];
    __syncthreads();
    return r;
}

// the sum over the CTA, on every thread; `sm` needs 32 * sizeof(T) bytes
template <class T>
__device__ __forceinline__ T block_sum(T v, T *sm)
{
    v = warp_sum(v);
    if (lane_id() == 0) sm[warp_in_block()] = v;
    __syncthreads();
    const T r = warp_sum(lane_id() < (int)(blockDim.x >> 5) ? sm[lane_id()] : T(0));
    __syncthreads();
    return r;
}

template <class T>
__device__ __forceinline__ T block_max(T v, T *sm)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T n = __shfl_xor_sync(FULL, v, o);
        v = n > v ? n : v;
    }
    if (lane_id() == 0) sm[warp_in_block()] = v;
    __syncthreads();
    T r = sm[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = sm[k] > r ? sm[k] : r;
    __syncthreads();
    return r;
}

template <class T>
__device__ __forceinline__ T block_min(T v, T *sm)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T n = __shfl_xor_sync(FULL, v, o);
        v = n < v ? n : v;
    }
    if (lane_id() == 0) sm[warp_in_block()] = v;
    __syncthreads();
    T r = sm[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = sm[k] < r ? sm[k] : r;
    __syncthreads();
    return r;
}

// contiguous chunk of [0,n) owned by this CTA (multiple of blockDim)
template <class Team>
__device__ __forceinline__ void block_chunk(const Team &t, int64_t n, int64_t &lo, int64_t &hi)
{
    const int64_t nb = t.nblocks();
    int64_t ch = (n + nb - 1) / nb;
    ch = (ch + blockDim.x - 1) / blockDim.x * blockDim.x;
    lo = (int64_t)t.block() * ch;
    hi = lo + ch;
    if (lo > n) lo = n;
    if (hi > n) hi = n;
}

// ---------------------------------------------------------------------------
// team reductions (integer / min / max): one team sync
// ---------------------------------------------------------------------------

// The CTA's dynamic shared memory keeps no state between primitives, so the
// results that one warp computes for the whole CTA go through static words,
// two of them in turn: a thread that runs ahead into the next primitive writes
// the other one, and passes a barrier before it comes back to the first.

// Combines the per-CTA partials part[0, nb) written before the last team
// sync: a warp reads them with independent L2 loads (ld.global.cg: the values
// come from other SMs, so L1 must not serve them) spread over its lanes, in
// batches, then combines the lanes; the result is valid on every lane.  Only
// for exact operations (integer sums, min, max), whose result does not depend
// on the combination order.
template <class T, class Op>
__device__ __forceinline__ T warp_fold_parts(const T *part, int nb, T init, Op op)
{
    T r = init;
    constexpr int U = 5;
    for (int b = lane_id(); b < nb; b += 32 * U) {
        T v[U];
#pragma unroll
        for (int k = 0; k < U; ++k) v[k] = __ldcg(part + min(b + 32 * k, nb - 1));
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (b + 32 * k < nb) r = op(r, v[k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = op(r, __shfl_xor_sync(FULL, r, o));
    return r;
}

// The same for the whole CTA.  With every warp reading all partials, a grid of
// 296 CTAs moved 11 MB from L2 per reduction; here one warp reads them and the
// others wait for it.
template <class Team, class T, class Op>
__device__ __forceinline__ T cta_fold_parts(const Team &t, Scratch &sc, const T *part, T init, Op op)
{
    __shared__ T res[2];
    if (warp_in_block() == 0) {
        const T r = warp_fold_parts<T>(part, t.nblocks(), init, op);
        if (lane_id() == 0) res[sc.parity] = r;
    }
    __syncthreads();
    return res[sc.parity];
}

// Grid-stride loop over [0, n) in batches of U strides: load(i) for every
// item of a batch first (loads only), then store(i, value) for each, so a
// batch waits for one memory round trip instead of U.  Per thread the items
// keep their order; a load must not read what the store of an earlier item
// of the same thread writes.
template <int U = 4, class Team, class Load, class Store>
__device__ __forceinline__ void team_for_batched(const Team &t, int64_t n, Load load, Store store)
{
    const int64_t S = t.size();
    int64_t i0 = t.rank();
    for (; i0 + (U - 1) * S < n; i0 += S * U) {
        decltype(load(int64_t(0))) v[U];
#pragma unroll
        for (int k = 0; k < U; ++k) v[k] = load(i0 + k * S);
#pragma unroll
        for (int k = 0; k < U; ++k) store(i0 + k * S, v[k]);
    }
    for (; i0 < n; i0 += S) store(i0, load(i0));
}

// the sum over the team of one value per thread; one team sync
template <class Team, class T>
__device__ T team_total(const Team &t, Scratch &sc, char *sm, T v)
{
    const T s = block_sum<T>(v, reinterpret_cast<T *>(sm));
    if (t.nblocks() == 1) return s;  // the block's total, behind the block's barriers
    T *part = reinterpret_cast<T *>(sc.next_part());
    if (threadIdx.x == 0) part[t.block()] = s;
    t.sync();
    return cta_fold_parts<Team, T>(t, sc, part, T(0), [](T a, T b) { return a + b; });
}

template <class Team, class T, class Get>
__device__ T team_sum(const Team &t, Scratch &sc, char *sm, int64_t n, Get get)
{
    T s = T(0);
    {
        // four strides at a time, loads issued together
        constexpr int U = 4;
        const int64_t S = t.size();
        int64_t i = t.rank();
        for (; i + (U - 1) * S < n; i += U * S) {
            T v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) v[k] = get(i + k * S);
#pragma unroll
            for (int k = 0; k < U; ++k) s += v[k];
        }
        for (; i < n; i += S) s += get(i);
    }
    s = block_sum<T>(s, reinterpret_cast<T *>(sm));
    if (t.nblocks() == 1) return s;  // the block's total, behind the block's barriers
    T *part = reinterpret_cast<T *>(sc.next_part());
    if (threadIdx.x == 0) part[t.block()] = s;
    t.sync();
    return cta_fold_parts<Team, T>(t, sc, part, T(0), [](T a, T b) { return a + b; });
}

template <class Team, class T, class Get>
__device__ T team_max(const Team &t, Scratch &sc, char *sm, int64_t n, T init, Get get)
{
    T s = init;
    {
        constexpr int U = 4;
        const int64_t S = t.size();
        int64_t i = t.rank();
        for (; i + (U - 1) * S < n; i += U * S) {
            T x[U];
#pragma unroll
            for (int k = 0; k < U; ++k) x[k] = get(i + k * S);
#pragma unroll
            for (int k = 0; k < U; ++k) s = x[k] > s ? x[k] : s;
        }
        for (; i < n; i += S) {
            T x = get(i);
            s = x > s ? x : s;
        }
    }
    s = block_max<T>(s, reinterpret_cast<T *>(sm));
    if (t.nblocks() == 1) return s;  // the block's total, behind the block's barriers
    T *part = reinterpret_cast<T *>(sc.next_part());
    if (threadIdx.x == 0) part[t.block()] = s;
    t.sync();
    return cta_fold_parts<Team, T>(t, sc, part, init, [](T a, T b) { return b > a ? b : a; });
}

template <class Team, class T, class Get>
__device__ T team_min(const Team &t, Scratch &sc, char *sm, int64_t n, T init, Get get)
{
    T s = init;
    for (int64_t i = t.rank(); i < n; i += t.size()) {
        T x = get(i);
        s = x < s ? x : s;
    }
    s = block_min<T>(s, reinterpret_cast<T *>(sm));
    if (t.nblocks() == 1) return s;  // the block's total, behind the block's barriers
    T *part = reinterpret_cast<T *>(sc.next_part());
    if (threadIdx.x == 0) part[t.block()] = s;
    t.sync();
    return cta_fold_parts<Team, T>(t, sc, part, init, [](T a, T b) { return b < a ? b : a; });
}

// The maximum of a and the minimum of b over the team's threads, on every
// thread; one team sync.
template <class Team>
__device__ void team_fold_maxi_minf(const Team &t, Scratch &sc, char *sm, int32_t &a, float &b)
{
    auto lanes = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int32_t x = __shfl_xor_sync(FULL, a, o);
            const float y = __shfl_xor_sync(FULL, b, o);
            a = x > a ? x : a;
            b = y < b ? y : b;
        }
    };
    __shared__ int32_t ra[2];
    __shared__ float rb[2];
    lanes();
    int32_t *sa = reinterpret_cast<int32_t *>(sm);
    float *sb = reinterpret_cast<float *>(sm + 128);
    if (lane_id() == 0) {
        sa[warp_in_block()] = a;
        sb[warp_in_block()] = b;
    }
    __syncthreads();
    a = sa[0];
    b = sb[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
        a = sa[k] > a ? sa[k] : a;
        b = sb[k] < b ? sb[k] : b;
    }
    __syncthreads();
    if (t.nblocks() == 1) return;
    int32_t *part = reinterpret_cast<int32_t *>(sc.next_part());
    if (threadIdx.x == 0) {
        part[2 * t.block()] = a;
        part[2 * t.block() + 1] = __float_as_int(b);
    }
    t.sync();
    if (warp_in_block() == 0) {
        constexpr int U = 5;
        const int nb = t.nblocks();
        const int2 *p = reinterpret_cast<const int2 *>(part);
        for (int k = lane_id(); k < nb; k += 32 * U) {
            int2 v[U];
#pragma unroll
            for (int q = 0; q < U; ++q) v[q] = __ldcg(p + min(k + 32 * q, nb - 1));
#pragma unroll
            for (int q = 0; q < U; ++q) {  // (a partial read twice changes nothing)
                a = v[q].x > a ? v[q].x : a;
                b = __int_as_float(v[q].y) < b ? __int_as_float(v[q].y) : b;
            }
        }
        lanes();
        if (lane_id() == 0) {
            ra[sc.parity] = a;
            rb[sc.parity] = b;
        }
    }
    __syncthreads();
    a = ra[sc.parity];
    b = rb[sc.parity];
}

// The maximum of ia(i) and the minimum of fb(i) over [0, n) in one pass and
// one team sync (both exact, so the result does not depend on the order).
template <class Team, class IA, class FB>
__device__ void team_maxi_minf(const Team &t, Scratch &sc, char *sm, int64_t n, int32_t iinit, float finit, IA ia,
                               FB fb, int32_t &imax, float &fmin)
{
    int32_t a = iinit;
    float b = finit;
    {
        constexpr int U = 4;
        const int64_t S = t.size();
        int64_t i = t.rank();
        for (; i + (U - 1) * S < n; i += U * S) {
            int32_t x[U];
            float y[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                x[k] = ia(i + k * S);
                y[k] = fb(i + k * S);
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                a = x[k] > a ? x[k] : a;
                b = y[k] < b ? y[k] : b;
            }
        }
        for (; i < n; i += S) {
            const int32_t x = ia(i);
            const float y = fb(i);
            a = x > a ? x : a;
            b = y < b ? y : b;
        }
    }
    team_fold_maxi_minf(t, sc, sm, a, b);
    imax = a;
    fmin = b;
}

// The sum of the partials of the CTAs before this one, and of all.
template <class Team, class T>
__device__ __forceinline__ void cta_prefix_parts(const Team &t, Scratch &sc, const T *part, T &base, T &total)
{
    __shared__ T res[2][2];
    if (warp_in_block() == 0) {
        T b = T(0), a = T(0);
        constexpr int U = 5;
        const int nb = t.nblocks();
        for (int x = lane_id(); x < nb; x += 32 * U) {
            T v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) v[k] = __ldcg(part + min(x + 32 * k, nb - 1));
#pragma unroll
            for (int k = 0; k < U; ++k) {
                if (x + 32 * k < nb) a += v[k];
                if (x + 32 * k < t.block()) b += v[k];
            }
        }
        b = warp_sum(b);
        a = warp_sum(a);
        if (lane_id() == 0) {
            res[sc.parity][0] = b;
            res[sc.parity][1] = a;
        }
    }
    __syncthreads();
    base = res[sc.parity][0];
    total = res[sc.parity][1];
}

// ---------------------------------------------------------------------------
// team exclusive scan: out(i, prefix, value) is called for every i in [0,n)
// in chunk order; returns the total.  Two team syncs; outputs are visible to
// the whole team on return.  The second pass takes tiles of blockDim * ITEMS
// elements (ITEMS = 4 for 8-byte sums, 8 for 4-byte ones): each warp a contiguous segment of 32 * SCAN_ITEMS,
// lane l its elements l, l + 32, ... (coalesced loads); the warp scans them
// in order with shuffles, and one block scan of the warp totals per tile
// keeps the CTA's barriers few.  Integer sums only, so the result does not
// depend on the tiling.
//
// Where every CTA's chunk is at most one tile (up to 303,000 elements on 148
// CTAs) the values are read and scanned once, before the team sync, and stay
// in registers: such scans wait for round trips, not for bandwidth.
// ---------------------------------------------------------------------------
template <class T>
struct ScanItems {
    static constexpr int value = sizeof(T) == 8 ? 4 : 8;
};

// team_scan_while ends after the total (one team sync) when go_on(total) is
// false.
template <class Team, class T, class In, class Go, class Out>
__device__ T team_scan_while(const Team &t, Scratch &sc, char *sm, int64_t n, In in, Go go_on, Out out)
{
    constexpr int ITEMS = ScanItems<T>::value;
    T *tsm = reinterpret_cast<T *>(sm);
    int64_t lo, hi;
    block_chunk(t, n, lo, hi);
    const int64_t TILE = (int64_t)blockDim.x * ITEMS;
    const int64_t wseg = (int64_t)warp_in_block() * 32 * ITEMS;
    const bool one = (n + TILE - 1) / TILE <= t.nblocks();
    T base = T(0), total = T(0);
    auto prefix = [&](T mine) {  // base and total from the CTAs' sums; one team sync
        total = mine;
        if (t.nblocks() == 1) return;
        T *part = reinterpret_cast<T *>(sc.next_part());
        if (threadIdx.x == 0) part[t.block()] = mine;
        t.sync();
        cta_prefix_parts(t, sc, part, base, total);
    };
    if (!one) {
        T s = T(0);
        // four strides at a time, loads issued together
        constexpr int U = 4;
        const int64_t S = blockDim.x;
        int64_t i = lo + threadIdx.x;
        for (; i + (U - 1) * S < hi; i += U * S) {
            T v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) v[k] = in(i + k * S);
#pragma unroll
            for (int k = 0; k < U; ++k) s += v[k];
        }
        for (; i < hi; i += S) s += in(i);
        prefix(block_sum<T>(s, tsm));
        if (!go_on(total)) return total;
    }
    for (int64_t tile = lo; one || tile < hi; tile += TILE) {
        const int64_t i0 = tile + wseg + lane_id();
        T v[ITEMS], ex[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) v[k] = i0 + 32 * k < hi ? in(i0 + 32 * k) : T(0);
        T wrun = T(0);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const T x = warp_incl_scan(v[k]);
            ex[k] = wrun + x - v[k];
            wrun += __shfl_sync(FULL, x, 31);
        }
        T ts;
        const T wofs = block_excl_scan<T>(lane_id() == 0 ? wrun : T(0), tsm, ts);
        if (one) {
            prefix(ts);
            if (!go_on(total)) return total;
        }
        const T wbase = base + __shfl_sync(FULL, wofs, 0);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k)
            if (i0 + 32 * k < hi) out(i0 + 32 * k, wbase + ex[k], v[k]);
        if (one) break;
        base += ts;
    }
    t.sync();
    return total;
}

template <class Team, class T, class In, class Out>
__device__ T team_scan(const Team &t, Scratch &sc, char *sm, int64_t n, In in, Out out)
{
    return team_scan_while<Team, T>(t, sc, sm, n, in, [](T) { return true; }, out);
}

// stable compaction: emit(i, pos) for every kept i; returns the count
template <class Team, class Keep, class Emit>
__device__ int64_t team_compact(const Team &t, Scratch &sc, char *sm, int64_t n, Keep keep, Emit emit)
{
    return team_scan_while<Team, int64_t>(
        t, sc, sm, n, [=](int64_t i) -> int64_t { return keep(i) ? 1 : 0; }, [](int64_t total) { return total != 0; },
        [=](int64_t i, int64_t pos, int64_t v) {
            if (v) emit(i, pos);
        });
}

// ---------------------------------------------------------------------------
// CSUM: compensated FP64 sum of floats.  Every thread adds its elements with
// TwoSum (the sum and its error, about 106 bits together), the pairs of a CTA
// and then of the team are merged the same way, and the result is rounded
// once.
//
// Its error.  The sum's part of a merge is exact together with the error that
// joins the compensation; what is lost are the roundings of the compensation,
// two a merge.  After k merges of values that add up to X in magnitude the
// compensation is at most k u X (u = 2^-53), so m of them lose at most
// m^2 u^2 X in all, m being a thread's additions and the some 20 merges over
// its team.  Against the last place of the result S that is m^2 u (X / |S|):
// for 25 M elements 2^-36 on the whole GPU (m = 350), 2^-30 on a cluster of 16
// CTAs (3,050), 2^-22 on one CTA (48,800), and the oracle's fixed tree (m = 320)
// 2^-36, all times X / |S|.  So for values of one sign (X = |S|: the bounds and
// the thresholds) the result is the correctly rounded sum whatever the team,
// and the oracle's, unless the exact sum comes that close to the middle between
// two doubles without lying on it.  Where values cancel (the objective), the
// factor X / |S| comes in: two teams may round differently once it takes up
// those bits.
//
// What bounds it: the passes over memory for large n (7 FP64 additions per
// element take less), the team sync and the L2 round trips for small n.  So
// the elements are strided over all threads and there is one team sync.  One
// warp per 4,096 elements with its 128-step chain, and two team syncs, took
// 1.34 ms
// for the six matching thresholds of the 24.8 M edge volume (with what is timed
// beside them); this takes 0.74.
// ---------------------------------------------------------------------------
struct csum_t {
    double s, c;
};

__device__ __forceinline__ csum_t cs_merge(csum_t a, csum_t b)
{
    double s = __dadd_rn(a.s, b.s);
    double bb = __dsub_rn(s, a.s);
    double e = __dadd_rn(__dsub_rn(a.s, __dsub_rn(s, bb)), __dsub_rn(b.s, bb));
    csum_t r;
    r.s = s;
    r.c = __dadd_rn(__dadd_rn(a.c, b.c), e);
    return r;
}

__device__ __forceinline__ csum_t cs_add(csum_t a, float x) { return cs_merge(a, csum_t{(double)x, 0.0}); }

// The totals over the team of two pairs per thread, rounded, on every thread
// (a count rides along as a second pair: its additions are exact).  One team
// sync, which also makes the caller's earlier stores visible to the team.
struct csum2_t {
    double a, b;
    float m;  // the minimum of the threads' third values
};

template <class Team>
__device__ __noinline__ csum2_t team_csum_fold(const Team &t, Scratch &sc, csum_t a, csum_t b, float m = 3.4e38f)
{
    __shared__ csum_t wa[32], wb[32];
    __shared__ float wm[32];
    __shared__ csum2_t res[2];
    // merging is commutative, so a butterfly leaves the same pair on every lane
    auto fold = [&](int lanes) {
        for (int off = 1; off < lanes; off <<= 1) {
            csum_t x, y;
            x.s = __shfl_xor_sync(FULL, a.s, off);
            x.c = __shfl_xor_sync(FULL, a.c, off);
            y.s = __shfl_xor_sync(FULL, b.s, off);
            y.c = __shfl_xor_sync(FULL, b.c, off);
            a = cs_merge(a, x);
            b = cs_merge(b, y);
            m = fminf(m, __shfl_xor_sync(FULL, m, off));
        }
    };
    const int nw = blockDim.x >> 5;
    fold(32);
    if (lane_id() == 0) {
        wa[warp_in_block()] = a;
        wb[warp_in_block()] = b;
        wm[warp_in_block()] = m;
    }
    __syncthreads();
    csum_t *part = reinterpret_cast<csum_t *>(sc.next_part());  // 48 B per CTA
    if (warp_in_block() == 0) {
        a = lane_id() < nw ? wa[lane_id()] : csum_t{0.0, 0.0};
        b = lane_id() < nw ? wb[lane_id()] : csum_t{0.0, 0.0};
        m = wm[lane_id() < nw ? lane_id() : 0];
        fold(nw);
        if (lane_id() == 0) {
            if (t.nblocks() == 1) {
                res[sc.parity].a = __dadd_rn(a.s, a.c);
                res[sc.parity].b = __dadd_rn(b.s, b.c);
                res[sc.parity].m = m;
            } else {
                part[3 * t.block()] = a;
                part[3 * t.block() + 1] = b;
                part[3 * t.block() + 2].s = (double)m;
            }
        }
    }
    t.sync();
    if (t.nblocks() > 1) {
        if (warp_in_block() == 0) {
            a = b = csum_t{0.0, 0.0};
            const double2 *p = reinterpret_cast<const double2 *>(part);
            constexpr int U = 5;
            const int nb = t.nblocks();
            for (int k = lane_id(); k < nb; k += 32 * U) {
                double2 x[U], y[U];
                double z[U];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const int c = min(k + 32 * q, nb - 1);
                    x[q] = __ldcg(p + 3 * c);
                    y[q] = __ldcg(p + 3 * c + 1);
                    z[q] = __ldcg(reinterpret_cast<const double *>(p + 3 * c + 2));
                }
#pragma unroll
                for (int q = 0; q < U; ++q)
                    if (k + 32 * q < nb) {
                        a = cs_merge(a, csum_t{x[q].x, x[q].y});
                        b = cs_merge(b, csum_t{y[q].x, y[q].y});
                        m = fminf(m, (float)z[q]);
                    }
            }
            fold(32);
            if (lane_id() == 0) {
                res[sc.parity].a = __dadd_rn(a.s, a.c);
                res[sc.parity].b = __dadd_rn(b.s, b.c);
                res[sc.parity].m = m;
            }
        }
        __syncthreads();
    }
    return res[sc.parity];
}

// The sum of get(k) over [0, n) on every thread; *count receives the number
// of k with cnt(k).
template <class Team, class Get, class Cnt>
__device__ double team_csum_count(const Team &t, Scratch &sc, int64_t n, Get get, Cnt cnt, int64_t *count)
{
    csum_t a = {0.0, 0.0};
    int64_t c = 0;
    {
        // eight strides at a time, loads issued together
        constexpr int U = 8;
        const int64_t S = t.size();
        int64_t i = t.rank();
        for (; i + (U - 1) * S < n; i += U * S) {
            float x[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                x[k] = get(i + k * S);
                c += cnt(i + k * S) ? 1 : 0;
            }
#pragma unroll
            for (int k = 0; k < U; ++k) a = cs_add(a, x[k]);
        }
        for (; i < n; i += S) {
            a = cs_add(a, get(i));
            c += cnt(i) ? 1 : 0;
        }
    }
    const csum2_t r = team_csum_fold(t, sc, a, csum_t{(double)c, 0.0});
    *count = (int64_t)r.b;
    return r.a;
}

template <class Team, class Get>
__device__ double team_csum(const Team &t, Scratch &sc, int64_t n, Get get)
{
    int64_t unused = 0;
    return team_csum_count(t, sc, n, get, [](int64_t) { return false; }, &unused);
}

// RSUM of n <= 64 values v(k), k in [0, n), by one thread: the loads of a
// group of 8 together, then the tree over the 32 lanes (a lane holds values l
// and l + 32) as the pairwise sum of four trees over 8; +0.0 in the empty
// lanes changes no sum.
template <class Get>
__device__ __forceinline__ float rsum_upto64(int n, Get v)
{
    auto group = [&](int q) {
        double x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = 8 * q + k < n ? __dadd_rn(0.0, (double)v(8 * q + k)) : 0.0;
        if (n > 32) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (8 * q + k + 32 < n) x[k] = __dadd_rn(x[k], (double)v(8 * q + k + 32));
        }
        return __dadd_rn(__dadd_rn(__dadd_rn(x[0], x[1]), __dadd_rn(x[2], x[3])),
                         __dadd_rn(__dadd_rn(x[4], x[5]), __dadd_rn(x[6], x[7])));
    };
    if (n <= 8) return (float)group(0);
    return (float)__dadd_rn(__dadd_rn(group(0), group(1)), __dadd_rn(group(2), group(3)));
}

// RSUM over values v(k), k in [0,n) by ONE thread (n <= 32): the oracle's
// 32-lane FP64 sum with one element per lane, then a pairwise tree over the
// lanes (empty lanes hold +0.0).  Computed with a stack of complete subtrees,
// which merges exactly the same pairs in the same order.
template <class Get>
__device__ __forceinline__ float rsum_serial(int n, Get v)
{
    double st[7];
    int sz[7];
    int top = 0;
    for (int k = 0; k < n; ++k) {
        double x = __dadd_rn(0.0, (double)v(k));
        int s = 1;
        while (top > 0 && sz[top - 1] == s) {
            x = __dadd_rn(st[top - 1], x);
            s <<= 1;
            --top;
        }
        st[top] = x;
        sz[top] = s;
        ++top;
    }
    double r = 0.0;
    if (top > 0) {
        r = st[top - 1];
        for (int q = top - 2; q >= 0; --q) r = __dadd_rn(st[q], r);
    }
    return (float)r;
}

// runs up to this length are summed in the pass over all edges, longer ones
// from a list
constexpr int RSUM_THREAD_MAX = 8;

// Sums of more than RSUM_CHUNK values are defined by chunks: each chunk of
// RSUM_CHUNK consecutive values is summed as above (kept in double), and the
// chunk sums are summed the same way (chunk c to lane c mod 32), so that many
// warps can share one long sum.
constexpr int64_t RSUM_CHUNK = 4096;

// the pairwise tree over a warp's 32 lane values; the result on every lane
__device__ __forceinline__ double rsum_lane_tree(double a)
{
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        double o = __shfl_down_sync(FULL, a, off);
        if ((lane_id() & (2 * off - 1)) == 0) a = __dadd_rn(a, o);
    }
    return __shfl_sync(FULL, a, 0);
}

// the RSUM of at most RSUM_CHUNK values v(0..len) by a warp, in double (not
// rounded); a lane adds its values k, k + 32, ... in that order, eight of them
// loaded at a time
template <class Get>
__device__ __forceinline__ double rsum_chunk_warp(int64_t len, Get v)
{
    double a = 0.0;
    int64_t k = lane_id();
    for (; k + 7 * 32 < len; k += 8 * 32) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = v(k + 32 * j);
#pragma unroll
        for (int j = 0; j < 8; ++j) a = __dadd_rn(a, (double)x[j]);
    }
    for (; k < len; k += 32) a = __dadd_rn(a, (double)v(k));
    return rsum_lane_tree(a);
}

// the same sum by a whole warp (any n); result valid on every lane
template <class Get>
__device__ __forceinline__ float rsum_warp(int64_t n, Get v)
{
    if (n <= RSUM_CHUNK) return (float)rsum_chunk_warp(n, v);
    double acc = 0.0;  // this lane's chunks: c = lane, lane + 32, ...
    for (int64_t c = 0; c * RSUM_CHUNK < n; ++c) {
        const int64_t base = c * RSUM_CHUNK;
        const int64_t len = n - base < RSUM_CHUNK ? n - base : RSUM_CHUNK;
        const double d = rsum_chunk_warp(len, [=](int64_t k) { return v(base + k); });
        if (lane_id() == (int)(c & 31)) acc = __dadd_rn(acc, d);
    }
    return (float)rsum_lane_tree(acc);
}

// ---------------------------------------------------------------------------
// LSD radix sort of (uint64 key, 4- or 8-byte value) pairs, 8-bit digits, stable.
// The sorted data ends in (*keys, *vals) (pointers may be swapped with the
// spare buffers).
//
// One read of the keys counts the digits of every pass at once (a pass only
// permutes the keys, so its digit totals are known up front).  Each pass then
// moves the data once.  The input is cut into tiles of blockDim * SORT_ITEMS
// keys (half as many with 8-byte values); CTA b takes tiles b, b + nblocks,
// ... in increasing order.  Per tile it
//   - ranks the keys stably: per-warp digit counters, and ballots over the
//     digit bits for the lanes holding the same digit;
//   - finds the tile's output offset per digit by decoupled look-back over
//     the counts the preceding tiles published;
//   - stages the tile in digit order in shared memory and writes each digit's
//     run contiguously.
// One team sync per pass.  The look-back waits are bounded; a wait that gives
// up sets the scratch error word and the sort stops with the last complete
// pass (a permutation of the input).  A single-CTA team keeps running
// offsets instead of looking back.  A pass in which one digit holds every key
// is the identity and is skipped.
// ---------------------------------------------------------------------------
constexpr int SORT_ITEMS = 8;
constexpr uint64_t LB_VALUE = (uint64_t(1) << 58) - 1;
constexpr uint64_t LB_AGG = uint64_t(1) << 62;     // tile count published
constexpr uint64_t LB_PREFIX = uint64_t(2) << 62;  // inclusive prefix published
constexpr int LB_SPIN_LIMIT = 1 << 20;

__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t *p)
{
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t *p, uint64_t v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// values travel through shared memory as raw 4- or 8-byte words
template <class V>
struct SortWord {
    static_assert(sizeof(V) == 4 || sizeof(V) == 8, "sort values are 4 or 8 bytes");
    using type = typename std::conditional<sizeof(V) == 8, uint64_t, uint32_t>::type;
    static __device__ __forceinline__ type to(V v)
    {
        type u;
        memcpy(&u, &v, sizeof(V));
        return u;
    }
    static __device__ __forceinline__ V from(type u)
    {
        V v;
        memcpy(&v, &u, sizeof(V));
        return v;
    }
};

// Decoupled look-back of one tile for all 256 digits: the exclusive count of
// digit d over tiles [0, tile) in the words of pass tag `tag`.  The CTA loads
// the published words of LB_WINDOW preceding tiles per digit at once (into
// `win`, LB_WINDOW * 256 words of shared memory); each digit's thread then
// adds tile counts from the nearest tile back until it meets an inclusive
// prefix, or a tile that has not published yet (the next window starts
// there).  Called by every thread of the CTA; returns the count on threads
// d < 256.  Waits are bounded: after LB_SPIN_LIMIT rounds without progress
// the error word is set and the count is left incomplete.
constexpr int LB_WINDOW = 16;

// bytes of the sort's staging area: a tile of keys and values, or the
// look-back window, whichever is larger
__host__ __device__ constexpr int sort_stage_bytes(int threads)
{
    return threads * SORT_ITEMS * 12 > LB_WINDOW * 256 * 8 ? threads * SORT_ITEMS * 12 : LB_WINDOW * 256 * 8;
}

__device__ __forceinline__ int64_t sort_lookback(const uint64_t *flags, int64_t tile, uint64_t tag, uint64_t *win,
                                                 int64_t *posS, int32_t *err)
{
    const int d = threadIdx.x;
    int64_t excl = 0;
    bool done = tile == 0;
    if (d < 256) posS[d] = done ? -1 : tile - 1;
    int idle = 0;
    for (;;) {
        if (!__syncthreads_or(d < 256 && !done)) break;
        for (int x = threadIdx.x; x < LB_WINDOW * 256; x += blockDim.x) {
            const int64_t j = posS[x & 255] - (x >> 8);
            if (posS[x & 255] >= 0) win[x] = j >= 0 ? ld_relaxed(flags + j * 256 + (x & 255)) : (LB_PREFIX | tag);
        }
        __syncthreads();
        bool stuck = false;
        if (d < 256 && !done) {
            int64_t pos = posS[d];
            int k = 0;
            for (; k < LB_WINDOW; ++k) {
                const uint64_t w = win[k * 256 + d];
                if ((w & (uint64_t(15) << 58)) != tag || !(w >> 62)) break;  // not published yet
                excl += (int64_t)(w & LB_VALUE);
                if ((w >> 62) == 2) {
                    done = true;
                    break;
                }
            }
            stuck = k == 0 && !done;
            pos -= k;
            if (done) pos = -1;
            posS[d] = pos;
        }
        if (__syncthreads_or(stuck)) {
            if (++idle > LB_SPIN_LIMIT || (idle % 1024 == 0 && *(volatile int32_t *)err)) {
                if (d == 0) atomicOr(err, 1);
                break;
            }
            if (idle > 16) __nanosleep(256);
        } else {
            idle = 0;
        }
    }
    return excl;
}

// Lanes of the warp holding the same 9-bit label (a digit, or 256 for "no
// key"), from nine ballots over the label's bits.
__device__ __forceinline__ unsigned warp_peers9(unsigned label)
{
    unsigned m = FULL;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const unsigned bit = (label >> b) & 1u;
        const unsigned ball = __ballot_sync(FULL, bit);
        m &= bit ? ball : ~ball;
    }
    return m;
}

template <class Team, class V>
__device__ __noinline__ void team_sort_pairs(const Team &t, Scratch &sc, char *, uint64_t *&keys_io, V *&vals_io,
                                             uint64_t *&keys2_io, V *&vals2_io, int64_t n, int bits)
{
    if (n <= 1 || bits <= 0) return;
    char *sm = team_smem();
    uint64_t *keys = keys_io, *keys2 = keys2_io;
    V *vals = vals_io, *vals2 = vals2_io;
    using W = typename SortWord<V>::type;
    constexpr int ITEMS = sizeof(V) == 8 ? SORT_ITEMS / 2 : SORT_ITEMS;
    const int P = (bits + 7) / 8;
    const int nb = t.nblocks();
    const int NW = blockDim.x >> 5;
    const int TILE = blockDim.x * ITEMS;
    const int64_t ntiles = (n + TILE - 1) / TILE;
    uint64_t am = sc.arena.mark();
    uint32_t *ghist = sc.arena.take<uint32_t>(8 * 256);
    uint64_t *flags = nb > 1 ? sc.arena.take<uint64_t>((uint64_t)ntiles * 256) : nullptr;
    if (!sc.arena.ok()) return;
    uint32_t *wcnt = reinterpret_cast<uint32_t *>(sm);  // NW * 256
    uint64_t *skeys = reinterpret_cast<uint64_t *>(sm + NW * 1024);
    W *svals = reinterpret_cast<W *>(sm + NW * 1024 + TILE * 8);
    char *q = sm + NW * 1024 + sort_stage_bytes(blockDim.x);  // staging area: either tile or the window
    uint32_t *tstart = reinterpret_cast<uint32_t *>(q);
    int64_t *gbase = reinterpret_cast<int64_t *>(q + 1024);
    int64_t *bucket = reinterpret_cast<int64_t *>(q + 3072);
    int64_t *run = reinterpret_cast<int64_t *>(q + 5120);
    int64_t *ssm = reinterpret_cast<int64_t *>(q + 7168);   // 34
    int64_t *posS = reinterpret_cast<int64_t *>(q + 7440);  // 256
    uint64_t *win = skeys;                                  // LB_WINDOW * 256, look-back only
    uint32_t *lh = reinterpret_cast<uint32_t *>(skeys);    // P * 256, counting only
    const int w = warp_in_block();

    // 0. digit totals of every pass
    for (int i = threadIdx.x; i < P * 256; i += blockDim.x) lh[i] = 0;
    for (int64_t i = t.rank(); i < 8 * 256; i += t.size()) ghist[i] = 0;
    if (flags)
        for (int64_t i = t.rank(); i < ntiles * 256; i += t.size()) flags[i] = 0;
    __syncthreads();
    for (int64_t i = t.rank(); i < n; i += t.size()) {
        const uint64_t k = keys[i];
        for (int p = 0; p < P; ++p) atomicAdd(&lh[p * 256 + (int)((k >> (8 * p)) & 255)], 1u);
    }
    __syncthreads();
    t.sync();
    for (int i = threadIdx.x; i < P * 256; i += blockDim.x)
        if (lh[i]) atomicAdd(&ghist[i], lh[i]);
    t.sync();

    for (int p = 0; p < P; ++p) {
        const int shift = 8 * p;
        const uint64_t tag = (uint64_t)(p + 1) << 58;
        const int64_t tot = threadIdx.x < 256 ? (int64_t)__ldcg(ghist + p * 256 + threadIdx.x) : 0;
        int64_t all;
        const int64_t ex = block_excl_scan<int64_t>(tot, ssm, all);
        if (threadIdx.x < 256) {
            bucket[threadIdx.x] = ex;
            run[threadIdx.x] = 0;
        }
        if (__syncthreads_or(threadIdx.x < 256 && tot == n)) continue;  // identity pass
        for (int64_t tile = t.block(); tile < ntiles; tile += nb) {
            const int64_t t0 = tile * TILE;
            const int tn = (int)((n - t0) < TILE ? (n - t0) : TILE);
            for (int d = lane_id(); d < 256; d += 32) wcnt[w * 256 + d] = 0;
            uint64_t mk[ITEMS];
            W mv[ITEMS];
            uint32_t mr[ITEMS];
            const int wb = w * 32 * ITEMS;
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const int li = wb + k * 32 + lane_id();
                const bool valid = li < tn;
                mk[k] = valid ? keys[t0 + li] : 0;
                mv[k] = valid ? SortWord<V>::to(vals[t0 + li]) : W(0);
            }
            __syncwarp();
            // 1. stable rank within the warp
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const bool valid = wb + k * 32 + lane_id() < tn;
                const int d = valid ? (int)((mk[k] >> shift) & 255) : 256;
                const unsigned peers = warp_peers9((unsigned)d);
                const int leader = __ffs(peers) - 1;
                uint32_t b0 = 0;
                if (valid && lane_id() == leader) {
                    b0 = wcnt[w * 256 + d];
                    wcnt[w * 256 + d] = b0 + __popc(peers);
                }
                b0 = __shfl_sync(FULL, b0, leader);
                mr[k] = b0 + __popc(peers & lanemask_lt());
                __syncwarp();
            }
            __syncthreads();
            // 2. per digit: offsets of the warps, the tile's count and start
            uint32_t cnt = 0;
            if (threadIdx.x < 256) {
                for (int qw = 0; qw < NW; ++qw) {
                    const uint32_t c = wcnt[qw * 256 + threadIdx.x];
                    wcnt[qw * 256 + threadIdx.x] = cnt;
                    cnt += c;
                }
            }
            int64_t tt;
            const int64_t ts = block_excl_scan<int64_t>((int64_t)cnt, ssm, tt);
            // 3. output offset of the tile per digit
            if (threadIdx.x < 256) tstart[threadIdx.x] = (uint32_t)ts;
            int64_t excl = 0;
            if (nb == 1) {
                if (threadIdx.x < 256) {
                    excl = run[threadIdx.x];
                    run[threadIdx.x] = excl + cnt;
                }
            } else {
                if (threadIdx.x < 256)
                    st_relaxed(flags + tile * 256 + threadIdx.x, (tile == 0 ? LB_PREFIX : LB_AGG) | tag | (uint64_t)cnt);
                excl = sort_lookback(flags, tile, tag, win, posS, sc.err);
                if (threadIdx.x < 256 && tile > 0)
                    st_relaxed(flags + tile * 256 + threadIdx.x, LB_PREFIX | tag | (uint64_t)(excl + cnt));
            }
            if (threadIdx.x < 256) gbase[threadIdx.x] = bucket[threadIdx.x] + excl;
            __syncthreads();
            // 4. stage the tile in digit order
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                if (wb + k * 32 + lane_id() < tn) {
                    const int d = (int)((mk[k] >> shift) & 255);
                    const uint32_t loc = tstart[d] + wcnt[w * 256 + d] + mr[k];
                    skeys[loc] = mk[k];
                    svals[loc] = mv[k];
                }
            }
            __syncthreads();
            // 5. write the digit runs
            for (int i = threadIdx.x; i < tn; i += blockDim.x) {
                const uint64_t key = skeys[i];
                const int d = (int)((key >> shift) & 255);
                const int64_t dst = gbase[d] + (i - (int64_t)tstart[d]);
                if (dst >= 0 && dst < n) {
                    keys2[dst] = key;
                    vals2[dst] = SortWord<V>::from(svals[i]);
                }
            }
            __syncthreads();
        }
        t.sync();
        if (__ldcg(sc.err)) break;  // keep the last complete pass
        uint64_t *tk = keys;
        keys = keys2;
        keys2 = tk;
        V *tv = vals;
        vals = vals2;
        vals2 = tv;
    }
    keys_io = keys;
    keys2_io = keys2;
    vals_io = vals;
    vals2_io = vals2;
    sc.arena.release(am);
}

// shared-memory bytes the sort needs for a CTA of `threads` threads
__host__ __device__ constexpr int sort_smem_bytes(int threads)
{
    return (threads / 32) * 1024 + sort_stage_bytes(threads) + 7440 + 256 * 8;
}

// ---------------------------------------------------------------------------
// Bucket sort: n items ordered by (bucket(i), sub(i)), bucket(i) in [0, nb),
// sub(i) below 2^64 - 1.  Items with equal (bucket, sub) end in no particular
// order: callers fold the item index into sub when the order must be stable,
// and otherwise use it only where equal keys stand for equal items.  Each item takes a slot in
// its bucket by an atomic counter (one atomic per bucket and warp), an
// exclusive scan of the counts gives the bucket starts, one scatter places
// the items, and each bucket is then sorted by its sub keys: buckets of up to
// 64 items by ranking every item (it lands after the keys of its bucket that
// are smaller), up to 256 items by a warp and up to BUCKET_MAX by a CTA
// (bitonic networks in shared memory).  The
// atomic slots only decide where an item lands before its bucket is sorted,
// so with distinct keys the result is the one sorted order.
// Outputs: keys_out[p] = sub of the p-th item, idx_out[p] = its index,
// bstart[0, nb] = first position of each bucket.  Returns false, having
// written nothing useful, when a bucket holds more than BUCKET_MAX items (the
// caller then sorts with team_sort_pairs).
// ---------------------------------------------------------------------------
constexpr int BUCKET_MAX = 4096;

// bitonic sort of (key, idx) pairs in shared memory, `m` items padded to the
// power of two P with +inf keys; threads [lo, lo + nth) of the group work,
// `bar` synchronises them
template <class Bar>
__device__ __forceinline__ void smem_bitonic(uint64_t *key, int32_t *idx, int m, int P, int lane, int nth, Bar bar)
{
    for (int i = m + lane; i < P; i += nth) {
        key[i] = ~uint64_t(0);
        idx[i] = -1;
    }
    bar();
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < P; i += nth) {
                const int x = i ^ j;
                if (x > i) {
                    const uint64_t a = key[i], b = key[x];
                    if ((a > b) == ((i & k) == 0)) {
                        key[i] = b;
                        key[x] = a;
                        const int32_t t = idx[i];
                        idx[i] = idx[x];
                        idx[x] = t;
                    }
                }
            }
            bar();
        }
    }
}

// Items handled at once by a thread in the sort's streaming passes: their
// loads are issued together, so a pass waits for one memory round trip per
// batch instead of one per item.
constexpr int SORT_BATCH = 4;

// the slot of this lane's item in bucket b (-1: no item): the lanes of a warp
// that share a bucket take theirs with one atomic; every lane must call
__device__ __forceinline__ int32_t bucket_slot(int32_t *counts, int32_t b)
{
    const unsigned peers = __match_any_sync(FULL, b);
    const int leader = __ffs(peers) - 1;
    int32_t s = 0;
    if (b >= 0 && lane_id() == leader) s = atomicAdd(&counts[b], __popc(peers));
    return __shfl_sync(FULL, s, leader) + __popc(peers & lanemask_lt());
}

// The same for U items a lane at a time: the atomics of all of them are in
// flight together (the contraction's slot passes of the 24.8 M edge volume
// waited for four in turn before).
template <int U>
__device__ __forceinline__ void bucket_slots(int32_t *counts, const int32_t (&b)[U], int32_t (&s)[U])
{
    unsigned peers[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
        peers[k] = __match_any_sync(FULL, b[k]);
        s[k] = 0;
        if (b[k] >= 0 && lane_id() == __ffs(peers[k]) - 1) s[k] = atomicAdd(&counts[b[k]], __popc(peers[k]));
    }
#pragma unroll
    for (int k = 0; k < U; ++k)
        s[k] = __shfl_sync(FULL, s[k], __ffs(peers[k]) - 1) + __popc(peers[k] & lanemask_lt());
}

// bucket(i) and sub(i) must only load.
template <class Team, class Bk, class Sub>
__device__ bool team_bucket_sort(const Team &t, Scratch &sc, char *sm, int64_t n, int32_t nb, Bk bucket, Sub sub,
                                 uint64_t *keys_out, int32_t *idx_out, int32_t *bstart)
{
    uint64_t am = sc.arena.mark();
    int32_t *slot = sc.arena.take<int32_t>(n + 1);
    int32_t *tb = sc.arena.take<int32_t>(n + 1);    // bucket of the item at each scattered position
    int32_t *ti = sc.arena.take<int32_t>(n + 1);    // item index at each scattered position
    uint64_t *tk = sc.arena.take<uint64_t>(n + 1);  // sub key at each scattered position
    int32_t *lists = sc.arena.take<int32_t>(2 * ((int64_t)nb + 1));  // warp buckets, CTA buckets
    int32_t *nlist = sc.arena.take<int32_t>(4);
    if (!sc.arena.ok()) return false;
    int32_t *wlist = lists, *clist = lists + nb + 1;
    for (int64_t b = t.rank(); b <= nb; b += t.size()) bstart[b] = 0;
    if (t.rank() < 4) nlist[t.rank()] = 0;
    t.sync();
    // slots: the lanes of a warp that share a bucket take theirs with one
    // atomic; a warp handles SORT_BATCH strides at once (item k of a batch is
    // base + k * size + lane)
    {
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        for (int64_t base = (int64_t)t.rank() - lane_id(); base < n; base += S * U) {
            int32_t b[U], s[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const int64_t i = base + k * S + lane_id();
                b[k] = i < n ? (int32_t)bucket(i) : -1;
            }
            bucket_slots<U>(bstart, b, s);
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (base + k * S + lane_id() < n) slot[base + k * S + lane_id()] = s[k];
        }
    }
    t.sync();
    // bucket starts; buckets of more than 64 items go to the warp and CTA
    // lists (any order); one of more than BUCKET_MAX ends the sort
    team_scan<Team, int64_t>(
        t, sc, sm, nb, [=](int64_t b) -> int64_t { return bstart[b]; },
        [=](int64_t b, int64_t pre, int64_t c) {
            bstart[b] = (int32_t)pre;
            if (c > BUCKET_MAX)
                nlist[2] = 1;
            else if (c > 256)
                clist[atomicAdd(&nlist[1], 1)] = (int32_t)b;
            else if (c > 64)
                wlist[atomicAdd(&nlist[0], 1)] = (int32_t)b;
        });
    if (uread(&nlist[2]) != 0) {
        t.sync();  // every thread has seen it before the memory is handed on
        sc.arena.release(am);
        return false;
    }
    if (t.rank() == 0) bstart[nb] = (int32_t)n;
    t.sync();
    {
        // full batches of SORT_BATCH strides (loads first, then the
        // gathers of the bucket starts, then the stores), then one at a time
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        int64_t i0 = t.rank();
        for (; i0 + (U - 1) * S < n; i0 += U * S) {
            int32_t b[U], p[U];
            uint64_t kv[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                b[k] = (int32_t)bucket(i0 + k * S);
                p[k] = slot[i0 + k * S];
                kv[k] = sub(i0 + k * S);
            }
#pragma unroll
            for (int k = 0; k < U; ++k) p[k] += bstart[b[k]];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                tk[p[k]] = kv[k];
                ti[p[k]] = (int32_t)(i0 + k * S);
                tb[p[k]] = b[k];
            }
        }
        for (; i0 < n; i0 += S) {
            const int32_t b = (int32_t)bucket(i0);
            const int64_t p = (int64_t)bstart[b] + slot[i0];
            tk[p] = sub(i0);
            ti[p] = (int32_t)i0;
            tb[p] = b;
        }
    }
    t.sync();
    // up to 64 items: each item's rank in its bucket is the number of smaller
    // keys there (neighbouring threads read the same bucket)
    {
        // the place of item p: its rank in its bucket (a bucket of more than
        // 64 items is copied as it is and sorted below)
        auto place = [=](int64_t p, int32_t s, int32_t e, uint64_t key) -> int32_t {
            if (e - s > 64) return (int32_t)p;
            int32_t r = 0;
            for (int32_t q = s; q < e; ++q) {
                const uint64_t o = tk[q];
                r += o < key || (o == key && q < p);
            }
            return s + r;
        };
        constexpr int U = SORT_BATCH;
        const int64_t S = t.size();
        int64_t p0 = t.rank();
        for (; p0 + (U - 1) * S < n; p0 += U * S) {
            int32_t b[U], s[U], e[U], iv[U], dst[U];
            uint64_t kv[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                b[k] = tb[p0 + k * S];
                kv[k] = tk[p0 + k * S];
                iv[k] = ti[p0 + k * S];
            }
#pragma unroll
            for (int k = 0; k < U; ++k) {
                s[k] = bstart[b[k]];
                e[k] = bstart[b[k] + 1];
            }
#pragma unroll
            for (int k = 0; k < U; ++k) dst[k] = place(p0 + k * S, s[k], e[k], kv[k]);
#pragma unroll
            for (int k = 0; k < U; ++k) {
                keys_out[dst[k]] = kv[k];
                idx_out[dst[k]] = iv[k];
            }
        }
        for (; p0 < n; p0 += S) {
            const int32_t b = tb[p0];
            const uint64_t key = tk[p0];
            const int32_t dst = place(p0, bstart[b], bstart[b + 1], key);
            keys_out[dst] = key;
            idx_out[dst] = ti[p0];
        }
    }
    t.sync();
    // 65..256 items: a warp, bitonic in its share of the staging area
    {
        const int NW = blockDim.x >> 5;
        const int w = warp_in_block();
        char *stage = sm + NW * 1024;
        uint64_t *wk = reinterpret_cast<uint64_t *>(stage) + w * 256;
        int32_t *wi = reinterpret_cast<int32_t *>(stage + NW * 256 * 8) + w * 256;
        const int32_t nw = uread(&nlist[0]);
        for (int64_t q = team_warp(t); q < nw; q += team_nwarps(t)) {
            const int32_t b = wlist[q], s = bstart[b], m = bstart[b + 1] - s;
            int P = 32;
            while (P < m) P <<= 1;
            for (int x = lane_id(); x < m; x += 32) {
                wk[x] = keys_out[s + x];
                wi[x] = idx_out[s + x];
            }
            __syncwarp();
            smem_bitonic(wk, wi, m, P, lane_id(), 32, [] { __syncwarp(); });
            for (int x = lane_id(); x < m; x += 32) {
                keys_out[s + x] = wk[x];
                idx_out[s + x] = wi[x];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // 257..BUCKET_MAX items: a CTA
    {
        const int NW = blockDim.x >> 5;
        char *stage = sm + NW * 1024;
        uint64_t *ck = reinterpret_cast<uint64_t *>(stage);
        int32_t *ci = reinterpret_cast<int32_t *>(stage + BUCKET_MAX * 8);
        const int32_t nc = uread(&nlist[1]);
        for (int64_t q = t.block(); q < nc; q += t.nblocks()) {
            const int32_t b = clist[q], s = bstart[b], m = bstart[b + 1] - s;
            int P = 512;
            while (P < m) P <<= 1;
            for (int x = threadIdx.x; x < m; x += blockDim.x) {
                ck[x] = keys_out[s + x];
                ci[x] = idx_out[s + x];
            }
            __syncthreads();
            smem_bitonic(ck, ci, m, P, threadIdx.x, blockDim.x, [] { __syncthreads(); });
            for (int x = threadIdx.x; x < m; x += blockDim.x) {
                keys_out[s + x] = ck[x];
                idx_out[s + x] = ci[x];
            }
            __syncthreads();
        }
    }
    t.sync();
    sc.arena.release(am);
    return true;
}

// ---------------------------------------------------------------------------
// Grouping by a bucket, for passes that know their items: the caller counts
// each item into its bucket with an atomic whose result is the item's slot
// (in the pass that computes the bucket anyway), team_bucket_starts turns the
// counts into starts, the caller scatters one key per item to start + slot,
// and every item then finds its place as the number of smaller keys in its
// bucket (bucket_rank).  Buckets of more than BUCKET_SMALL keys are listed by
// team_bucket_starts and sorted by team_sort_long_buckets (a warp each up to
// 256 keys, a CTA up to BUCKET_MAX); what lies beyond is the caller's general
// path.  Against team_bucket_sort this moves one key per item instead of
// an index, a bucket and a key in and out, and takes five team syncs
// instead of eight.
// ---------------------------------------------------------------------------
constexpr int BUCKET_SMALL = 64;

struct BucketLists {
    int32_t *warp, *cta;  // buckets of 65..256 and of 257..BUCKET_MAX keys
    int32_t *n;           // [0], [1]: their numbers, [2]: some bucket is larger, the rest is the caller's, who zeroes
                          // what is used
    bool some;            // some bucket holds more than BUCKET_SMALL keys (comes with the scan of the counts, so
                          // that the numbers are read only then)
    __device__ __forceinline__ bool has_long() const { return some && uread(&n[0]) + uread(&n[1]) > 0; }
    __device__ __forceinline__ bool has_big() const { return some && uread(&n[2]) != 0; }
};

__device__ __forceinline__ BucketLists bucket_lists(Scratch &sc, int64_t nitems)
{
    BucketLists L;
    L.warp = sc.arena.take<int32_t>(nitems / (BUCKET_SMALL + 1) + 1);
    L.cta = sc.arena.take<int32_t>(nitems / 257 + 1);
    L.n = sc.arena.take<int32_t>(8);
    L.some = false;
    return L;
}

// counts[0, nb) -> starts, counts[nb] = the total (also returned); each(b,
// start, count) is called once per bucket.  Two team syncs.
template <class Team, class Each>
__device__ __forceinline__ int64_t team_bucket_starts(const Team &t, Scratch &sc, char *sm, int32_t nb,
                                                      int32_t *counts, BucketLists &lists, Each each)
{
    // sums of counts below 2^36, the number of long buckets above
    constexpr int64_t LONG = int64_t(1) << 36;
    const BucketLists L = lists;
    const int64_t total = team_scan<Team, int64_t>(
        t, sc, sm, nb,
        [=](int64_t b) -> int64_t {
            const int32_t c = counts[b];
            return c > BUCKET_SMALL ? c + LONG : c;
        },
        [=](int64_t b, int64_t sums, int64_t v) {
            const int64_t pre = sums & (LONG - 1), c = v & (LONG - 1);
            counts[b] = (int32_t)pre;
            if (b == nb - 1) counts[nb] = (int32_t)(pre + c);
            if (c > BUCKET_MAX)
                L.n[2] = 1;
            else if (c > 256)
                L.cta[atomicAdd(&L.n[1], 1)] = (int32_t)b;
            else if (c > BUCKET_SMALL)
                L.warp[atomicAdd(&L.n[0], 1)] = (int32_t)b;
            each(b, (int32_t)pre, (int32_t)c);
        });
    lists.some = total >= LONG;
    return total & (LONG - 1);
}

// keys in [s, e) ordered before the one at p (equal keys by position); four
// loads at a time, past the end the last key again, which is not counted
template <class K>
__device__ __forceinline__ int32_t bucket_rank(const K *keys, int32_t s, int32_t e, K key, int32_t p)
{
    int32_t r = 0;
    for (int32_t x = s; x < e; x += 4) {
        K a[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = keys[min(x + k, e - 1)];
#pragma unroll
        for (int k = 0; k < 4; ++k) r += x + k < e && (a[k] < key || (a[k] == key && x + k < p));
    }
    return r;
}

template <class K, class Bar>
__device__ __forceinline__ void smem_bitonic_keys(K *key, int m, int P, int lane, int nth, Bar bar)
{
    for (int i = m + lane; i < P; i += nth) key[i] = ~K(0);
    bar();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < P; i += nth) {
                const int x = i ^ j;
                if (x > i) {
                    const K a = key[i], b = key[x];
                    if ((a > b) == ((i & k) == 0)) {
                        key[i] = b;
                        key[x] = a;
                    }
                }
            }
            bar();
        }
}

// Sorts the listed buckets of the keys load(p) and calls emit(b, p, key) for
// every sorted position p, after all loads of the bucket.  Keys are below
// ~K(0).  The caller syncs.
template <class K, class Team, class Load, class Emit>
__device__ __forceinline__ void team_sort_long_buckets(const Team &t, char *sm, BucketLists L, const int32_t *start,
                                                       Load load, Emit emit)
{
    {
        K *wk = reinterpret_cast<K *>(sm) + warp_in_block() * 256;
        const int32_t nw = uread(&L.n[0]);
        for (int64_t q = team_warp(t); q < nw; q += team_nwarps(t)) {
            const int32_t b = L.warp[q], s = start[b], m = start[b + 1] - s;
            int P = 128;
            while (P < m) P <<= 1;
            for (int x = lane_id(); x < m; x += 32) wk[x] = load(s + x);
            __syncwarp();
            smem_bitonic_keys(wk, m, P, lane_id(), 32, [] { __syncwarp(); });
            for (int x = lane_id(); x < m; x += 32) emit(b, s + x, wk[x]);
            __syncwarp();
        }
    }
    __syncthreads();
    {
        K *ck = reinterpret_cast<K *>(sm);
        const int32_t nc = uread(&L.n[1]);
        for (int64_t q = t.block(); q < nc; q += t.nblocks()) {
            const int32_t b = L.cta[q], s = start[b], m = start[b + 1] - s;
            int P = 512;
            while (P < m) P <<= 1;
            for (int x = threadIdx.x; x < m; x += blockDim.x) ck[x] = load(s + x);
            __syncthreads();
            smem_bitonic_keys(ck, m, P, threadIdx.x, blockDim.x, [] { __syncthreads(); });
            for (int x = threadIdx.x; x < m; x += blockDim.x) emit(b, s + x, ck[x]);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// off[v] = first k with ids(k) >= v, v in [0, nv]; ids sorted ascending
// ---------------------------------------------------------------------------
template <class Team, class Ids>
__device__ void team_offsets(const Team &t, int64_t n, int32_t nv, Ids ids, int32_t *off)
{
    for (int64_t k = t.rank(); k <= n; k += t.size()) {
        int32_t cur = k < n ? ids(k) : nv;
        int32_t prev = k == 0 ? -1 : ids(k - 1);
        for (int32_t v = prev + 1; v <= cur; ++v) off[v] = (int32_t)k;
    }
    t.sync();
}

// ---------------------------------------------------------------------------
// connected components: lab[v] = minimum vertex id of v's component.
// Edges are given as pairs (a(e), b(e)), e in [0,m).  Hook-and-compress with
// parent[x] <= x throughout (so chains strictly decrease and every loop ends);
// repeats until no edge joins two trees, at most 64 rounds.
// ---------------------------------------------------------------------------
template <class Team, class EA, class EB>
__device__ bool team_cc(const Team &t, Scratch &sc, int32_t nv, int64_t m, EA ea, EB eb, int32_t *lab)
{
    uint64_t am = sc.arena.mark();
    int32_t *flags = sc.arena.take<int32_t>(65);
    if (!sc.arena.ok()) return false;
    for (int64_t v = t.rank(); v < nv; v += t.size()) lab[v] = (int32_t)v;
    for (int k = t.rank(); k < 65; k += t.size()) flags[k] = 0;
    t.sync();
    bool converged = false;
    for (int it = 0; it < 64; ++it) {
        for (int64_t e = t.rank(); e < m; e += t.size()) {
            int32_t a = ea(e), b = eb(e);
            if (a == b) continue;
            int32_t ra = a, rb = b;
            for (int s = 0; s < 1 << 16; ++s) {
                int32_t p = ((volatile int32_t *)lab)[ra];
                if (p == ra) break;
                ra = p;
            }
            for (int s = 0; s < 1 << 16; ++s) {
                int32_t p = ((volatile int32_t *)lab)[rb];
                if (p == rb) break;
                rb = p;
            }
            if (ra != rb) {
                int32_t hi = ra > rb ? ra : rb, lo = ra > rb ? rb : ra;
                atomicMin(&lab[hi], lo);
                flags[it] = 1;
            }
        }
        t.sync();
        for (int64_t v = t.rank(); v < nv; v += t.size()) {
            int32_t x = lab[v];
            for (int s = 0; s < 1 << 16; ++s) {
                int32_t p = ((volatile int32_t *)lab)[x];
                if (p == x) break;
                x = p;
            }
            lab[v] = x;
        }
        t.sync();
        if (!uread(&flags[it])) {
            converged = true;
            break;
        }
    }
    sc.arena.release(am);
    return converged;
}

}  // namespace rama
