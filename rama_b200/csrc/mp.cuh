// mp.cuh -- triangle message passing (src/multicut_message_passing.cu:15-360)
// and the dual solver loop (src/dual_solver.cu:7-63).
//
// Layout (all SoA in the arena): triangles t1<t2<t3 sorted and unique; their
// edge indices e12/e13/e23 into the merged edge list (the graph's edges plus
// the triangle chords it lacks, cost 0).  The messages a triangle sends to
// its edges go to `slot`, which holds each edge's incoming messages
// contiguously in incidence order (triangle order); pos[3t + corner] is the
// slot of triangle t's message to that corner's edge.  Each edge then takes
// the RSUM of its run of slots, which replaces the reference's float
// atomicAdd by a deterministic sum.
#pragma once
#include "cycles.cuh"

namespace rama {

struct Mp {
    int64_t T, E;
    int32_t *t1, *t2, *t3;
    int32_t *e12, *e13, *e23;
    float *c12, *c13, *c23;
    float *slot;  // 3T: incoming messages, edge by edge in incidence order
    int32_t *pos;  // 3T: slot of triangle t's message to corner c at 3t + c
    int32_t *row, *col;
    float *cost;
    float *share;      // E: cost / number of incident triangles (covered edges)
    int32_t *inc_off;  // E + 1: first slot of each edge
    int32_t *longe;    // edges with more than RSUM_THREAD_MAX incident triangles
    int64_t nlong;     // ... of them those with up to 64, from the front
    int64_t nhuge;     // ... and the others, from the back (longe_cap)
    int64_t longe_cap;
    int inplace;  // row, col and cost are the graph's own arrays (no chords)
};

// position of (a,b) in a (row,col)-sorted list with row offsets `off`
__device__ __forceinline__ int64_t find_edge(const int32_t *off, const int32_t *col, int32_t a, int32_t b)
{
    int32_t lo = off[a], hi = off[a + 1];
    while (lo < hi) {
        int32_t m = (lo + hi) >> 1;
        if (col[m] < b)
            lo = m + 1;
        else
            hi = m;
    }
    return (lo < off[a + 1] && col[lo] == b) ? lo : -1;
}

// find_edge of N (a, b) pairs at once: the binary searches step in lockstep,
// so each step's loads are in flight together
template <int N>
__device__ __forceinline__ void find_edges(const int32_t *off, const int32_t *col, const int32_t (&a)[N],
                                           const int32_t (&b)[N], int32_t (&out)[N])
{
    int32_t lo[N], hi[N], end[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        lo[k] = off[a[k]];
        hi[k] = end[k] = off[a[k] + 1];
    }
    for (int step = 0; step < 32; ++step) {
        int32_t m[N], c[N];
        bool any = false;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            m[k] = (lo[k] + hi[k]) >> 1;
            c[k] = lo[k] < hi[k] ? col[m[k]] : 0;
        }
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (lo[k] < hi[k]) {
                any = true;
                if (c[k] < b[k])
                    lo[k] = m[k] + 1;
                else
                    hi[k] = m[k];
            }
        if (!any) break;
    }
    int32_t c[N];
#pragma unroll
    for (int k = 0; k < N; ++k) c[k] = lo[k] < end[k] ? col[lo[k]] : 0;
#pragma unroll
    for (int k = 0; k < N; ++k) out[k] = (lo[k] < end[k] && c[k] == b[k]) ? lo[k] : -1;
}

// number of entries of row a with col < b, plus all rows < a
__device__ __forceinline__ int64_t lower_edge(const int32_t *off, const int32_t *col, int32_t a, int32_t b)
{
    int32_t lo = off[a], hi = off[a + 1];
    while (lo < hi) {
        int32_t m = (lo + hi) >> 1;
        if (col[m] < b)
            lo = m + 1;
        else
            hi = m;
    }
    return lo;
}

// multicut_message_passing ctor (:65-176)
//
// Bound by the number of dependent passes for small and mid-size graphs (a
// team sync and one or two L2 round trips each), by the gathers of the edge
// lookups for large ones.  So everything that can share a pass does: the
// lookup of a triangle's sides counts the chords of each row, or, where every
// side is known to be an edge (3-cycles), the triangles of each edge; the scan
// of those counts gives the edges' shares and the list of long edges; and one
// key per item is moved to order chords and incidences (team_bucket_starts).
// On the 201,720-edge cube in PD+ mode the builds took 7.5 ms as passes of their own,
// and 4.3 this way; the lists of attractive neighbours 5.3 and 1.8.
template <class Team>
__device__ __noinline__ bool mp_build(const Team &t, Scratch &sc, char *, const Graph &graph, TriBuf &tb, Mp &out)
{
    char *sm = team_smem();
    const Graph A = graph;  // pointers in registers
    Mp mp;
    const int32_t nmax = A.max_dim();
    // normalize_triangles (:79)
    const int64_t T = tri_normalize(t, sc, sm, tb, tb.num, nmax);
    prof_mark(t, sc, PH_MP_NORM);
    if (!sc.arena.ok()) return false;
    mp.T = T;
    mp.t1 = tb.t1;
    mp.t2 = tb.t2;
    mp.t3 = tb.t3;
    mp.e12 = sc.arena.take<int32_t>(T + 1);
    mp.e13 = sc.arena.take<int32_t>(T + 1);
    mp.e23 = sc.arena.take<int32_t>(T + 1);
    mp.c12 = sc.arena.take<float>(T + 1);
    mp.c13 = sc.arena.take<float>(T + 1);
    mp.c23 = sc.arena.take<float>(T + 1);
    mp.slot = sc.arena.take<float>(3 * T + 1);
    mp.pos = sc.arena.take<int32_t>(3 * T + 1);
    int32_t *aoff = sc.arena.take<int32_t>((int64_t)nmax + 2);  // row offsets of A over [0, nmax]
    int32_t *slot = sc.arena.take<int32_t>(3 * T + 1);          // a side's slot among the chords of its row,
                                                                // then among the triangles of its edge
    int32_t *key = sc.arena.take<int32_t>(3 * T + 1);           // the keys moved to their buckets
    if (!sc.arena.ok()) return false;
    const bool closed = tb.closed != 0;
    const int32_t nbk = nmax + 1;
    // the counts of the first grouping: triangles per edge, or chords per row
    const uint64_t cm = sc.arena.mark();
    BucketLists L = bucket_lists(sc, 3 * T);
    int32_t *cst = nullptr;
    if (closed) {
        mp.inc_off = sc.arena.take<int32_t>(A.n + 2);
        if (!sc.arena.ok()) return false;
        for (int64_t e = t.rank(); e <= A.n; e += t.size()) mp.inc_off[e] = 0;
    } else {
        cst = sc.arena.take<int32_t>((int64_t)nbk + 1);
        if (!sc.arena.ok()) return false;
        for (int64_t v = t.rank(); v <= nbk; v += t.size()) cst[v] = 0;
    }
    if (t.rank() < 8) L.n[t.rank()] = 0;
    team_offsets(t, A.n, nmax, [=](int64_t e) { return A.row[e]; }, aoff);
    // the triangles' sides among the graph's edges; `each` gets the three
    // positions (-1: not an edge) with all lanes of the warp present.  Two
    // triangles a lane at a time where there are that many.
    auto lookup = [=](auto each) {
        const int64_t S = t.size();
        int64_t k0 = (int64_t)t.rank() - lane_id();
        for (; k0 + S + 31 < T; k0 += 2 * S) {
            const int64_t k[2] = {k0 + lane_id(), k0 + S + lane_id()};
            int32_t f[6], from[6], to[6];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int32_t a = mp.t1[k[q]], b = mp.t2[k[q]], c = mp.t3[k[q]];
                from[3 * q] = from[3 * q + 1] = a;
                from[3 * q + 2] = to[3 * q] = b;
                to[3 * q + 1] = to[3 * q + 2] = c;
            }
            find_edges<6>(aoff, A.col, from, to, f);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int32_t g[3] = {f[3 * q], f[3 * q + 1], f[3 * q + 2]};
                mp.e12[k[q]] = g[0];
                mp.e13[k[q]] = g[1];
                mp.e23[k[q]] = g[2];
                const int32_t h[3] = {from[3 * q], from[3 * q + 1], from[3 * q + 2]};
                each(k[q], true, h, g);
            }
        }
        for (; k0 < T; k0 += S) {
            const int64_t k = k0 + lane_id();
            int32_t f[3] = {-1, -1, -1}, from[3] = {0, 0, 0};
            if (k < T) {
                const int32_t a = mp.t1[k], b = mp.t2[k], c = mp.t3[k];
                const int32_t to[3] = {b, c, c};
                from[0] = from[1] = a;
                from[2] = b;
                find_edges<3>(aoff, A.col, from, to, f);
                mp.e12[k] = f[0];
                mp.e13[k] = f[1];
                mp.e23[k] = f[2];
            }
            each(k, k < T, from, f);
        }
    };
    // counts a triangle's sides into their edges (neighbouring triangles share
    // their first side often, the others seldom)
    auto count_sides = [=](int64_t k, bool valid, const int32_t (&f)[3], int32_t *inc) {
        const int32_t s0 = bucket_slot(inc, valid ? f[0] : -1);
        if (valid) {
            const int32_t s1 = atomicAdd(&inc[f[1]], 1), s2 = atomicAdd(&inc[f[2]], 1);
            slot[3 * k] = s0;
            slot[3 * k + 1] = s1;
            slot[3 * k + 2] = s2;
        }
    };
    int64_t nn = 0;
    if (closed) {
        int32_t *inc = mp.inc_off;
        lookup([=](int64_t k, bool valid, const int32_t (&)[3], const int32_t (&f)[3]) {
            count_sides(k, valid, f, inc);
        });
        t.sync();
    } else {
        // chords: sides that are no edges, by their row
        lookup([=](int64_t k, bool valid, const int32_t (&from)[3], const int32_t (&f)[3]) {
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const bool chord = valid && f[s] < 0;
                const int32_t x = bucket_slot(cst, chord ? from[s] : -1);
                if (valid) slot[3 * k + s] = chord ? x : -1;
            }
        });
        t.sync();
        nn = team_bucket_starts(t, sc, sm, nbk, cst, L, [](int64_t, int32_t, int32_t) {});
    }
    mp.inplace = nn == 0;
    if (mp.inplace) {
        mp.E = A.n;
        mp.row = A.row;
        mp.col = A.col;
        mp.cost = A.cost;
        prof_mark(t, sc, PH_MP_CHORDS);
        if (!closed) {
            sc.arena.release(cm);
            L = bucket_lists(sc, 3 * T);
            mp.inc_off = sc.arena.take<int32_t>(A.n + 2);
            if (!sc.arena.ok()) return false;
            for (int64_t e = t.rank(); e <= A.n; e += t.size()) mp.inc_off[e] = 0;
            if (t.rank() < 8) L.n[t.rank()] = 0;
            t.sync();
            int32_t *inc = mp.inc_off;
            for (int64_t k0 = (int64_t)t.rank() - lane_id(); k0 < T; k0 += t.size()) {
                const int64_t k = k0 + lane_id();
                int32_t f[3] = {-1, -1, -1};
                if (k < T) {
                    f[0] = mp.e12[k];
                    f[1] = mp.e13[k];
                    f[2] = mp.e23[k];
                }
                count_sides(k, k < T, f, inc);
            }
            t.sync();
        }
    } else {
        // the chords' columns, ascending within each row (equal ones adjacent),
        // and their rows
        int32_t *ccol = sc.arena.take<int32_t>(nn + 1), *crow = sc.arena.take<int32_t>(nn + 1);
        int32_t *upre = sc.arena.take<int32_t>(nn + 1);  // distinct chords before each position
        int32_t *ucol = sc.arena.take<int32_t>(nn + 1), *urow = sc.arena.take<int32_t>(nn + 1);
        if (!sc.arena.ok()) return false;
        auto side_from = [=](int64_t q) { return q % 3 == 2 ? mp.t2[q / 3] : mp.t1[q / 3]; };
        auto side_to = [=](int64_t q) { return q % 3 == 0 ? mp.t2[q / 3] : mp.t3[q / 3]; };
        int32_t *corner_edge[3] = {mp.e12, mp.e13, mp.e23};
        if (!L.has_big()) {
            struct Sides {
                int32_t p[3], b, c;  // positions (-1: an edge) and the two larger vertices
            };
            team_for_batched<2>(
                t, T,
                [=](int64_t k) {
                    const int32_t a = mp.t1[k], s0 = slot[3 * k], s1 = slot[3 * k + 1], s2 = slot[3 * k + 2];
                    Sides x;
                    x.b = mp.t2[k];
                    x.c = mp.t3[k];
                    const int32_t ca = cst[a], cb = cst[x.b];
                    x.p[0] = s0 < 0 ? -1 : ca + s0;
                    x.p[1] = s1 < 0 ? -1 : ca + s1;
                    x.p[2] = s2 < 0 ? -1 : cb + s2;
                    return x;
                },
                [=](int64_t, const Sides &x) {
                    if (x.p[0] >= 0) key[x.p[0]] = x.b;
                    if (x.p[1] >= 0) key[x.p[1]] = x.c;
                    if (x.p[2] >= 0) key[x.p[2]] = x.c;
                });
            t.sync();
            // a chord's place goes to the triangle too, as -2 - place (a chord
            // of a long row keeps -1 and is searched for below)
            for (int64_t k = t.rank(); k < T; k += t.size()) {
                const int32_t a = mp.t1[k], b = mp.t2[k], c = mp.t3[k];
                const int32_t sl[3] = {slot[3 * k], slot[3 * k + 1], slot[3 * k + 2]};
                const int32_t from[3] = {a, a, b}, to[3] = {b, c, c};
                const int32_t sa = cst[a], ea = cst[a + 1], sb = cst[b], eb = cst[b + 1];
                const int32_t s[3] = {sa, sa, sb}, e[3] = {ea, ea, eb};
                int32_t p[3];
#pragma unroll
                for (int c3 = 0; c3 < 3; ++c3) {
                    p[c3] = -1;
                    if (sl[c3] >= 0 && e[c3] - s[c3] <= BUCKET_SMALL)
                        p[c3] = s[c3] + bucket_rank(key, s[c3], e[c3], to[c3], s[c3] + sl[c3]);
                }
#pragma unroll
                for (int c3 = 0; c3 < 3; ++c3)
                    if (p[c3] >= 0) {
                        ccol[p[c3]] = to[c3];
                        crow[p[c3]] = from[c3];
                        corner_edge[c3][k] = -2 - p[c3];
                    }
            }
            if (L.has_long())
                team_sort_long_buckets<uint32_t>(
                    t, sm, L, cst, [=](int32_t p) { return (uint32_t)key[p]; },
                    [=](int32_t b, int32_t p, uint32_t c) {
                        ccol[p] = (int32_t)c;
                        crow[p] = b;
                    });
            t.sync();
        } else {
            // a row with more than BUCKET_MAX chords: LSD radix sort of (row, col)
            const int nb = bits_for((uint64_t)(nmax > 0 ? nmax : 1));
            const uint64_t rm = sc.arena.mark();
            uint64_t *k1 = sc.arena.take<uint64_t>(nn + 1), *k2 = sc.arena.take<uint64_t>(nn + 1);
            int32_t *v1 = sc.arena.take<int32_t>(nn + 1), *v2 = sc.arena.take<int32_t>(nn + 1);
            if (!sc.arena.ok()) return false;
            team_compact(
                t, sc, sm, 3 * T, [=](int64_t q) { return slot[q] >= 0; },
                [=](int64_t q, int64_t p) {
                    k1[p] = pack_key(side_from(q), side_to(q), nb);
                    v1[p] = 0;
                });
            team_sort_pairs(t, sc, sm, k1, v1, k2, v2, nn, 2 * nb);
            for (int64_t p = t.rank(); p < nn; p += t.size()) {
                ccol[p] = (int32_t)(k1[p] & ((uint64_t(1) << nb) - 1));
                crow[p] = (int32_t)(k1[p] >> nb);
            }
            t.sync();
            sc.arena.release(rm);
        }
        const int64_t nu = team_scan<Team, int64_t>(
            t, sc, sm, nn,
            [=](int64_t p) -> int64_t { return p == 0 || crow[p] != crow[p - 1] || ccol[p] != ccol[p - 1]; },
            [=](int64_t p, int64_t pre, int64_t v) {
                upre[p] = (int32_t)pre;
                if (p == nn - 1) upre[nn] = (int32_t)(pre + v);
                if (v) {
                    ucol[pre] = ccol[p];
                    urow[pre] = crow[p];
                }
            });
        // merged edge list (set_union_by_key, :130-158) and its row offsets;
        // an edge counts the chords before it among those of its own row
        const int64_t E = A.n + nu;
        mp.E = E;
        mp.row = sc.arena.take<int32_t>(E + 1);
        mp.col = sc.arena.take<int32_t>(E + 1);
        mp.cost = sc.arena.take<float>(E + 1);
        int32_t *moff = sc.arena.take<int32_t>((int64_t)nmax + 2);
        mp.inc_off = sc.arena.take<int32_t>(E + 2);
        const uint64_t pm = sc.arena.mark();
        int32_t *apos = sc.arena.take<int32_t>(A.n + 1);  // places of the graph's edges in the merged list
        int32_t *upos = sc.arena.take<int32_t>(nu + 1);   // ... and of the distinct chords
        if (!sc.arena.ok()) return false;
        team_for_batched(
            t, A.n,
            [=](int64_t e) {
                const int32_t r = A.row[e], c = A.col[e];
                int32_t lo = upre[cst[r]], hi = upre[cst[r + 1]];
                while (lo < hi) {
                    const int32_t m = (lo + hi) >> 1;
                    if (ucol[m] < c)
                        lo = m + 1;
                    else
                        hi = m;
                }
                return make_int4(lo, r, c, __float_as_int(A.cost[e]));
            },
            [=](int64_t e, int4 v) {
                const int64_t p = e + v.x;
                apos[e] = (int32_t)p;
                mp.row[p] = v.y;
                mp.col[p] = v.z;
                mp.cost[p] = __int_as_float(v.w);
            });
        for (int64_t k = t.rank(); k < nu; k += t.size()) {
            const int32_t a = urow[k], b = ucol[k];
            const int64_t p = k + lower_edge(aoff, A.col, a, b);
            upos[k] = (int32_t)p;
            mp.row[p] = a;
            mp.col[p] = b;
            mp.cost[p] = 0.0f;
        }
        for (int64_t v = t.rank(); v <= nmax; v += t.size()) moff[v] = aoff[v] + upre[cst[v]];
        for (int64_t e = t.rank(); e <= E; e += t.size()) mp.inc_off[e] = 0;
        if (t.rank() < 8) L.n[t.rank()] = 0;
        t.sync();
        prof_mark(t, sc, PH_MP_CHORDS);
        // correspondences (compute_triangle_edge_correspondence, :15-62), from
        // the positions that the lookup and the chords' order gave
        int32_t *inc = mp.inc_off;
        for (int64_t k0 = (int64_t)t.rank() - lane_id(); k0 < T; k0 += t.size()) {
            const int64_t k = k0 + lane_id();
            int32_t f[3] = {-1, -1, -1};
            if (k < T) {
                int32_t u[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) f[c] = corner_edge[c][k];
#pragma unroll
                for (int c = 0; c < 3; ++c) u[c] = f[c] <= -2 ? upre[-1 - f[c]] - 1 : 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    if (f[c] == -1) {
                        const int32_t a = c == 2 ? mp.t2[k] : mp.t1[k], b = c == 0 ? mp.t2[k] : mp.t3[k];
                        f[c] = (int32_t)find_edge(moff, mp.col, a, b);
                    } else {
                        f[c] = f[c] >= 0 ? apos[f[c]] : upos[u[c]];
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) corner_edge[c][k] = f[c];
            }
            count_sides(k, k < T, f, inc);
        }
        t.sync();
        sc.arena.release(pm);
    }
    // first slot of each edge, its share of its cost, and the edges whose
    // incoming messages a whole warp sums
    mp.share = sc.arena.take<float>(mp.E + 1);
    mp.longe_cap = 3 * T / (RSUM_THREAD_MAX + 1) + 1;
    mp.longe = sc.arena.take<int32_t>(mp.longe_cap);
    if (!sc.arena.ok()) return false;
    team_bucket_starts(t, sc, sm, (int32_t)mp.E, mp.inc_off, L, [=](int64_t e, int32_t, int32_t n) {
        mp.share[e] = n > 0 ? __fdiv_rn(mp.cost[e], (float)n) : 0.0f;
        if (n > 64)
            mp.longe[mp.longe_cap - 1 - atomicAdd(&L.n[4], 1)] = (int32_t)e;
        else if (n > RSUM_THREAD_MAX)
            mp.longe[atomicAdd(&L.n[3], 1)] = (int32_t)e;
    });
    mp.nlong = uread(&L.n[3]);
    mp.nhuge = uread(&L.n[4]);
    // incidence order: 3t + corner ascending within each edge; the rank of
    // each (triangle, corner) in that order is its slot
    if (!L.has_big()) {
        struct Runs {
            int32_t s[3], e[3], p[3];
        };
        auto runs = [=](int64_t k) {
            const int32_t x[3] = {mp.e12[k], mp.e13[k], mp.e23[k]};
            Runs r;
#pragma unroll
            for (int c = 0; c < 3; ++c) r.p[c] = slot[3 * k + c];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                r.s[c] = mp.inc_off[x[c]];
                r.e[c] = mp.inc_off[x[c] + 1];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) r.p[c] += r.s[c];
            return r;
        };
        team_for_batched<2>(t, T, runs, [=](int64_t k, const Runs &r) {
#pragma unroll
            for (int c = 0; c < 3; ++c) key[r.p[c]] = (int32_t)(3 * k + c);
        });
        t.sync();
        team_for_batched<2>(
            t, T,
            [=](int64_t k) {
                Runs r = runs(k);
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    r.p[c] = r.e[c] - r.s[c] <= BUCKET_SMALL
                                 ? r.s[c] + bucket_rank(key, r.s[c], r.e[c], (int32_t)(3 * k + c), r.p[c])
                                 : -1;
                return r;
            },
            [=](int64_t k, const Runs &r) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (r.p[c] >= 0) mp.pos[3 * k + c] = r.p[c];
            });
        if (L.has_long())
            team_sort_long_buckets<uint32_t>(
                t, sm, L, mp.inc_off, [=](int32_t p) { return (uint32_t)key[p]; },
                [=](int32_t, int32_t p, uint32_t q) { mp.pos[q] = p; });
        t.sync();
    } else {
        const uint64_t rm = sc.arena.mark();
        uint64_t *k1 = sc.arena.take<uint64_t>(3 * T + 1), *k2 = sc.arena.take<uint64_t>(3 * T + 1);
        int32_t *v1 = sc.arena.take<int32_t>(3 * T + 1), *v2 = key;
        if (!sc.arena.ok()) return false;
        for (int64_t k = t.rank(); k < T; k += t.size()) {
            k1[3 * k] = (uint64_t)mp.e12[k];
            k1[3 * k + 1] = (uint64_t)mp.e13[k];
            k1[3 * k + 2] = (uint64_t)mp.e23[k];
            for (int c = 0; c < 3; ++c) v1[3 * k + c] = (int32_t)(3 * k + c);
        }
        t.sync();
        team_sort_pairs(t, sc, sm, k1, v1, k2, v2, 3 * T, bits_for((uint64_t)(mp.E > 0 ? mp.E : 1)));
        for (int64_t q = t.rank(); q < 3 * T; q += t.size()) mp.pos[v1[q]] = (int32_t)q;
        t.sync();
        sc.arena.release(rm);
    }
    prof_mark(t, sc, PH_MP_INCID);
    out = mp;
    return true;
}

// triangle_lb_func (:186-199)
__device__ __forceinline__ float tri_lb(float c12, float c13, float c23)
{
    float lb = 0.0f;
    lb = fminf(lb, __fadd_rn(c12, c13));
    lb = fminf(lb, __fadd_rn(c12, c23));
    lb = fminf(lb, __fadd_rn(c13, c23));
    lb = fminf(lb, __fadd_rn(__fadd_rn(c12, c13), c23));
    return lb;
}

// decrease_triangle_costs_func::min_marginal (:275-280)
__device__ __forceinline__ float min_marginal(float x, float y, float z)
{
    float mm1 = fminf(__fadd_rn(__fadd_rn(x, y), z), fminf(__fadd_rn(x, y), __fadd_rn(x, z)));
    float yz = __fadd_rn(y, z);
    float mm0 = 0.0f < yz ? 0.0f : yz;
    return __fsub_rn(mm1, mm0);
}

// a -+ s * mm in FP64, rounded to float (the reference's expression type).
// Halving is exact (down to the smallest normal float) and a difference of
// two floats rounded to 53 and then to 24 bits equals the one rounded to 24
// bits at once, so the half steps need no conversions.
__device__ __forceinline__ float sub_third(float a, double tm) { return (float)__dsub_rn((double)a, tm); }
__device__ __forceinline__ float add_third(float a, double tm) { return (float)__dadd_rn((double)a, tm); }

// The dual iterations (:350-354) and the lower bound (:201-216).
//
// One iteration: send_messages_to_triplets (:241-269) fused with the six
// min-marginal moves of send_messages_to_edges (:271-348); then each covered
// edge takes the RSUM of its incoming messages.  The bound of the new state
// (CSUM over the negative edge costs, and over triangle_lb_func of the
// triangles' costs) is added up in the same two passes, in registers, so the
// test that ends the loop costs one fold of the team's partial sums and
// there are two team syncs per iteration.  With the bound as two sums of
// their own (two more passes over the data and four more syncs) the
// iterations of a 201,720-edge cube in PD+ mode took 11.7 ms
// (127.8 on the 11 M edge k-NN graph in D mode); this takes 2.8 (93.2).
//
// Bound by memory for large graphs (per triangle 24 B of indices, 24 B of
// costs, 12 B of messages and the gathers of three shares), by the two syncs
// and four dependent loads per pass for small ones.
// min_gain: the loop ends after an iteration that gains less (the reference's
// 1e-3).  Returns the bound of the final state; *lb0, if given, receives the
// bound before the first iteration, *cmin the smallest edge cost.
//
// What holds a pass back is the number of loads that wait for one another, so
// everything a triangle needs by index (its edges, its message slots, its
// costs) is loaded before its first store: with the slots loaded between the
// stores (which may alias them) a pair of triangles waited for eight round
// trips instead of two.
struct TriState {
    int32_t e[3], p[3];  // edges and message slots of the corners 12, 13, 23
    float c[3];          // costs, then with the edges' shares
};

__device__ __forceinline__ void mp_load(const Mp &mp, int64_t k, bool first, TriState &x)
{
    x.e[0] = mp.e12[k];
    x.e[1] = mp.e13[k];
    x.e[2] = mp.e23[k];
#pragma unroll
    for (int q = 0; q < 3; ++q) x.p[q] = mp.pos[3 * k + q];
    x.c[0] = x.c[1] = x.c[2] = 0.0f;
    if (!first) {
        x.c[0] = mp.c12[k];
        x.c[1] = mp.c13[k];
        x.c[2] = mp.c23[k];
    }
}

// the triangle's moves; its bound is added to bt
__device__ __forceinline__ void mp_moves(const Mp &mp, int64_t k, const TriState &x, const float (&s)[3], csum_t &bt)
{
    const double third = 1.0 / 3.0;
    float t12 = __fadd_rn(x.c[0], s[0]), t13 = __fadd_rn(x.c[1], s[1]), t23 = __fadd_rn(x.c[2], s[2]);
    float e12, e13, e23;
    {
        const double tm = __dmul_rn(third, (double)min_marginal(t12, t13, t23));
        t12 = sub_third(t12, tm);
        e12 = add_third(0.0f, tm);
    }
    {
        const float hm = 0.5f * min_marginal(t13, t12, t23);
        t13 = __fsub_rn(t13, hm);
        e13 = __fadd_rn(0.0f, hm);
    }
    {
        const float mm = min_marginal(t23, t12, t13);
        t23 = __fsub_rn(t23, mm);
        e23 = __fadd_rn(0.0f, mm);
    }
    {
        const float hm = 0.5f * min_marginal(t12, t13, t23);
        t12 = __fsub_rn(t12, hm);
        e12 = __fadd_rn(e12, hm);
    }
    {
        const float mm = min_marginal(t13, t12, t23);
        t13 = __fsub_rn(t13, mm);
        e13 = __fadd_rn(e13, mm);
    }
    {
        const float mm = min_marginal(t12, t13, t23);
        t12 = __fsub_rn(t12, mm);
        e12 = __fadd_rn(e12, mm);
    }
    mp.c12[k] = t12;
    mp.c13[k] = t13;
    mp.c23[k] = t23;
    mp.slot[x.p[0]] = e12;
    mp.slot[x.p[1]] = e13;
    mp.slot[x.p[2]] = e23;
    bt = cs_add(bt, tri_lb(t12, t13, t23));
}

template <class Team>
__device__ __noinline__ double mp_run(const Team &t, Scratch &sc, const Mp &state, int num_iter, double min_gain,
                                      float *cmin, double *lb0 = nullptr)
{
    const Mp mp = state;  // pointers in registers
    csum_t be, bt;        // this thread's parts of the bound
    float mn = 3.4e38f;   // ... and its smallest edge cost
    auto edge_bound = [&](float c) {
        be = cs_add(be, c < 0.0f ? c : 0.0f);
        mn = fminf(mn, c);
    };
    // the bound before the first iteration: the triangles' costs are 0
    double lb = team_csum(t, sc, mp.E, [=](int64_t e) -> float {
        const float c = mp.cost[e];
        return c < 0.0f ? c : 0.0f;
    });
    if (lb0) *lb0 = lb;
    double prev = 0.0;
    const int64_t S = t.size();
    for (int it = 0; it < num_iter; ++it) {
        sc.alg_bytes += 4.0 * (double)mp.E + 12.0 * (double)mp.T;
        if (it > 0 && (lb - prev) < min_gain) break;
        prev = lb;
        be = bt = csum_t{0.0, 0.0};
        mn = 3.4e38f;
        // two triangles a thread at a time: their loads and the gathers of
        // the edges' shares are in flight together
        int64_t k = t.rank();
        for (; k + S < mp.T; k += 2 * S) {
            TriState x, y;
            mp_load(mp, k, it == 0, x);
            mp_load(mp, k + S, it == 0, y);
            float sx[3], sy[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                sx[q] = mp.share[x.e[q]];
                sy[q] = mp.share[y.e[q]];
            }
            mp_moves(mp, k, x, sx, bt);
            mp_moves(mp, k + S, y, sy, bt);
        }
        for (; k < mp.T; k += S) {
            TriState x;
            mp_load(mp, k, it == 0, x);
            const float sx[3] = {mp.share[x.e[0]], mp.share[x.e[1]], mp.share[x.e[2]]};
            mp_moves(mp, k, x, sx, bt);
        }
        t.sync();
        // covered edges: c = 0 + RSUM(messages); long runs by a warp
        {
            // four edges a thread at a time: offsets, then the first four
            // messages of each (most edges have no more), then the rest and
            // the stores
            constexpr int U = 4;
            auto first4 = [&](float (&x)[4], int32_t s, int32_t n, int64_t e) {
                if (n > RSUM_THREAD_MAX) n = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = j < n ? mp.slot[s + j] : 0.0f;
                if (n == 0) x[0] = mp.cost[e];
            };
            auto finish = [&](const float (&x)[4], int32_t s, int32_t n, int64_t e) {
                if (n > RSUM_THREAD_MAX) return;
                float c = x[0];
                if (n > 0) {
                    double y[8];
#pragma unroll
                    for (int j = 0; j < 4; ++j) y[j] = __dadd_rn(0.0, (double)x[j]);
                    double sum = __dadd_rn(__dadd_rn(y[0], y[1]), __dadd_rn(y[2], y[3]));
                    if (n > 4) {
#pragma unroll
                        for (int j = 4; j < 8; ++j) y[j] = j < n ? __dadd_rn(0.0, (double)mp.slot[s + j]) : 0.0;
                        sum = __dadd_rn(sum, __dadd_rn(__dadd_rn(y[4], y[5]), __dadd_rn(y[6], y[7])));
                    }
                    c = __fadd_rn(0.0f, (float)sum);
                    mp.cost[e] = c;
                    mp.share[e] = __fdiv_rn(c, (float)n);
                }
                edge_bound(c);
            };
            int64_t e0 = t.rank();
            for (; e0 + (U - 1) * S < mp.E; e0 += U * S) {
                int32_t s[U], n[U];
                float x[U][4];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    s[q] = mp.inc_off[e0 + q * S];
                    n[q] = mp.inc_off[e0 + q * S + 1] - s[q];
                }
#pragma unroll
                for (int q = 0; q < U; ++q) first4(x[q], s[q], n[q], e0 + q * S);
#pragma unroll
                for (int q = 0; q < U; ++q) finish(x[q], s[q], n[q], e0 + q * S);
            }
            for (; e0 < mp.E; e0 += S) {
                const int32_t s = mp.inc_off[e0], n = mp.inc_off[e0 + 1] - s;
                float x[4];
                first4(x, s, n, e0);
                finish(x, s, n, e0);
            }
        }
        // longer runs: up to 64 messages by a thread, more by a warp.  (With a
        // warp for every run of more than 8 its few round trips came in turn
        // for some 80 edges a warp: 0.3 of the 0.5 ms this pass took on the
        // 1M-point k-NN graph's dual with 398,000 such edges.)
        for (int64_t q = t.rank(); q < mp.nlong; q += S) {
            const int32_t e = mp.longe[q];
            const int32_t s = mp.inc_off[e], n = mp.inc_off[e + 1] - s;
            const float c = __fadd_rn(0.0f, rsum_upto64(n, [=](int x) { return mp.slot[s + x]; }));
            mp.cost[e] = c;
            mp.share[e] = __fdiv_rn(c, (float)n);
            edge_bound(c);
        }
        for (int64_t q = team_warp(t); q < mp.nhuge; q += team_nwarps(t)) {
            const int32_t e = mp.longe[mp.longe_cap - 1 - q];
            const int32_t s = mp.inc_off[e], n = mp.inc_off[e + 1] - s;
            const float c = __fadd_rn(0.0f, rsum_warp(n, [=](int64_t x) { return mp.slot[s + x]; }));
            if (lane_id() == 0) {
                mp.cost[e] = c;
                mp.share[e] = __fdiv_rn(c, (float)n);
                edge_bound(c);
            }
        }
        const csum2_t b = team_csum_fold(t, sc, be, bt, mn);
        lb = b.a + b.b;
        *cmin = b.m;
        sc.alg_bytes += 84.0 * (double)mp.T + 12.0 * (double)mp.E;
    }
    return lb;
}

// dual_update_cycle_length (src/dual_solver.cu:7-35).  On success the graph
// in the top slot is replaced by the reparametrised one (without chords, its
// costs are updated where they lie).
template <class Team>
__device__ double dual_update_cycle_length(const Team &t, Scratch &sc, char *sm, Graph &A, int c, int num_iter,
                                           float tri_factor, float tol, int64_t *num_tri, bool *failed,
                                           bool *no_cycles)
{
    uint64_t m = sc.arena.mark();
    TriBuf tb;
    prof_mark(t, sc, PH_OTHER);
    conflicted_cycles(t, sc, sm, A, c, tri_factor, tol, false, tb);
    prof_mark(t, sc, PH_CYC_SEARCH);
    *failed = !sc.arena.ok();
    if (*failed) {
        sc.arena.release(m);
        return 0.0;
    }
    *num_tri = tb.count;
    *no_cycles = tb.none != 0;
    if (tb.count == 0) {
        sc.arena.release(m);
        return graph_lb(t, sc, A);
    }
    Mp mp;
    if (!mp_build(t, sc, sm, A, tb, mp)) {
        *failed = true;
        sc.arena.release(m);
        return 0.0;
    }
    prof_mark(t, sc, PH_MP_BUILD);
    float cmin = unknown_cost();
    const double fin = mp_run(t, sc, mp, num_iter, 1e-3, &cmin);
    prof_mark(t, sc, PH_MP_ITER);
    // dims of the edge list: a chord joins two ends of edges, so the largest
    // column stays what it was
    Graph g = A;
    g.rows = uread(&mp.row[mp.E - 1]) + 1;
    g.cols = A.ecols;
    g.cmin = cmin;
    *failed = false;
    if (!mp.inplace) {
        g.row = mp.row;
        g.col = mp.col;
        g.cost = mp.cost;
        g.n = mp.E;
        g = graph_commit(t, sc, g);
        *failed = !sc.arena.ok();
    }
    prof_mark(t, sc, PH_DUAL_COMMIT);
    if (!*failed) A = g;
    sc.arena.release(m);
    return fin;
}

// dual_solver (src/dual_solver.cu:37-63); an arena overflow plays the role of
// the reference's bad_alloc: the trivial bound of the current graph is
// returned and the graph keeps its last committed state.
template <class Team>
__device__ double dual_solver(const Team &t, Scratch &sc, char *sm, Graph &A, int max_len, int num_iter,
                              float tri_factor, int num_outer, float tol, int64_t *num_tri_last, int *oom)
{
    if (num_tri_last) *num_tri_last = 0;
    if (max_len < 3 || num_iter == 0 || num_outer == 0) return graph_lb(t, sc, A);
    double prev = 0.0, fin = 0.0;
    int64_t nt = 0;
    for (int o = 0; o < num_outer; ++o) {
        for (int c = 3; c <= max_len; ++c) {
            bool failed = false, none = false;
            fin = dual_update_cycle_length(t, sc, sm, A, c, num_iter, tri_factor, tol, &nt, &failed, &none);
            if (failed) {
                sc.arena.failed = 0;
                if (oom) *oom = 1;
                return graph_lb(t, sc, A);
            }
            // the graph is unchanged and no repulsive edge can close a cycle:
            // the longer cycle lengths find nothing either (nt == 0 ends the
            // outer loop too)
            if (none) break;
        }
        if (nt == 0 || (o > 0 && (fin - prev) < 1e-3)) break;
        prev = fin;
    }
    if (num_tri_last) *num_tri_last = nt;
    return fin;
}

}  // namespace rama
