"""Sizes at which a kernel changes its way through the data, against the CPU
oracle (bit for bit: every sum follows one order of additions, or carries
enough bits that the order does not show): buckets of 64, 256 and 4,096
entries, runs of 4, 8 and 64 messages or parallel edges, tiles of 2,048
elements, and the 16-byte groups of the text parser."""
import ctypes as C

import numpy as np
import pytest

from rama_b200 import instances

pytestmark = pytest.mark.gpu


def same_as_oracle(solver, oracle, i, j, c, mode, team, **kw):
    olab, olb, _ = oracle.solve(i, j, c, mode, **kw)
    glab, glb, _ = solver.solve(i, j, c, mode=mode, team=team, **kw)
    assert glb == olb
    assert np.array_equal(glab, olab)


def book(pages, seed):
    """A repulsive edge and `pages` triangles on it; two of these joined by an edge."""
    rng = np.random.default_rng(seed)
    k = np.arange(2, 2 + pages, dtype=np.int32)
    i = np.concatenate([[0], np.zeros(pages), np.ones(pages)]).astype(np.int32)
    j = np.concatenate([[1], k, k]).astype(np.int32)
    c = np.concatenate([[-2.0 * pages], rng.uniform(0.1, 3.0, 2 * pages)]).astype(np.float32)
    m = pages + 2
    return (np.concatenate([i, i + m, [0]]).astype(np.int32), np.concatenate([j, j + m, [m]]).astype(np.int32),
            np.concatenate([c, c, [0.5]]).astype(np.float32))


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("pages", (1, 4, 5, 8, 9, 32, 33, 64, 65, 256, 257, 4097))
def test_messages_of_one_edge(solver, oracle, pages, team):
    same_as_oracle(solver, oracle, *book(pages, pages), "D", team)
    same_as_oracle(solver, oracle, *book(pages, pages), "PD", team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("degree", (63, 64, 65, 256, 257, 4096, 4097))
def test_neighbours_of_one_vertex(solver, oracle, degree, team):
    """A hub with `degree` neighbours on a ring with chords."""
    rng = np.random.default_rng(degree)
    k = np.arange(1, degree + 1, dtype=np.int32)
    i = np.concatenate([np.zeros(degree, np.int32), k[:-1], k[:-2]])
    j = np.concatenate([k, k[1:], k[2:]])
    c = rng.normal(0.4, 1.0, len(i)).astype(np.float32)
    for mode in ("P", "PD+"):
        same_as_oracle(solver, oracle, i, j, c, mode, team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("gap", (1, 11))
def test_hub_among_unused_ids(solver, oracle, gap, team):
    """More attractive neighbours than the list sort takes, with and without
    gaps in the node ids."""
    degree = 4200
    rng = np.random.default_rng(gap)
    k = np.arange(1, degree + 1, dtype=np.int32)
    i = np.concatenate([np.zeros(degree, np.int32), k[:-1]]) * gap
    j = np.concatenate([k, k[1:]]) * gap
    c = np.concatenate([rng.uniform(0.1, 1.0, degree), rng.normal(-0.2, 1.0, degree - 1)]).astype(np.float32)
    for mode in ("PD", "D"):
        same_as_oracle(solver, oracle, i, j, c, mode, team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("copies", (2, 3, 8, 33, 64, 65, 200))
def test_parallel_edges(solver, oracle, copies, team):
    """Every edge `copies` times: neighbour lists with repeated entries and
    equal triangles."""
    i, j, _ = instances.random_graph(24, 4, seed=3)
    order = np.random.default_rng(copies).permutation(len(i) * copies)
    c = np.random.default_rng(copies + 1).normal(0.2, 1.0, len(i) * copies).astype(np.float32)
    same_as_oracle(solver, oracle, np.tile(i, copies)[order], np.tile(j, copies)[order], c, "D", team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("nodes", (2, 3, 511, 513, 2047, 2048, 2049, 4097))
def test_tiles_of_nodes_and_edges(solver, oracle, nodes, team):
    """A path with as many nodes (and one edge less), costs of both signs."""
    k = np.arange(nodes - 1, dtype=np.int32)
    c = np.random.default_rng(nodes).normal(0.3, 1.0, nodes - 1).astype(np.float32)
    c[::7] = 0.0
    c[::11] = -0.0
    for mode in ("P", "PD"):
        same_as_oracle(solver, oracle, k, k + 1, c, mode, team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("stride", (2, 3, 5, 8))
@pytest.mark.parametrize("edges", (2, 700, 30000))
def test_more_nodes_than_edges(solver, oracle, edges, stride, team):
    """Edges that share no node, node ids with gaps between them: lists of
    vertices that reach beyond what the sort of the edges took of the
    workspace."""
    k = np.random.default_rng(edges + stride).permutation(edges).astype(np.int32) * stride
    c = np.random.default_rng(stride).normal(0.1, 1.0, edges).astype(np.float32)
    for mode in ("P", "PD", "PD+", "D"):
        same_as_oracle(solver, oracle, k, k + 1, c, mode, team)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("factor", (0.01, 0.3, 1.0, 5.0))
def test_truncated_cycles(solver, oracle, factor, team):
    """Few emissions an expansion, and some with more than the histogram's
    1,023 (a hub next to every vertex)."""
    rng = np.random.default_rng(8)
    n = 1300
    k = np.arange(2, n, dtype=np.int32)
    i = np.concatenate([[0], np.zeros(n - 2), np.ones(n - 2), k[:-1]]).astype(np.int32)
    j = np.concatenate([[1], k, k, k[1:]]).astype(np.int32)
    c = np.concatenate([[-9.0], rng.uniform(0.1, 2.0, 2 * (n - 2)), rng.normal(-0.5, 0.5, n - 3)]).astype(np.float32)
    same_as_oracle(solver, oracle, i, j, c, "D", team, tri_memory_factor=factor)


@pytest.mark.parametrize("team", (1, 2, 3))
@pytest.mark.parametrize("pages", (1, 5, 300))
def test_no_room_for_any_triangle(solver, oracle, pages, team):
    """A budget of no triangle, and one that the first cycle length fills."""
    i, j, c = book(pages, pages)
    for mode in ("PD", "PD+", "D"):
        for factor in (0.0, 0.1, 0.5 * pages, float(pages)):
            same_as_oracle(solver, oracle, i, j, c, mode, team, tri_memory_factor=factor)


@pytest.mark.parametrize("team", (1, 2))
@pytest.mark.parametrize("seed", range(6))
def test_cycles_beside_self_loops(solver, oracle, seed, team):
    """The cycle search alone takes graphs with self-loops, whose vertices
    stand twice in their own lists of neighbours."""
    i, j, c = instances.random_graph(60, 6, seed=seed)
    k = np.arange(60, dtype=np.int32)
    loops = np.random.default_rng(seed).uniform(0.1, 1.0, 60).astype(np.float32)
    G = oracle.Graph.from_edges(np.concatenate([i, k]), np.concatenate([j, k]), np.concatenate([c, loops]))
    row, col, cost = G.arrays()
    for length in (3, 4, 5):
        want, raw = oracle.conflicted_cycles(G, length, 5.0)
        got, graw = solver.step_cycles(row, col, cost, *G.dims, length, 5.0, team=team)
        assert graw == raw and np.array_equal(got, want)


@pytest.fixture(scope="module")
def by_kernel():
    """A solver and a call for each kernel that one small instance alone, on
    an untuned handle, does not run on."""
    from rama_b200.solver import Solver

    handles = {}

    def tuned(**kw):
        s = Solver(0)
        t = s.handle.tuning()
        for k, v in kw.items():
            setattr(t, k, v)
        s.handle.set_tuning(t)
        return s

    def run(kernel, i, j, c, mode, **kw):
        if kernel not in handles:
            handles[kernel] = tuned(**{"k_solve_grid": {"grid_small_max": 0},
                                       "k_solve_cta_small": {"cta_threads": 256}}.get(kernel, {}))
        s = handles[kernel]
        if kernel == "k_solve_grid":
            lab, lb, _ = s.solve(i, j, c, mode=mode, team=2, **kw)
            got = [(lab, lb)]
        else:  # the instance twice
            nodes = int(max(i.max(), j.max())) + 1
            got, _, rc = s.solve_batch(_batch([(i, j, c)] * 2, [nodes] * 2), mode=mode,
                                       team=3 if kernel == "k_solve_mixed" else 1, **kw)
            assert rc == 0
        assert s.handle.solve_kernel() == kernel
        return got

    return run


def _shapes():
    def hub(degree):
        rng = np.random.default_rng(degree)
        k = np.arange(1, degree + 1, dtype=np.int32)
        i = np.concatenate([np.zeros(degree, np.int32), k[:-1], k[:-2]])
        return i, np.concatenate([k, k[1:], k[2:]]), rng.normal(0.4, 1.0, len(i)).astype(np.float32)

    def copies(m):
        i, j, _ = instances.random_graph(24, 4, seed=3)
        c = np.random.default_rng(m).normal(0.2, 1.0, len(i) * m).astype(np.float32)
        return np.tile(i, m), np.tile(j, m), c

    def path(nodes):
        k = np.arange(nodes - 1, dtype=np.int32)
        return k, k + 1, np.random.default_rng(nodes).normal(0.3, 1.0, nodes - 1).astype(np.float32)

    def pairs(edges):
        k = np.arange(edges, dtype=np.int32) * 5
        return k, k + 1, np.random.default_rng(edges).normal(0.1, 1.0, edges).astype(np.float32)

    every = ("P", "PD+", "D")
    out = [("messages%d" % n, book(n, n), every, {}) for n in (4, 5, 8, 9, 64, 65, 257, 4097)]
    out += [("neighbours%d" % n, hub(n), every, {}) for n in (64, 65, 256, 257, 4096, 4097)]
    out += [("copies%d" % n, copies(n), ("D",), {}) for n in (2, 33, 65)]  # (contractions of these go bad)
    out += [("path%d" % n, path(n), every, {}) for n in (2, 511, 2048, 2049)]
    out += [("pairs%d" % n, pairs(n), every, {}) for n in (2, 3000)]
    out += [("budget%g" % f, book(300, 1), every, {"tri_memory_factor": f}) for f in (0.0, 0.1, 100.0, 300.0)]
    return out


SHAPES = _shapes()


@pytest.mark.parametrize("shape", SHAPES, ids=[s[0] for s in SHAPES])
@pytest.mark.parametrize("kernel", ("k_solve_grid", "k_solve_cta", "k_solve_cta_small", "k_solve_mixed"))
def test_shapes_on_the_other_kernels(by_kernel, oracle, kernel, shape):
    """The sizes above on the kernels of two CTAs per SM and of batches."""
    _, (i, j, c), modes, kw = shape
    for mode in modes:
        olab, olb, _ = oracle.solve(i, j, c, mode, **kw)
        for lab, lb in by_kernel(kernel, i, j, c, mode, **kw):
            assert lb == olb and np.array_equal(lab, olab)


@pytest.mark.parametrize("mode", ("P", "PD"))
def test_several_tiles_a_cta(solver, by_kernel, oracle, mode):
    """More edges than a tile for each of the 148 or 296 CTAs of a grid."""
    i, j, c = instances.grid3d_longrange(64, 64, 32, seed=7)
    olab, olb, _ = oracle.solve(i, j, c, mode)
    lab, lb, _ = solver.solve(i, j, c, mode=mode, team=2)
    assert solver.handle.solve_kernel() == "k_solve_grid_alone"
    assert lb == olb and np.array_equal(lab, olab)
    for lab, lb in by_kernel("k_solve_grid", i, j, c, mode):
        assert lb == olb and np.array_equal(lab, olab)


@pytest.mark.parametrize("mode", ("P", "PD"))
def test_clusters_of_every_size(solver, oracle, mode):
    """Batches of few, some and many instances for clusters, and one alone on
    either side of the sizes at which the team changes."""
    rng = np.random.default_rng(4)
    graphs = {n: instances.delaunay(n, rng) for n in (1200, 1500, 2700, 4200, 5200)}
    want = {n: oracle.solve(*g, mode)[:2] for n, g in graphs.items()}
    for n, g in graphs.items():
        lab, lb, _ = solver.solve(*g, mode=mode)
        assert lb == want[n][1] and np.array_equal(lab, want[n][0])
    for count in (2, 14, 40):
        sizes = [(4200, 5200, 1200)[k % 3] for k in range(count)]
        out, status, rc = solver.solve_batch(_batch([graphs[n] for n in sizes], sizes), mode=mode)
        assert rc == 0
        for n, (lab, lb) in zip(sizes, out):
            assert lb == want[n][1] and np.array_equal(lab, want[n][0])


def _batch(graphs, nodes):
    class B:
        pass

    b = B()
    b.count = len(graphs)
    b.i, b.j, b.c = (np.concatenate([g[k] for g in graphs]) for k in range(3))
    b.edge_offsets = np.cumsum([0] + [len(g[2]) for g in graphs]).astype(np.int64)
    b.node_counts = np.array(nodes, np.int64)
    return b


@pytest.mark.parametrize("head", (b"MULTICUT\n", b"MULTICUT\r\n", b"MULTICUT\n\n  "))
@pytest.mark.parametrize("shift", range(0, 17))
def test_text_at_any_alignment(solver, head, shift):
    """Texts whose length and device address lie anywhere within the parser's
    16-byte groups."""
    import torch

    from rama_b200 import _lib

    rows = [(k, k + 1, k * 0.25 - 3.0) for k in range(40 + shift)]
    text = head + b"".join(b"%d %d %s\n" % (a, b, repr(x).encode()) for a, b, x in rows) + b" " * (shift % 3)
    want = [np.array(x) for x in zip(*rows)]
    for got in (solver.parse_multicut(text), solver.parse_multicut(text[:-1 - shift % 3]),
                solver.parse_multicut(bytearray(text))):
        assert all(np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want))
    d = torch.zeros(len(text) + 64, dtype=torch.uint8, device="cuda")
    d[shift:shift + len(text)] = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    out = [torch.empty(200, dtype=t, device="cuda") for t in (torch.int32, torch.int32, torch.float32)]
    n = C.c_int64(0)
    _lib.check(_lib.load().rama_parse_multicut(solver.handle.h, C.c_void_p(d.data_ptr() + shift), len(text),
                                               *[C.c_void_p(x.data_ptr()) for x in out], 200, C.byref(n),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert n.value == len(rows)
    assert all(np.array_equal(g[:n.value].cpu().numpy(), w) for g, w in zip(out, want))
