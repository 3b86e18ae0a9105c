"""The autotuner of the launch parameters (rama_b200.autotune): its
decisions from timing tables and its cache on the CPU; on the GPU, that the
tuning it chooses leaves every result unchanged."""
import json

import numpy as np
import pytest

from rama_b200 import autotune


def test_pick_fastest_prefers_the_first_of_equal_times():
    assert autotune.pick_fastest({4: 2.0, 8: 1.0, 16: 1.0}) == 8
    assert autotune.pick_fastest({1: 3.0}) == 1


def test_crossover_between_last_loss_and_the_run_of_wins():
    sizes = [1000, 4000, 16000, 64000]
    # the larger team loses at 1k and 4k, wins from 16k on: switch at sqrt(4k * 16k)
    assert autotune.crossover(sizes, [1, 2, 9, 30], [3, 4, 6, 10], default=7) == 8000
    # a win that does not last: the unbroken run starts at 64k
    assert autotune.crossover(sizes, [1, 5, 9, 30], [3, 4, 12, 10], default=7) == int(round((16000 * 64000) ** 0.5))
    assert autotune.crossover(sizes, [5, 5, 5, 5], [1, 1, 1, 1], default=7) == 1000
    assert autotune.crossover(sizes, [1, 1, 1, 1], [5, 5, 5, 5], default=7) == 64001


def test_threshold_keeps_the_automatic_line_where_it_agrees():
    from rama_b200 import _lib

    sizes = [1000, 4000, 16000, 64000]
    cta, clu = [1, 2, 9, 30], [3, 4, 6, 10]  # the switch lies between 4,000 and 16,000
    assert autotune.threshold(sizes, cta, clu, 5000) == _lib.MIN_AUTO
    assert autotune.threshold(sizes, cta, clu, 16000) == _lib.MIN_AUTO
    assert autotune.threshold(sizes, cta, clu, 4000) == 8000
    assert autotune.threshold(sizes, cta, clu, 16001) == 8000


def test_cache_round_trip(tmp_path):
    p = str(tmp_path / "t.json")
    assert autotune.load_cache(p) == {}
    autotune.save_cache("B200|148|abc", {"tuning": {"cluster_ctas": 8}}, p)
    autotune.save_cache("other|1|x", {"tuning": {"cluster_ctas": 4}}, p)
    d = autotune.load_cache(p)
    assert d["B200|148|abc"]["tuning"]["cluster_ctas"] == 8 and len(d) == 2
    with open(p, "w") as f:
        f.write("not json")
    assert autotune.load_cache(p) == {}


def test_automatic_values_are_those_of_the_header():
    import os
    import re

    from rama_b200 import _lib

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with open(os.path.join(root, "include", "rama_b200.h")) as f:
        defs = dict(re.findall(r"#define (RAMA_\w*AUTO\w*) \(?(-?\d+)\)?", f.read()))
    assert {k: int(v) for k, v in defs.items()} == {
        "RAMA_CLUSTER_CTAS_AUTO": _lib.CLUSTER_CTAS_AUTO, "RAMA_MIN_AUTO": _lib.MIN_AUTO,
        "RAMA_AUTO_CLUSTER_MIN": _lib.AUTO_CLUSTER_MIN, "RAMA_AUTO_GRID_MIN": _lib.AUTO_GRID_MIN}
    t = _lib.RamaTuning(single_grid_min=_lib.MIN_AUTO)
    assert t.grid_min() == _lib.AUTO_GRID_MIN
    t.single_grid_min = 7
    assert t.grid_min() == 7


@pytest.mark.gpu
def test_thresholds_mean_what_they_say(oracle):
    """A caller's thresholds hold in every mode; the automatic ones count twice
    without a dual.  Any cluster size a caller asks for is accepted, 8 among
    them, and changes no result."""
    from rama_b200 import _lib, instances
    from rama_b200.solver import Solver

    g = instances.delaunay(1800, np.random.default_rng(6))  # 5,4xx edges: between the automatic line and its double
    n = len(g[2])
    assert _lib.AUTO_CLUSTER_MIN < n < 2 * _lib.AUTO_CLUSTER_MIN
    s = Solver(0)
    auto = s.handle.tuning()
    assert (auto.cluster_ctas, auto.single_cluster_min, auto.single_grid_min) == (0, -1, -1)
    for low, high, teams in ((-1, -1, {"P": 1, "PD": 3, "D": 3}), (n, -1, {"P": 3, "PD": 3}),
                             (n + 1, n + 1, {"P": 1, "PD": 1}), (0, n, {"P": 2, "PD": 2}),
                             (4000, 100000, {"P": 3, "PD": 3})):
        t = s.handle.tuning()
        t.single_cluster_min, t.single_grid_min = low, high
        s.handle.set_tuning(t)
        for mode, team in teams.items():
            s.solve(*g, mode=mode)
            assert s.stats().team == team
    want = oracle.solve(*g, "PD")[:2]
    for size in (0, 2, 4, 8, 16):
        t = s.handle.tuning()
        t.cluster_ctas = size
        s.handle.set_tuning(t)
        assert s.handle.tuning().cluster_ctas == size
        lab, lb, _ = s.solve(*g, mode="PD", team=3)
        assert np.array_equal(lab, want[0]) and lb == want[1]
    t.single_grid_min = -2
    with pytest.raises(_lib.RamaError):
        s.handle.set_tuning(t)


@pytest.mark.gpu
def test_tuned_parameters_give_identical_results(tmp_path):
    """A quick tuning run (which itself checks every trial against the first
    result of its instance), then solves with the default and the tuned
    parameters on every team: identical labels and bounds."""
    from rama_b200 import instances
    from rama_b200.solver import Solver

    entry = autotune.tune(0, budget_s=20.0, quick=True)
    json.dumps(entry, default=str)
    s = Solver(0)
    t = s.handle.tuning()
    for k in autotune.KNOBS:
        setattr(t, k, entry["tuning"][k])
    rng = np.random.default_rng(3)
    graphs = [instances.delaunay(n, rng) for n in (400, 3000, 12000)]
    for g in graphs:
        want = [Solver(0).solve(*g, mode="PD", team=tm)[:2] for tm in (1, 3, 2)]
        s.handle.set_tuning(t)
        got = [s.solve(*g, mode="PD", team=tm)[:2] for tm in (0, 1, 3, 2)]
        for lab, lb in want[1:] + got:
            assert np.array_equal(lab, want[0][0]) and lb == want[0][1]


@pytest.mark.gpu
def test_set_tuning_rejects_values_out_of_range():
    from rama_b200 import _lib
    from rama_b200.solver import Solver

    s = Solver(0)
    t = s.handle.tuning()
    t.cluster_ctas = 3
    with pytest.raises(_lib.RamaError):
        s.handle.set_tuning(t)
    t = s.handle.tuning()
    t.grid_ctas_per_sm = 0
    with pytest.raises(_lib.RamaError):
        s.handle.set_tuning(t)
    t = s.handle.tuning()
    t.cta_threads = 300
    with pytest.raises(_lib.RamaError):
        s.handle.set_tuning(t)


@pytest.mark.gpu
def test_small_cta_kernel_gives_the_same_batch_results():
    """A batch without cluster instances on CTAs of 256 threads (three per SM)
    and on CTAs of 512: the same labels and bounds."""
    from rama_b200 import instances
    from rama_b200.solver import Solver

    b = instances.delaunay_batch(count=40, nmin=300, nmax=6000, seed=17)
    s = Solver(0)
    want, _, rc = s.solve_batch(b, mode="PD")
    assert rc == 0
    t = s.handle.tuning()
    t.cta_threads, t.batch_cluster_min = 256, 1 << 40
    s.handle.set_tuning(t)
    got, _, rc = s.solve_batch(b, mode="PD")
    assert rc == 0
    for (lab, lb), (glab, glb) in zip(want, got):
        assert np.array_equal(lab, glab) and lb == glb


@pytest.mark.gpu
def test_one_instance_runs_on_the_kernel_for_one(oracle):
    """The CTA size is about batches: a single solve keeps the kernel that has
    an SM to itself."""
    from rama_b200 import instances
    from rama_b200.solver import Solver

    g = instances.delaunay(400, np.random.default_rng(5))
    b = instances.delaunay_batch(count=2, nmin=300, nmax=500, seed=18)
    want = oracle.solve(*g, "PD")[:2]
    s = Solver(0)
    for threads, kernel in ((512, "k_solve_cta"), (256, "k_solve_cta_small")):
        t = s.handle.tuning()
        t.cta_threads = threads
        s.handle.set_tuning(t)
        lab, lb, _ = s.solve(*g, mode="PD")
        assert s.handle.solve_kernel() == "k_solve_cta_alone"
        assert np.array_equal(lab, want[0]) and lb == want[1]
        _, _, rc = s.solve_batch(b, mode="PD")
        assert rc == 0 and s.handle.solve_kernel() == kernel
