"""Which solver a graph is given: the one inside a thread-block cluster (pcg_cluster.cu) or the
grid-wide one, by their estimated times. Graphs with long rows, whose values do not fit the
cluster's shared memory, or with closures to random poses, whose halo rows are sent one by one,
ran up to 3.4 times slower in a cluster than on the whole GPU.

test_absent_cta beyond every grid is no CTA at all and keeps a handle off the cluster solver.
Where the choice is right, the chosen solver takes at most 1.3 times as long as the grid-wide one
(device times of the same solve, the best of six; a wrong choice took 1.8 times and more)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = dict(test_absent_cta=1 << 20)
ITS = 200


@pytest.fixture(scope="module")
def synth():
    return importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth")


def _random_closures(synth, n, k, seed=1):
    """A walk with k closures per pose to random poses: (init, i, j, meas, log_w) and the walk."""
    cg = synth.city_grid(n, seed=seed)
    rng = np.random.default_rng(seed)
    i, j = rng.integers(0, n, k * n).astype(np.uint32), rng.integers(0, n, k * n).astype(np.uint32)
    i, j = i[i != j], j[i != j]
    rel = rng.normal(size=(len(i), 3)) * 0.1
    cg.edge_i, cg.edge_j = np.concatenate([cg.edge_i, i]), np.concatenate([cg.edge_j, j])
    cg.meas, cg.log_w = np.concatenate([cg.meas, rel]), np.concatenate([cg.log_w, np.zeros_like(rel)])
    return cg


def _single_us(make):
    g = make()
    g.linearise()
    g.assemble()
    t = [g.solve().solve_ms for _ in range(6)]
    g.close()
    return min(t)


@pytest.mark.parametrize("kind", ["random closures", "landmark cliques"])
def test_single_graph_avoids_a_slow_cluster(pkg, synth, kind):
    opts = dict(tol=0.0, max_iter=ITS)
    if kind == "landmark cliques":
        log = synth.landmark_log(7120, seed=3, density=1e-2, max_obs=20)
        make = lambda **o: pkg.PoseGraph.from_log(log, 0.1, **opts, **o)  # noqa: E731
    else:
        cg = _random_closures(synth, 6000, 8)
        make = lambda **o: pkg.PoseGraph.from_se2(cg.init, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, 0.1,  # noqa: E731
                                                  **opts, **o)
    assert _single_us(make) <= 1.3 * _single_us(lambda: make(**GRID))


def _batch(pkg, graphs, prec, rounds, its_cap=ITS, **opts):
    """(best solve ms, pose steps of every graph after one round, iterations) of a batch."""
    b = pkg.PoseGraphBatch.from_se2_list(graphs, 0.1, tol=0.0, max_iter=its_cap, inner_tol=0.0,
                                         inner_max_iter=its_cap, precision=prec, **opts)
    t, dx, its = [], None, None
    for _ in range(rounds):
        b.poses = b.init_poses
        st = b.round_all()
        t.append(st[0].solve_ms)
        its = [s.iterations for s in st]
        dx = [b.graph_poses(q, b.poses - b.init_poses) for q in range(len(graphs))]
    b.close()
    return min(t), dx, its


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_batch_with_a_graph_too_large_is_not_split(pkg, synth, prec):
    """The other graphs in clusters and then the large one alone took 1.1 to 1.25 times as long as all
    of them grid-wide."""
    graphs = [synth.city_grid(25_000, seed=0)] + [synth.city_grid(1000, seed=1 + s) for s in range(4)]
    for part, expected in ((graphs, False), (graphs[1:], True)):
        b = pkg.PoseGraphBatch.from_se2_list(part, 0.1, precision=prec)
        assert b.in_clusters is expected
        b.close()


def test_batch_avoids_slow_clusters(pkg, synth):
    graphs = [_random_closures(synth, 15_000, 2, seed=s) for s in range(2)]
    assert _batch(pkg, graphs, 0, 8)[0] <= 1.3 * _batch(pkg, graphs, 0, 8, **GRID)[0]


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_batch_in_clusters_takes_the_grid_wide_iterates(pkg, synth, prec):
    """Clusters of 1 to 16 CTAs, with one and two rows per thread, are chosen here (the solve takes
    about half as long) and take the grid-wide solver's steps: after 60 iterations the two
    orders of the dot products' sums differ by far less than 1e-9; in FP32 they round a
    coefficient differently now and then (1e-3 allowed)."""
    graphs = [synth.city_grid(n, seed=n) for n in (37, 320, 330, 640, 650, 5000, 10240, 10250, 20480)]
    ta, xa, ia = _batch(pkg, graphs, prec, 4, 60)
    tb, xb, ib = _batch(pkg, graphs, prec, 4, 60, **GRID)
    assert ta <= 0.7 * tb
    assert ia == ib
    for a, b in zip(xa, xb):
        assert np.linalg.norm(a - b) <= (1e-9 if prec == 0 else 1e-3) * np.linalg.norm(b) + 1e-12
