"""Waits that run out: the solve reports GSLAM_ERR_DEVICE_TIMEOUT, every block leaves its kernel, and
the handle solves as before afterwards."""
import importlib

import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def synth():
    return importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth")


def _random_closures(synth, n, k):
    cg = synth.city_grid(n, seed=n)
    rng = np.random.default_rng(n)
    i, j = rng.integers(0, n, k * n).astype(np.uint32), rng.integers(0, n, k * n).astype(np.uint32)
    i, j = i[i != j], j[i != j]
    rel = rng.normal(size=(len(i), 3)) * 0.1
    return (cg.init, np.concatenate([cg.edge_i, i]), np.concatenate([cg.edge_j, j]), np.concatenate([cg.meas, rel]),
            np.concatenate([cg.log_w, np.zeros_like(rel)]))


@pytest.mark.parametrize("absent", [0, 1, 147])
def test_absent_cta_of_a_graph_with_long_halos(pkg, synth, absent):
    """12,000 poses with 4 random closures each: a CTA of the grid-wide resident solver reads more rows
    of others than it has threads, so its warps poll them while others are still at the first sums;
    all of them must leave by the same decision."""
    opts = dict(tol=0.0, max_iter=20, barrier_timeout_ms=20.0)
    with pkg.PoseGraph.from_se2(*_random_closures(synth, 12_000, 4), 0.1, **opts) as g:
        g.linearise()
        g.assemble()
        assert g.solve().iterations == 20
        ref = g.dx()
        for _ in range(3):
            g.set_opts(test_absent_cta=absent, **opts)
            with pytest.raises(pkg.abi.GslamError) as e:
                g.solve()
            assert e.value.code == pkg.abi.ERR_DEVICE_TIMEOUT
            g.set_opts(**opts)
            assert g.solve().iterations == 20
            assert_bitwise(g.dx(), ref, "the solve after a timeout")


@pytest.mark.parametrize("n, prec", [(300, 0), (2000, 0), (7000, 0), (9000, 0), (9000, 1), (9000, 2)],
                         ids=["one-cta", "cluster", "cluster-16", "resident", "mixed", "one-reduction"])
def test_limit_shorter_than_any_wait(pkg, synth, n, prec):
    """A limit of about one clock cycle: whichever waits it ends (the copy of the matrix into shared
    memory among them), the solve says so or is right, and the next solve on the SMs is right."""
    cg = synth.city_grid(n, seed=n)
    opts = dict(tol=0.0, max_iter=20, inner_tol=0.0, inner_max_iter=20, precision=prec)
    with pkg.PoseGraph.from_se2(cg.init, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, 0.1, **opts) as g:
        g.linearise()
        g.assemble()
        assert g.solve().iterations == 20
        ref = g.dx()
        for _ in range(5):
            g.set_opts(barrier_timeout_ms=1e-6, **opts)
            try:
                assert g.solve().iterations == 20
                assert_bitwise(g.dx(), ref, "a solve that no limit ended")
            except pkg.abi.GslamError as e:
                assert e.code == pkg.abi.ERR_DEVICE_TIMEOUT
            g.set_opts(**opts)
            assert g.solve().iterations == 20
            assert_bitwise(g.dx(), ref, "the solve after it")


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_limit_shorter_than_any_wait_in_a_batch(pkg, synth, prec):
    graphs = [synth.city_grid(n, seed=n) for n in (300, 2000, 9000)]
    opts = dict(tol=0.0, max_iter=20, inner_tol=0.0, inner_max_iter=20, precision=prec)
    b = pkg.PoseGraphBatch.from_se2_list(graphs, 0.1, **opts)
    b.round_all()
    ref = b.poses
    for _ in range(5):
        b.poses = b.init_poses
        b.set_opts(barrier_timeout_ms=1e-6, **opts)
        try:
            b.round_all()
            assert_bitwise(b.poses, ref, "a round that no limit ended")
        except pkg.abi.GslamError as e:
            assert e.code == pkg.abi.ERR_DEVICE_TIMEOUT
        b.poses = b.init_poses
        b.set_opts(**opts)
        b.round_all()
        assert_bitwise(b.poses, ref, "the round after it")
    b.close()
