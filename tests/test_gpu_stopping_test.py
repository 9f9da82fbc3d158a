"""The stopping test ||r|| < tol ||xi|| at tolerances that no residual is below: with tol <= 0 (a
program's "run all iterations") every solver takes exactly max_iter iterations, the ones that
compare squares (cluster and grid-wide resident) like the streaming one that compares roots."""
import importlib

import pytest

pytestmark = pytest.mark.gpu

STOP_MAXIT = 1
ITS = 25


@pytest.fixture(scope="module")
def synth():
    return importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth")


@pytest.mark.parametrize("tol", [0.0, -0.0, -1e-300, -1.0, -1e200])
@pytest.mark.parametrize("n", [300, 2000, 9000])    # one CTA, a cluster, grid-wide
def test_single_graph_never_stops_early(pkg, synth, n, tol):
    cg = synth.city_grid(n, seed=n)
    for o in ({}, dict(disable_resident=1)):
        with pkg.PoseGraph.from_se2(cg.init, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, 0.1, tol=tol, max_iter=ITS,
                                    **o) as g:
            st = g.round()
            assert (st.iterations, st.reason) == (ITS, STOP_MAXIT), o


@pytest.mark.parametrize("tol", [0.0, -1.0])
def test_batch_never_stops_early(pkg, synth, tol):
    graphs = [synth.city_grid(n, seed=n) for n in (300, 2000, 9000)]
    for o in ({}, dict(disable_resident=1)):
        b = pkg.PoseGraphBatch.from_se2_list(graphs, 0.1, tol=tol, max_iter=ITS, **o)
        assert [(s.iterations, s.reason) for s in b.round_all()] == [(ITS, STOP_MAXIT)] * 3, o
        b.close()
