"""The one-reduction and mixed solvers (pcg_mixed.cu) on graphs with many closures to random
poses, where the rows that a CTA reads from others (its halo) are several times its own rows and
v of all of them does not fit shared memory: the graph is still solved, with the rest of v in
global memory. Sizes: the halo just too long in some CTAs (50,000 poses), in nearly all (80,000,
100,000), and with few rows but very many closures (20,000).

Against the streaming solver of the same graph, with the bounds that test_gpu_resident_edges.py
derives for these solvers after 40 iterations: 1e-6 (the same steps in another recurrence), and
5e-2 in FP32 (a row or block read from the wrong place is a step of another direction)."""
import importlib

import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu

PREC_MIXED, PREC_CG = 1, 2
ITS = 40


def _graph(n, k):
    """A walk and k closures per pose to random poses."""
    cg = importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth").city_grid(n, seed=n, k_closures=0)
    rng = np.random.default_rng(n)
    m = int(k * n)
    i, j = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    ok = i != j
    rel = rng.normal(size=(int(ok.sum()), 3)) * 0.1
    return (cg.init, np.concatenate([cg.edge_i, i[ok]]), np.concatenate([cg.edge_j, j[ok]]),
            np.concatenate([cg.meas, rel]), np.concatenate([cg.log_w, np.zeros_like(rel)]))


def _dx(pkg, graph, **opts):
    with pkg.PoseGraph.from_se2(*graph, lam=0.1, tol=0.0, max_iter=ITS, inner_tol=0.0, **opts) as g:
        g.linearise()
        g.assemble()
        out = []
        for _ in range(2):      # the second solve starts on what the first one left
            assert g.solve().iterations == ITS
            out.append(g.dx())
    assert_bitwise(out[1], out[0], "the same solve again")
    return out[0]


@pytest.mark.parametrize("n, k, prec, bound", [
    (20_000, 16, PREC_CG, 1e-6), (50_000, 5.5, PREC_CG, 1e-6), (80_000, 3, PREC_CG, 1e-6),
    (80_000, 5, PREC_MIXED, 5e-2), (100_000, 4, PREC_MIXED, 5e-2)])
def test_halo_too_long_for_shared_memory(pkg, n, k, prec, bound):
    graph = _graph(n, k)
    b = _dx(pkg, graph, disable_resident=1)
    a = _dx(pkg, graph, precision=prec)
    assert np.linalg.norm(a - b) <= bound * np.linalg.norm(b)
