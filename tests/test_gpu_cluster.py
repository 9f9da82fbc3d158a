"""The solver of a graph inside one thread-block cluster (pcg_cluster.cu) against the
grid-wide solvers on the same graphs, at the sizes where its split changes: one CTA (up to
13 slices of 32 rows), 2 to 16 CTAs, 144 slices and one more, and in a batch one and two
rows per thread and graphs that do not fit.

test_absent_cta beyond every grid is no CTA at all, but it names a CTA that no cluster has,
so such a handle runs the grid-wide solver. Both solvers take the same PCG iterates; above
one CTA only the order of the dot products' sums differs (relative 1e-15 per sum), which 60
iterations of these systems amplify by far less than the 1e-9 allowed."""
import importlib

import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu

GRID = dict(test_absent_cta=1 << 20)
PREC_FP64, PREC_MIXED = 0, 1


@pytest.fixture(scope="module")
def synth():
    return importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth")


def _se2(pkg, cg, lam=0.1, **opts):
    return pkg.PoseGraph.from_se2(cg.init, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, lam=lam, **opts)


def _solve(g):
    g.linearise()
    g.assemble()
    st = g.solve()
    dx = g.dx()
    g.close()
    return st, dx


@pytest.mark.parametrize("n", [1, 2, 31, 33, 100, 257, 416])
@pytest.mark.parametrize("kind", ["se2", "log"])
def test_one_cta_gives_the_grid_solvers_bits(pkg, synth, kind, n):
    """Full default solves (500 iterations, past convergence at these sizes)."""
    if kind == "se2":
        cg = synth.city_grid(n, seed=n) if n > 1 else None
        if cg is None:
            pytest.skip("a walk has two poses")
        make = lambda **o: _se2(pkg, cg, **o)  # noqa: E731
    else:
        if n == 1:
            u = np.array([[1.0, 0.1]])
            make = lambda **o: pkg.PoseGraph.from_reference(np.zeros((1, 3)), u, 1.0, 1.0, [], [],  # noqa: E731
                                                            np.zeros((0, 2)), **o)
        else:
            log = synth.landmark_log(n, seed=n)
            make = lambda **o: pkg.PoseGraph.from_log(log, 0.1, **o)  # noqa: E731
    (a, xa), (b, xb) = _solve(make()), _solve(make(**GRID))
    assert (a.iterations, a.reason, a.rel_residual) == (b.iterations, b.reason, b.rel_residual)
    assert_bitwise(xa, xb, f"{kind} n={n}")


@pytest.mark.parametrize("n", [417, 449, 1025, 2049, 4608, 4609, 5376, 5377, 7168, 7169])
@pytest.mark.parametrize("kind", ["se2", "far", "log"])
def test_cluster_takes_the_grid_solvers_iterates(pkg, synth, kind, n):
    opts = dict(tol=0.0, max_iter=60)
    if kind == "log":
        log = synth.landmark_log(n, seed=n)
        make = lambda **o: pkg.PoseGraph.from_log(log, 0.1, **opts, **o)  # noqa: E731
    else:
        cg = synth.city_grid(n, seed=n) if kind == "se2" else synth.city_grid(n, seed=n, k_closures=6, radius=3.0,
                                                                             far_fraction=0.02)
        make = lambda **o: _se2(pkg, cg, **opts, **o)  # noqa: E731
    (a, xa), (b, xb) = _solve(make()), _solve(make(**GRID))
    assert a.iterations == b.iterations == 60
    assert np.linalg.norm(xa - xb) <= 1e-9 * np.linalg.norm(xb)


def test_rows_too_wide_for_shared_memory(pkg, synth):
    """A pose that every other one closes to: one slice of 2,000 blocks per row does not fit a
    CTA's shared memory, so the graph is solved by the streaming solver as before."""
    cg = synth.city_grid(2000, seed=4)
    i = np.concatenate([cg.edge_i, np.zeros(1998, np.uint32)])
    j = np.concatenate([cg.edge_j, np.arange(2, 2000, dtype=np.uint32)])
    rel = cg.gt[2:] - cg.gt[0]
    meas = np.concatenate([cg.meas, rel])
    lw = np.concatenate([cg.log_w, np.zeros_like(rel)])
    out = []
    for o in ({}, dict(disable_resident=1)):
        out.append(_solve(pkg.PoseGraph.from_se2(cg.init, i, j, meas, lw, lam=0.1, tol=0.0, max_iter=30, **o)))
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-9 * np.linalg.norm(out[1][1])


def test_absent_cta_of_the_cluster_times_out(pkg, synth):
    g = _se2(pkg, synth.city_grid(2000, seed=5), barrier_timeout_ms=20.0, test_absent_cta=3)
    g.linearise()
    g.assemble()
    with pytest.raises(pkg.abi.GslamError) as e:
        g.solve()
    assert e.value.code == pkg.abi.ERR_DEVICE_TIMEOUT
    g.set_opts(test_absent_cta=-1)
    assert g.solve().iterations == 500
    g.close()


SIZES = (37, 320, 330, 640, 650, 5000, 10240, 10250, 20480, 20500)   # the last one fits no cluster


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_batch_clusters_take_the_grid_solvers_iterates(pkg, synth, prec):
    """FP32 sums are rounded to 6e-8 of the step's parts at every iteration; the two orders of
    the FP64 dot products change a rounded coefficient at most now and then."""
    graphs = [synth.city_grid(n, seed=n) for n in SIZES]
    out = []
    for o in ({}, GRID):
        b = pkg.PoseGraphBatch.from_se2_list(graphs, 0.1, tol=0.0, max_iter=60, inner_tol=0.0, inner_max_iter=60,
                                             precision=prec, **o)
        st = b.round_all()
        out.append((b.poses - b.init_poses, b))
        assert [s.iterations for s in st if s.reason != 0] == [60] * sum(s.reason != 0 for s in st)
    for q in range(len(SIZES)):
        da, db = (b.graph_poses(q, d) for d, b in out)
        assert np.linalg.norm(da - db) <= (1e-9 if prec == PREC_FP64 else 1e-3) * np.linalg.norm(db) + 1e-12
    for _, b in out:
        b.close()


def test_batch_options_still_shape_the_solve(pkg, synth):
    """Streamed-only batches, and a change of precision on a live handle."""
    graphs = [synth.city_grid(n, seed=n) for n in (300, 2000, 900)]
    ref = None
    for o in ({}, dict(disable_resident=1)):
        b = pkg.PoseGraphBatch.from_se2_list(graphs, (0.1, 0.5, 1.0), tol=0.0, max_iter=50, **o)
        b.round_all()
        p = b.poses
        ref = p if ref is None else ref
        assert np.linalg.norm(p - ref) <= 1e-9 * np.linalg.norm(ref)
        b.poses = b.init_poses
        b.set_opts(precision=PREC_MIXED, inner_tol=1e-5)
        st = b.round_all()
        assert all(s.refinements != 0 for s in st)
        b.close()


@pytest.mark.parametrize("n", [300, 450, 2500])
def test_adjoint_keeps_the_grid_solvers_bits(pkg, synth, n):
    """The exact Hessian can be indefinite, where two orders of the sums end far apart (4e-3
    of mu measured at 800 poses): the adjoint's sums keep the grid-wide solver's order."""
    cg = synth.city_grid(n, seed=1)
    rng = np.random.default_rng(n)
    poses = cg.gt + rng.normal(size=cg.gt.shape) * [0.01, 0.01, 0.002]
    grad = rng.normal(size=cg.gt.shape)
    out = []
    for o in ({}, GRID):
        with pkg.PoseGraph.from_se2(poses, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, lam=0.5, **o) as g:
            out.append(g.adjoint(grad))
    assert out[0][0] == out[1][0]
    assert_bitwise(out[0][1], out[1][1], "dL/dlog_w")
    assert_bitwise(out[0][2], out[1][2], "mu")
