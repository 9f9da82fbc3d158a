"""The grid-wide resident solvers (pcg_resident.cu; pcg_mixed.cu in FP64 and FP32) at the sizes
where the kernel or its shared-memory split changes, against the streaming solver of the same graph
(disable_resident): 12, 16, 24 and 32 slices in the largest CTA, values that do not all fit,
halos longer than the CTA's threads. The two add the dot products in other orders (relative
1e-15 per sum), which 60 iterations amplify by far less than the 1e-9 allowed. The
one-reduction solver takes the same steps in another recurrence (1e-6 allowed after 40), the
mixed one in FP32 (6e-8 per operation; 5e-2 allowed after 40: a row or block read from the
wrong place shows as a step of another direction altogether)."""
import importlib

import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu


def _dx(pkg, cg, i, j, meas, lw, its=60, **opts):
    with pkg.PoseGraph.from_se2(cg.init, i, j, meas, lw, lam=0.1, tol=0.0, max_iter=its, **opts) as g:
        g.linearise()
        g.assemble()
        out = []
        for _ in range(2):      # a second solve on the same buffers: the same bits
            assert g.solve().iterations == its
            out.append(g.dx())
    assert_bitwise(out[1], out[0], "the same solve again")
    return out[0]


def _check(pkg, cg, i, j, meas, lw):
    b = _dx(pkg, cg, i, j, meas, lw, disable_resident=1)
    a = _dx(pkg, cg, i, j, meas, lw)
    assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)
    if (cg.n_poses + 31) // 32 <= 32 * 148:
        b = _dx(pkg, cg, i, j, meas, lw, its=40, disable_resident=1)
        for prec, bound in ((2, 1e-6), (1, 5e-2)):
            a = _dx(pkg, cg, i, j, meas, lw, its=40, precision=prec, inner_tol=0.0)
            assert np.linalg.norm(a - b) <= bound * np.linalg.norm(b)


@pytest.mark.parametrize("n", [4700, 33000, 45000, 60001, 90000, 120000, 151552, 151553])
def test_resident_matches_streamed(pkg, n):
    cg = importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth").city_grid(n, seed=n)
    _check(pkg, cg, cg.edge_i, cg.edge_j, cg.meas, cg.log_w)


@pytest.mark.parametrize("n", [12000, 30000, 80000])
def test_long_halos(pkg, n):
    """A closure from every pose to a random one: almost every block column is another CTA's."""
    cg = importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth").city_grid(n, seed=n)
    rng = np.random.default_rng(n)
    j = rng.permutation(n).astype(np.uint32)
    i = np.arange(n, dtype=np.uint32)
    i, j = i[i != j], j[i != j]
    rel = rng.normal(size=(len(i), 3)) * 0.1
    _check(pkg, cg, np.concatenate([cg.edge_i, i]), np.concatenate([cg.edge_j, j]), np.concatenate([cg.meas, rel]),
           np.concatenate([cg.log_w, np.zeros_like(rel)]))
