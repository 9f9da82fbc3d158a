"""Solvers of different kinds and sizes run one after another on one GPU: a solve must not
depend on what an earlier kernel left in shared memory (the one-reduction and mixed solvers
keep ||xi|| there and every thread reads it right after it is written)."""
import importlib

import numpy as np
import pytest

from conftest import assert_bitwise

pytestmark = pytest.mark.gpu

PREC_FP64, PREC_MIXED, PREC_CG = 0, 1, 2


@pytest.mark.parametrize("prec", [PREC_CG, PREC_MIXED], ids=["one-reduction", "mixed"])
def test_solve_is_independent_of_earlier_kernels(pkg, prec):
    synth = importlib.import_module("g-slam_on_gpu_and_fpga_b200.synth")
    cg = synth.city_grid(300, seed=3)
    # other solves in between, whose shared memory holds matrix values and sums of every size
    others = [(0.06, synth.city_grid(n, seed=1)) for n in (200, 1500, 9000)] + [(1e6, synth.city_grid(400, seed=2))]
    out = []
    with pkg.PoseGraph.from_se2(cg.init, cg.edge_i, cg.edge_j, cg.meas, cg.log_w, lam=0.06, precision=prec,
                                barrier_timeout_ms=200.0) as g:
        for lam, o in [(None, None)] + others:
            if o is not None:
                for p in (PREC_FP64, PREC_CG):
                    with pkg.PoseGraph.from_se2(o.init, o.edge_i, o.edge_j, o.meas, o.log_w, lam=lam, precision=p) as h:
                        h.round()
            g.poses = cg.init
            st = g.round()
            out.append((st.iterations, st.reason, g.poses))
    for it, reason, poses in out[1:]:
        assert (it, reason) == out[0][:2]
        assert_bitwise(poses, out[0][2], "poses after the same solve")
    assert np.isfinite(out[0][2]).all()
