"""The default tile kernels at the edges of their tiles.

A tile holds 4 x 4 x 4 nodes, so a box of n cells has n // 4 + 1 tiles per
axis and the last one is full, partial or a single layer of nodes.  One
teacher-forced step against the oracle at the parity bounds (relative L2
1e-10 in FP64, 1e-5 in FP32, every array and every particle), with the
momenta large enough that many particles change node along every axis, for
rows of nodes that are empty, hold one particle, or more than a batch of 32.
"""
import numpy as np
import pytest

import oracle as O
from parity import TOL_FP32, TOL_FP64, array_errors, particle_errors, periods

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu

# cells per axis with every remainder of 4, particles per cell, momentum spread
CASES = {"sparse": ((10, 13, 11), (1, 0), 0.5), "remainders": ((12, 11, 14), (3, 2), 0.3),
         "dense_rows": ((13, 12, 10), (40, 8), 0.05), "cold": ((16, 10, 12), (6, 6), 0.0)}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("period", [(1, 1, 1), (0, 1, 1)], ids=["periodic", "absorbing_x"])
def test_tile_edges_match_the_oracle(case, mem, precision, period):
    from pic3d_b200.simulation import Simulation
    (nx, ny, nz), ppc, u = CASES[case]
    w = W.Workload(name=case, nx=nx, ny=ny, nz=nz, mem=mem, period=period, ppc=ppc, u_th=(u, u), steps=3)
    states, _ = O.run_oracle(w, W.make_particles(w, seed=31), 3)
    tol, pos_tol = (TOL_FP64, 1e-11) if precision == "fp64" else (TOL_FP32, 2e-6)
    sim = Simulation(w, precision=precision)
    for n in range(3):
        sim.upload_state(states[n])
        sim.step = n
        sim.run_main_time_loop(1)
        got = sim.state()
        errs = array_errors(got, states[n + 1])
        bad = {k: v for k, v in errs.items() if v > tol}
        assert not bad, (n + 1, bad)
        for k in range(2):
            perr, merr = particle_errors(got["particles"][k], states[n + 1]["particles"][k], periods(w.params()))
            assert perr < pos_tol and merr < tol, (n + 1, k, perr, merr)
    sim.close()
