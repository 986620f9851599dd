"""Spin precession in the tile kernels of both orders and precisions.

One teacher-forced step of electrons with random spins in the fields of a hot
plasma, with a Schwinger field small enough that the g-factor table is read,
against the oracle: arrays and momenta at the one-step parity bounds, spins to
1e-12 in FP64 and 1e-5 in FP32 (unit vectors, stored in the context's
precision).
"""
import numpy as np
import pytest

import oracle as O
from golden_io import load
from parity import TOL_FP32, TOL_FP64, array_errors, by_id, particle_errors, periods

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("tile", [0, 2, -1], ids=["nodes", "cells", "global"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
def test_spins_match_the_oracle(mem, tile, precision):
    from pic3d_b200.simulation import Simulation
    g_data = load("spin_o2")["g_data"]
    w = W.Workload(name="spin", nx=12, ny=10, nz=11, mem=mem, period=(1, 1, 1), ppc=(2, 1), u_th=(0.3, 0.05), steps=3,
                   E_schwinger=0.5)
    parts = W.make_particles(w, seed=23)
    rng = np.random.default_rng(4)
    s = rng.normal(size=(len(parts[0]), 3))
    s /= np.linalg.norm(s, axis=1, keepdims=True)
    for d, f in enumerate(("sx", "sy", "sz")):
        parts[0][f] = s[:, d]
    states, _ = O.run_oracle(w, parts, 3, g_data=g_data)
    sim = Simulation(w, precision=precision, tile=tile)
    sim.set_g_table(g_data)
    tol, pos_tol, spin_tol = (TOL_FP64, 1e-11, 1e-12) if precision == "fp64" else (TOL_FP32, 2e-6, 1e-5)
    for n in range(3):
        sim.upload_state(states[n])
        sim.step = n
        sim.run_main_time_loop(1)
        got, ref = sim.state(), states[n + 1]
        errs = array_errors(got, ref)
        assert max(errs.values()) < tol, (n + 1, errs)
        for k in range(2):
            perr, merr = particle_errors(got["particles"][k], ref["particles"][k], periods(w.params()))
            assert perr < pos_tol and merr < tol, (n + 1, k, perr, merr)
        a, b = by_id(got["particles"][0]), by_id(ref["particles"][0])
        turned = max(np.max(np.abs(b[f] - by_id(parts[0])[f])) for f in ("sx", "sy", "sz"))
        assert turned > 1e-3   # the run turns them
        for f in ("sx", "sy", "sz"):
            assert np.max(np.abs(a[f] - b[f])) < spin_tol, (n + 1, f)
    sim.close()
