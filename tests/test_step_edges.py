"""Edges of the launches around the push.

* Between two steps of one pic_run_steps call on a fully periodic grid, the
  second E half-update of one and the first of the next are one pass; on other
  grids they are two, with the boundary conditions between them.  Several
  steps in one call against the same steps one by one: the rounding of the
  field updates is the same, the currents differ by the order of additions
  (relative L2 1e-10 in FP64, 1e-5 in FP32, the one-step parity bounds).
* Removal: none, one, most or all of the particles of one or both species
  leave in a step, against the oracle.  The index lists hold the particles that
  leave, the holes and the particles that fill them in one buffer.
"""
import numpy as np
import pytest

import oracle as O
from parity import TOL_FP32, TOL_FP64, array_errors, particle_errors, periods

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("period", [(1, 1, 1), (0, 1, 1), (1, 0, 1), (0, 0, 0)])
def test_steps_in_one_call_equal_single_steps(mem, precision, period):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="edges", nx=11, ny=10, nz=13, mem=mem, period=period, ppc=(2, 2), u_th=(0.1, 0.1), steps=5)
    parts = W.make_particles(w, seed=3)
    states = []
    for calls in ((5,), (1, 1, 1, 1, 1), (2, 3)):
        sim = Simulation(w, precision=precision)
        for k in range(2):
            sim.upload_particles(k, parts[k])
        sim.initial_push()
        for n in calls:
            sim.run_main_time_loop(n)
        states.append(sim.state())
        sim.close()
    tol = TOL_FP64 if precision == "fp64" else TOL_FP32
    for other in states[1:]:
        errs = array_errors(states[0], other)
        assert max(errs.values()) < tol, errs


# (part of species 0, part of species 1) that flies out of the x faces
LEAVERS = {"none": (0.0, 0.0), "one_species": (0.5, 0.0), "most": (0.9, 0.3), "all_of_one": (1.0, 0.2)}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("tile", [0, -1], ids=["tiles", "global"])
@pytest.mark.parametrize("case", list(LEAVERS))
def test_removal_of_many_particles(case, tile, precision):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name=case, nx=12, ny=10, nz=11, mem=2, period=(0, 1, 1), ppc=(3, 2), u_th=(0.05, 0.05), steps=3)
    parts = W.make_particles(w, seed=8)
    rng = np.random.default_rng(1)
    for k in range(2):
        out = rng.random(len(parts[k])) < LEAVERS[case][k]
        low = rng.random(len(parts[k])) < 0.5
        parts[k]["x"][out] = np.where(low, 0.03, w.nx - 0.03)[out]
        parts[k]["px"][out] = np.where(low, -2.0, 2.0)[out]
        q = parts[k]
        q["gamma"] = np.sqrt(1.0 + q["px"] ** 2 + q["py"] ** 2 + q["pz"] ** 2)
    states, _ = O.run_oracle(w, parts, 3)
    ref = states[-1]
    sim = Simulation(w, precision=precision, tile=tile)
    for k in range(2):
        sim.upload_particles(k, parts[k])
    sim.initial_push()
    sim.run_main_time_loop(3)
    got = sim.state()
    sim.close()
    tol, pos_tol = (1e-8, 1e-9) if precision == "fp64" else (1e-4, 1e-5)
    errs = array_errors(got, ref)
    assert max(errs.values()) < tol, errs
    for k in range(2):
        assert sorted(got["particles"][k]["id"]) == sorted(ref["particles"][k]["id"])
        if len(ref["particles"][k]):
            perr, merr = particle_errors(got["particles"][k], ref["particles"][k], periods(w.params()))
            assert perr < pos_tol and merr < tol, (k, perr, merr)
