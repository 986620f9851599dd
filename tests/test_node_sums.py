"""Sums over the particles of a node (tiles of nodes, both orders).

Every particle has a weight of its own, far from its neighbours', so that a
particle deposited with another's weight, or with inputs that were overwritten
before it read them, shows at once.  Nodes hold none to several batches of
particles, all moving or half of them at rest (those add rho, no current); one
step against the oracle at the one-step parity bounds (relative L2 1e-10 in
FP64, 1e-5 in FP32).
"""
import numpy as np
import pytest

import oracle as O
from parity import TOL_FP32, TOL_FP64, array_errors

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("ppc", [1, 9, 70])
def test_every_particle_deposits_its_own_weight(ppc, mem, precision):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="weights", nx=11, ny=10, nz=13, mem=mem, period=(1, 1, 1), ppc=(ppc, 2), u_th=(0.1, 0.02), steps=2)
    parts = W.make_particles(w, seed=41)
    rng = np.random.default_rng(6)
    for p in parts:
        p["weight"] *= 10.0 ** rng.uniform(-2.0, 0.0, len(p))
    states, _ = O.run_oracle(w, parts, 2)
    sim = Simulation(w, precision=precision)
    tol = TOL_FP64 if precision == "fp64" else TOL_FP32
    for n in range(2):
        sim.upload_state(states[n])
        sim.step = n
        sim.run_main_time_loop(1)
        errs = array_errors(sim.state(), states[n + 1])
        bad = {k: v for k, v in errs.items() if v > tol}
        assert not bad, (n + 1, bad)
    sim.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("steps", [1, 2], ids=["rho", "no_rho_first"])
def test_particles_at_rest_among_moving_ones(steps, mem, precision):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="rest", nx=12, ny=10, nz=11, mem=mem, period=(1, 1, 1), ppc=(6, 0), u_th=(0.2, 0.0), steps=steps)
    parts = W.make_particles(w, seed=9)
    still = np.random.default_rng(1).random(len(parts[0])) < 0.5
    for f in ("px", "py", "pz"):
        parts[0][f][still] = 0.0
    parts[0]["gamma"] = np.sqrt(1.0 + parts[0]["px"] ** 2 + parts[0]["py"] ** 2 + parts[0]["pz"] ** 2)
    o = O.Oracle(w, parts)
    for s in range(1, steps + 1):
        o.step(s)
    sim = Simulation(w, precision=precision)
    sim.upload_particles(0, parts[0])
    sim.run_main_time_loop(steps)
    errs = array_errors(sim.state(), o.state())
    sim.close()
    assert max(errs.values()) < (TOL_FP64 if precision == "fp64" else TOL_FP32), errs
