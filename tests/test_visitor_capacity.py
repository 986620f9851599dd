"""The visitor lists hold what a relativistic plasma needs between two sorts.

Isotropic electrons close to the speed of light cross 0.55 cells a step: three
pushes after a sort, the last time that lists are read at the default interval,
half of them or more are in another tile than the one whose slice holds them
(0.50 to 0.58, by the size of the box).  All of these are pushed from the
lists, none by the global kernel.
"""
import pytest

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("n", [(24, 24, 16), (12, 13, 14)])
def test_lists_hold_an_ultrarelativistic_plasma_between_sorts(n, mem):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="hot", nx=n[0], ny=n[1], nz=n[2], mem=mem, period=(1, 1, 1), ppc=(24, 0), u_th=(5.0, 0.0), steps=8)
    sim = Simulation(w, precision="fp32")
    sim.generate_thermal(0, 24, 1e-6, 5.0, 3)
    sim.initial_push()
    away = []
    for _ in range(8):
        sim.run_main_time_loop(1)
        s = sim.particle_order_stats(0)
        assert s["global_kernel"] == 0, s
        away.append(s["visitors"])
    sim.close()
    assert max(away) > 0.5 * w.num_particles   # the case is hot enough to need more than half
