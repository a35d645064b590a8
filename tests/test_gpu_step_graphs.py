"""Step graphs of the FP32-mixed form: what tsg_get_launch says of them."""
import ctypes

import pytest

from helpers import cfg_of, small_column, small_dambreak_2d

pytestmark = pytest.mark.gpu


def _steps_per_graph(lib, ps):
    from tisphi_gb300 import _native as nat
    c = nat.tsg_launch_cfg()
    nat.check(lib.tsg_get_launch(ps._h, ctypes.byref(c)), "tsg_get_launch")
    return c.steps_per_graph


def _launches_of(lib, sim, steps):
    before = lib.tsg_launch_count()
    sim.solver.step(steps)
    return lib.tsg_launch_count() - before


def test_get_launch_reports_the_graphs_replayed(native):
    """Single-step graphs for ten steps, five-step graphs after that; a caller's choice as given."""
    from tisphi_gb300 import _native as nat
    from tisphi_gb300.simulation import Simulation
    lib = native
    sim = Simulation(cfg_of(small_dambreak_2d()), precision="fp32_mixed")
    assert _steps_per_graph(lib, sim.ps) == 1
    sim.solver.step(4)
    assert _steps_per_graph(lib, sim.ps) == 1
    sim.solver.step(6)
    assert _steps_per_graph(lib, sim.ps) == 5
    # (a five-step graph checks the lists' expiry once: fewer launches than five single steps)
    five = _launches_of(lib, sim, 5)
    assert five < sum(_launches_of(lib, sim, 1) for _ in range(5))
    cfg = nat.tsg_launch_cfg(128, 0, 3)
    nat.check(lib.tsg_set_launch(sim.ps._h, ctypes.byref(cfg)), "tsg_set_launch")
    assert _steps_per_graph(lib, sim.ps) == 3
    sim.solver.step(20)
    assert _steps_per_graph(lib, sim.ps) == 3


@pytest.mark.parametrize("method", [1, 2])
def test_parameter_changes_start_with_single_step_graphs(native, method):
    """A five-step graph takes as long to capture as several steps take to run: a caller that
    sets a parameter every few steps gets single-step graphs, as a new handle does."""
    from tisphi_gb300.simulation import Simulation
    sim = Simulation(cfg_of(small_dambreak_2d() if method == 1 else small_column(2)), precision="fp32_mixed")
    sim.solver.step(12)
    assert _steps_per_graph(native, sim.ps) == 5
    if method == 1:
        sim.solver.viscosity = 0.006
    else:
        sim.solver.coh = 1.0
    assert _steps_per_graph(native, sim.ps) == 1
    sim.solver.step(10)
    assert _steps_per_graph(native, sim.ps) == 5


def test_a_write_of_x_leaves_no_trace_in_later_graphs(native):
    """mu(I): graphs captured after a write of x hold the same kernels as others (the five-step
    graph one displacement check, the regularisation the lists)."""
    from tisphi_gb300.simulation import Simulation
    a, b = (Simulation(cfg_of(small_column(2)), precision="fp32_mixed") for _ in range(2))
    for s in (a, b):
        s.solver.step(10)
    b.ps.write_field("x", b.ps.field("x").contiguous())
    for s in (a, b):
        s.solver.step(5)
    assert _launches_of(native, a, 5) == _launches_of(native, b, 5)
