"""Step graphs: what tsg_get_launch says of them, what they hold, and how they are counted."""
import ctypes
import threading

import pytest
import torch

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


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_launches_counted_while_other_threads_launch(native, precision):
    """Two threads, a handle each: every parameter change has the next step captured again, and
    neither thread's launches enter what the other counts for its graphs."""
    from tisphi_gb300.simulation import Simulation

    def work(sim):
        with torch.cuda.stream(torch.cuda.Stream()):
            for q in range(60):
                sim.solver.viscosity = 0.005 + 1e-6 * (q % 3)
                sim.solver.step(1 + 3 * (q % 2))
            torch.cuda.synchronize()

    def total(together):
        sims = [Simulation(cfg_of(small_dambreak_2d()), precision=precision) for _ in range(2)]
        for s in sims:
            s.solver.step(2)
        torch.cuda.synchronize()
        before = native.tsg_launch_count()
        if together:
            threads = [threading.Thread(target=work, args=(s,)) for s in sims]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
        else:
            for s in sims:
                work(s)
        return native.tsg_launch_count() - before

    alone = total(False)
    assert alone > 0 and [total(True) for _ in range(3)] == [alone] * 3


@pytest.mark.parametrize("precision,method", [("fp64", 1), ("fp64", 2), ("fp32_mixed", 1), ("fp32_mixed", 2)])
def test_graphs_made_while_another_thread_synchronises(native, precision, method):
    """A thread that waits for the device all the time, while parameter changes have every step's
    graph made anew: neither side fails, and the state is that of an undisturbed run, bit for bit."""
    from tisphi_gb300.simulation import Simulation

    def run():
        sim = Simulation(cfg_of(small_dambreak_2d() if method == 1 else small_column(2)), precision=precision)
        for q in range(40):
            if method == 1:
                sim.solver.viscosity = 0.005 + 1e-6 * (q % 3)
            else:
                sim.solver.coh = 0.1 * (q % 3)
            sim.solver.step(1 + q % 3)
        return [sim.ps.field(nm).cpu() for nm in ("x", "v", "density", "id0")]

    want = run()
    stop, failed, waits = threading.Event(), [], [0]

    def wait():
        try:
            while not stop.is_set():
                torch.cuda.synchronize()
                waits[0] += 1
        except RuntimeError as e:
            failed.append(e)

    t = threading.Thread(target=wait)
    t.start()
    got = run()
    stop.set()
    t.join()
    assert not failed and waits[0] > 10
    assert all(torch.equal(a, b) for a, b in zip(want, got))


FIELDS = ["x", "v", "density", "pressure", "id0"]


@pytest.mark.parametrize("precision,method", [(p, m) for p in ("fp64", "fp32_mixed") for m in (1, 2, 3)])
@pytest.mark.parametrize("warm", [12, 13])
def test_parameter_changes_reach_the_graphs(native, precision, method, warm):
    """Graphs hold the constants by value.  After enough steps for every length of graph, from
    either buffer of the FP64 sort, a changed parameter gives what steps launched one by one with
    it give, bit for bit, and not what the old one gives."""
    from tisphi_gb300.simulation import Simulation
    lib = native

    def sim():
        return Simulation(cfg_of(small_dambreak_2d() if method == 1 else small_column(method)), precision=precision)

    def change(s):
        if method == 1:
            s.solver.stiffness = 6.0e4
        elif method == 2:
            s.solver.mu = 0.5
        else:
            s.solver.coh = 500.0
            s.solver.fric = 0.3

    names = FIELDS + (["stress"] if method != 1 else [])
    graphs, eager, old = sim(), sim(), sim()
    for s in (graphs, eager, old):
        s.solver.step(warm)
        s.solver.step(1)  # (both lengths of graph)
    for s in (graphs, eager):
        change(s)
    for n in (1, 2, 6):
        graphs.solver.step(n)
        old.solver.step(n)
        lib.tsg_profile(1)
        try:
            eager.solver.step(n)
        finally:
            lib.tsg_profile(0)
        for nm in names:
            assert torch.equal(graphs.ps.field(nm), eager.ps.field(nm)), nm
    assert not torch.equal(graphs.ps.field("v"), old.ps.field("v"))


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_steps_while_another_thread_captures(native, precision):
    """A thread that captures a graph of its own in the default mode, which forbids every other
    thread what may touch the capture, while steps make, replay and drop theirs: neither notices."""
    from tisphi_gb300.simulation import Simulation

    def run(sim):
        for n in (1, 1, 2, 1, 5, 6, 12, 5):
            sim.solver.step(n)
        sim.solver.viscosity = 0.006
        sim.solver.step(4)

    a, b = (Simulation(cfg_of(small_dambreak_2d()), precision=precision) for _ in range(2))
    run(a)
    x = torch.ones(1000, device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    inside, stepped, got = threading.Event(), threading.Event(), []

    def capture():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                g = torch.cuda.CUDAGraph()
                g.capture_begin()
                torch.mul(x, 2, out=y)
                inside.set()
                stepped.wait(60)
                torch.add(y, 1, out=y)
                g.capture_end()
                g.replay()
                torch.cuda.current_stream().synchronize()
                got.append(float(y[0]))
        except RuntimeError as e:
            got.append(e)
        finally:
            inside.set()

    t = threading.Thread(target=capture)
    t.start()
    inside.wait(60)
    try:
        with torch.cuda.stream(torch.cuda.Stream()):
            run(b)
    finally:
        stepped.set()
        t.join()
    torch.cuda.synchronize()
    assert got == [3.0]
    for nm in ("x", "v", "density", "id0"):
        assert torch.equal(a.ps.field(nm), b.ps.field(nm)), nm


@pytest.mark.parametrize("warm", [0, 7])
@pytest.mark.parametrize("method", [1, 2])
def test_fp64_steps_inside_a_callers_capture(native, method, warm):
    """Two FP64 steps captured by the caller are the launches themselves, before and after the
    handle has graphs of its own: three replays are six steps, bit for bit."""
    from tisphi_gb300.simulation import Simulation
    a, b = (Simulation(cfg_of(small_dambreak_2d() if method == 1 else small_column(2)), precision="fp64")
            for _ in range(2))
    for s in (a, b):
        if warm:
            s.solver.step(warm)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.solver.step(2)
    for _ in range(3):
        g.replay()
    b.solver.step(6)
    torch.cuda.synchronize()
    for nm in FIELDS:
        assert torch.equal(a.ps.field(nm), b.ps.field(nm)), nm
