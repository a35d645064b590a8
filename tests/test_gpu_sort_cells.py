"""Order and cost of the sort where one cell holds most of the particles.

Up to 16,384 particles the reorder pass ranks every cell itself, whatever its size; the
out-of-grid bin of a run that has blown up then holds thousands.  Above that, cells of more than
256 particles are listed and ordered by a block each: in shared memory up to 4,096 particles, by a
scan over all particles above.  The order is the stable counting sort's
(eng/particle_system.py:228-257) for any start and length of the cell, and the sort of a blown-up
scene stays within a few times that of a healthy one.
"""
import contextlib
import ctypes

import numpy as np
import pytest

from helpers import cfg_of, small_dambreak_2d

pytestmark = pytest.mark.gpu


def _moved(precision, spacing, count):
    """A dambreak with `count` fluid particles far outside the grid, and their present places."""
    from tisphi_gb300.simulation import Simulation
    sim = Simulation(cfg_of(small_dambreak_2d(spacing=spacing)), precision=precision)
    ps = sim.ps
    fl = np.nonzero(ps.field("mat_type").cpu().numpy() == 1)[0]
    x = ps.field("x").cpu().numpy().astype(np.float64)
    rng = np.random.default_rng(count)
    moved = np.sort(rng.choice(fl, size=count, replace=False))
    x[moved, 0] = -5.0 - rng.random(count)
    ps.write_field("x", np.ascontiguousarray(x))
    return sim, fl, moved


def _sort(ps):
    from tisphi_gb300 import _native as nat
    with contextlib.suppress(nat.NativeError):  # out-of-grid status
        ps.initialize_particle_system()


# (lengths on both sides of the 64 up to which a cell is read entry by entry, of its chunks of 32
# and of the 256 entries of a trip)
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("count", [63, 64, 65, 95, 96, 97, 255, 256, 257, 2049, 9600])
def test_order_in_one_large_cell(native, precision, count):
    sim, fl, moved = _moved(precision, 0.005, count)
    ps = sim.ps
    assert ps.particle_max_num <= 16384
    before = ps.field("id0").cpu().numpy().copy()
    _sort(ps)
    ids = ps.field("id0").cpu().numpy()
    end = ids.size if precision == "fp64" else fl.size  # FP32-mixed: the bin ends the fluid's block
    np.testing.assert_array_equal(ids[end - count:end], before[moved])


# (256 / 257: ranked / listed; 4,096 / 4,097: shared memory / scan)
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
@pytest.mark.parametrize("count", [256, 257, 1000, 4096, 4097, 20000])
def test_order_in_listed_cells(native, precision, count):
    sim, fl, moved = _moved(precision, 0.003, count)
    ps = sim.ps
    assert fl.size > 16384  # the FP32-mixed form sorts the fluid by itself
    before = ps.field("id0").cpu().numpy().copy()
    _sort(ps)
    ids = ps.field("id0").cpu().numpy()
    end = ids.size if precision == "fp64" else fl.size
    np.testing.assert_array_equal(ids[end - count:end], before[moved])
    assert np.array_equal(np.sort(ids), np.arange(ids.size))


def _sort_ms(lib, ps, reps=20):
    """Fastest of `reps` sorts, device time of the sort phase."""
    best = float("inf")
    for _ in range(reps):
        lib.tsg_profile(1)
        _sort(ps)
        ms, n = (ctypes.c_double * 11)(), (ctypes.c_int64 * 11)()
        lib.tsg_profile_read(ms, n, 11)
        lib.tsg_profile(0)
        best = min(best, ms[0])
    return best


@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_sort_after_a_blow_up_costs_like_a_sort(native, precision):
    """Every fluid particle in the out-of-grid bin, against the same scene in place: three and a
    half times the sort at most (every thread reading the whole bin took seven to eight times)."""
    from tisphi_gb300.simulation import Simulation
    lib = native
    healthy = Simulation(cfg_of(small_dambreak_2d(spacing=0.005)), precision=precision)
    blown, _, _ = _moved(precision, 0.005, 9600)
    t_h, t_b = _sort_ms(lib, healthy.ps), _sort_ms(lib, blown.ps)
    print(f"{precision}: sort {1e3 * t_h:.1f} us in place, {1e3 * t_b:.1f} us blown up")
    assert t_b < 3.5 * t_h
