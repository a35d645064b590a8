"""The FP64 form without neighbour rows (a scene whose rows would not fit the free memory): every
loop walks the cells, in blocks of another shape, and rounds exactly like the oracle."""
import ctypes

import numpy as np
import pytest

from helpers import cfg_of, describe_diff, small_column, small_dambreak_2d, small_dambreak_3d
from tisphi_gb300 import scenes

pytestmark = pytest.mark.gpu

WC = ["x", "v", "density", "m_V", "pressure", "CSPM_f", "id0"]
SOIL = WC + ["stress", "strain_equ", "strain_equ_p"]


def _without_rows(cfg):
    """A Simulation whose handle is bound to no row memory at all."""
    from tisphi_gb300 import _native as nat
    from tisphi_gb300.simulation import Simulation
    sim = Simulation(cfg)
    lib, ps = nat.load(), sim.ps
    h = ctypes.c_void_p()
    nat.check(lib.tsg_create(ctypes.byref(ps._cfg), ctypes.byref(h)), "tsg_create")
    lib.tsg_limit_rows.argtypes = [ctypes.c_void_p, ctypes.c_int64]
    nat.check(lib.tsg_limit_rows(h, 0), "tsg_limit_rows")
    parts, keep = nat.host_particles(ps.scene)
    nat.check(lib.tsg_upload(h, ctypes.byref(parts), 0, None), "tsg_upload")
    lib.tsg_destroy(ps._h)
    ps._h = sim.solver._h = h
    return sim


def _bdy(d, mode):
    d["Configuration"]["boundary"] = mode
    return d


SCENES = {
    "wc2d_cspm_xsph": lambda: (small_dambreak_2d(corr=1, xsph=True), WC),
    "wc2d_rk4_cubic_cspm": lambda: (small_dambreak_2d(integration=4, kernel=0, corr=1), WC),
    "wc2d_repulsive": lambda: (_bdy(small_dambreak_2d(), 4), WC),
    "wc2d_collision": lambda: (_bdy(small_dambreak_2d(), 1), WC),
    "wc3d_cspm": lambda: (small_dambreak_3d(corr=1, spacing=0.025), WC),
    "wc3d_plain": lambda: (small_dambreak_3d(corr=0, spacing=0.025), WC),
    "rigid2d": lambda: (scenes.floating_box_2d(), WC),
    "mui_cspm": lambda: (small_column(2, corr=1), SOIL),
    "mui_lf": lambda: (small_column(2, integration=2), SOIL),
    "dp_lf_xsph": lambda: (small_column(3, integration=2, xsph=True), SOIL),
    "dp_cspm": lambda: (small_column(3, corr=1), SOIL),
}


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_steps_without_rows(oracle_lib, native, scene):
    """Two steps launched one by one, then a graph of two."""
    d, names = SCENES[scene]()
    cfg = cfg_of(d)
    sim = _without_rows(cfg)
    orc = oracle_lib.OracleSim(cfg)
    sim.solver.step(4)
    orc.step(4)
    bad = []
    for nm in names:
        a = sim.ps.field(nm).cpu().numpy().astype(np.float64)
        b = orc.get(nm)
        if not np.all((a == b) | (np.isnan(a) & np.isnan(b))):
            bad.append(describe_diff(nm, a, b))
    assert not bad, "; ".join(bad)


@pytest.mark.parametrize("scene", ["wc2d_cspm_xsph", "mui_cspm", "dp_lf_xsph"])
def test_stage_calls_without_rows(oracle_lib, native, scene):
    d, names = SCENES[scene]()
    cfg = cfg_of(d)
    sim = _without_rows(cfg)
    orc = oracle_lib.OracleSim(cfg)
    s = sim.solver
    for _ in range(2):
        sim.ps.initialize_particle_system()
        s.calc_kernel_corr()
        s.init_real2tmp()
        s.substep()
        s.advect_pos()
        s.advect_something()
    orc.step(2)
    for nm in names:
        a = sim.ps.field(nm).cpu().numpy().astype(np.float64)
        assert np.array_equal(a, orc.get(nm)), describe_diff(nm, a, orc.get(nm))
