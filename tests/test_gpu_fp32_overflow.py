"""Scenes in which most lists overflow (a second block over the first: twice the neighbours), above
the number of threads that one wave of the overflow pass has: every overflowed particle is served,
by whichever trip of the pass reaches it, and the values are the oracle's at the bounds of the
lists' own tests (rates 1e-4 normwise)."""
import copy

import numpy as np
import pytest

from helpers import cfg_of, small_column, small_dambreak_2d, small_dambreak_3d

pytestmark = pytest.mark.gpu


def _dense(d):
    h = d["Configuration"]["particleRadius"]
    b = copy.deepcopy(d["Blocks"][0])
    b["translation"] = [b["translation"][0] + h, b["translation"][1] + h, b["translation"][2]]
    b["velocity"] = [0.1, -0.05, 0.0]
    d["Blocks"].append(b)
    return d


SCENES = {
    "wc2d_cspm": lambda: small_dambreak_2d(spacing=0.0027, corr=1),
    "wc3d_cspm": lambda: small_dambreak_3d(spacing=0.0062),
    "mui2d": lambda: small_column(2, spacing=0.0007, corr=1),
}


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_more_overflowed_lists_than_threads(oracle_lib, native, scene):
    from tisphi_gb300.simulation import Simulation
    cfg = cfg_of(_dense(SCENES[scene]()))
    sim = Simulation(cfg, precision="fp32_mixed")
    orc = oracle_lib.OracleSim(cfg)
    sim.ps.initialize_particle_system()
    orc.sort()
    assert sim.ps.list_stats()["overflowed"] > 64 * 128  # the threads of the pass
    sim.solver.calc_kernel_corr()
    orc.call(oracle_lib.ORC_KERNEL_CORR)
    sim.solver.init_real2tmp()
    orc.call(oracle_lib.ORC_INIT_TMP)
    sim.solver.one_step()
    orc.call(oracle_lib.ORC_ONE_STEP)
    gid = sim.ps.field("id0").cpu().numpy()
    take = np.empty_like(gid)
    take[gid] = np.arange(gid.size)
    take = take[orc.get("id0").astype(np.int64)]
    f = orc.get("mat_type") > 0
    for nm in ("CSPM_f", "d_density", "d_vel"):
        a = sim.ps.field(nm).cpu().numpy().astype(np.float64)[take][f]
        b = orc.get(nm)[f]
        assert np.max(np.abs(a - b)) / np.max(np.abs(b)) < 1e-4, nm
