"""Neighbour rows of the FP64 form: every form of row against the oracle, bit for bit.

Rows have a fixed pitch; a particle with more neighbours than the pitch walks the cells instead.
It must round exactly like a listed row, which the other FP64 tests cover at lattice densities.
"""
import copy

import numpy as np
import pytest

from helpers import cfg_of, describe_diff, small_column, small_dambreak_2d, small_dambreak_3d

pytestmark = pytest.mark.gpu

WC = ["x", "v", "density", "m_V", "pressure", "CSPM_f", "id0"]
SOIL = WC + ["stress", "strain_equ", "strain_equ_p"]


def _dense(d):
    """A second block over the first, offset by half a spacing: about twice the lattice's
    neighbours inside the overlap (more than a row holds), the lattice's at its rim."""
    h = d["Configuration"]["particleRadius"]
    b = copy.deepcopy(d["Blocks"][0])
    b["translation"] = [b["translation"][0] + h, b["translation"][1] + h, b["translation"][2]]
    d["Blocks"].append(b)
    return d


def _check(d, oracle_lib, names, steps):
    from tisphi_gb300.simulation import Simulation
    cfg = cfg_of(d)
    sim = Simulation(cfg)
    orc = oracle_lib.OracleSim(cfg)
    sim.solver.step(steps)
    orc.step(steps)
    bad = []
    for nm in names:
        a = sim.ps.field(nm).cpu().numpy().astype(np.float64)
        b = orc.get(nm)
        if not np.all((a == b) | (np.isnan(a) & np.isnan(b))):
            bad.append(describe_diff(nm, a, b))
    assert not bad, "; ".join(bad)
    return sim


SCENES = {
    "wc2d_cspm_xsph": lambda: (small_dambreak_2d(corr=1, xsph=True), WC),
    "wc2d_rk4_cubic_cspm": lambda: (small_dambreak_2d(integration=4, kernel=0, corr=1), WC),
    "wc3d_cspm": lambda: (small_dambreak_3d(corr=1, spacing=0.025), WC),
    "mui_cspm": lambda: (small_column(2, corr=1), SOIL),
    "mui_lf_cspm": lambda: (small_column(2, integration=2, corr=1), SOIL),
    "dp_lf_xsph": lambda: (small_column(3, integration=2, xsph=True), SOIL),
}


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_rows_above_the_pitch(oracle_lib, native, scene):
    d, names = SCENES[scene]()
    sim = _check(_dense(d), oracle_lib, names, 2)
    counts, _ = sim.ps.neighbors()
    assert counts.max() > (150 if sim.ps.dim == 3 else 45)  # above any pitch of these scenes
