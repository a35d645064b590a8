"""Neighbour rows of the FP64 form: every form of row against the oracle, bit for bit.

Rows have a fixed pitch; a particle with more neighbours than the pitch walks the cells instead.
It must round exactly like a listed row, which the other FP64 tests cover at lattice densities.
The loops form most products, quotients and roots on the integer pipes; operands that those
leave out (zero, or far from 1) must give the same bits through the FP64 unit.
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


def _fast(d, speed):
    """The column split in two, the right half moving at `speed` (the dambreak's fluid block)."""
    b = d["Blocks"][0]
    w = b["size"][0] / 2
    b["size"][0] = w
    r = copy.deepcopy(b)
    r["translation"] = [b["translation"][0] + w] + b["translation"][1:]
    r["velocity"] = [speed, 0.5 * speed, 0.0]
    d["Blocks"].append(r)
    return d


ODD = {
    # a lattice at rest: separations, velocity differences and pressures that are exactly zero
    "lattice2d": lambda: (small_dambreak_2d(jitter=0.0, viscosity=0.0, corr=1), WC, 3),
    "lattice3d": lambda: (small_dambreak_3d(jitter_frac=0.0, spacing=0.025), WC, 2),
    "column_lattice": lambda: (small_column(2, jitter_frac=0.0, corr=1), SOIL, 2),
    "column_dp_lattice": lambda: (small_column(3, jitter_frac=0.0, xsph=True), SOIL, 2),
    # speeds inside, beyond and far beyond the integer product's range (2^257 = 2e77)
    "speed_1e-60": lambda: (_fast(small_dambreak_2d(xsph=True), 1e-60), WC, 2),
    "speed_1e-100": lambda: (_fast(small_dambreak_2d(corr=1), 1e-100), WC, 2),
    "speed_1e90": lambda: (_fast(small_dambreak_2d(corr=1, integration=1), 1e90), WC, 1),
    "speed_1e160": lambda: (_fast(small_dambreak_2d(integration=1), 1e160), WC, 1),
    "soil_1e90": lambda: (_fast(small_column(2), 1e90), SOIL, 1),
    # a support far from 1 m
    "spacing_1e-6": lambda: (small_dambreak_2d(spacing=1e-6, width=3e-5, height=2e-5, jitter=1e-8, dt=1e-9,
                                               domain=(6e-5, 4e-5)), WC, 2),
}


@pytest.mark.parametrize("scene", sorted(ODD))
def test_operands_outside_the_integer_pipes(oracle_lib, native, scene):
    d, names, steps = ODD[scene]()
    _check(d, oracle_lib, names, steps)


@pytest.mark.parametrize("spacing,size,domain", [
    (0.0085, (0.5, 0.3, 0.2), (0.9, 0.5, 0.25)),  # 113 k rows: three a warp
    (0.02, (0.3, 0.2, 0.02), (0.6, 0.4, 0.02)),   # three cells in z: none is left out
    (0.02, (0.3, 0.2, 0.08), (0.6, 0.4, 0.08)),   # few cells in z, some left out
])
def test_row_builder_in_3d(oracle_lib, native, spacing, size, domain):
    _check(small_dambreak_3d(spacing=spacing, size=size, domain=domain), oracle_lib, WC, 2)
