"""mu(I) stress regularisation of the FP32-mixed form: the step sequence, which reads the
neighbours' stress from the momentum pass's records, against the stage calls, which read the
stress planes; and the signs of the zeros in 2D."""
import numpy as np
import pytest

from helpers import cfg_of, small_column

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("corr", [0, 1])
def test_step_equals_stage_calls_bit_for_bit(native, corr):
    """Equal sums in the same order: equal bits, those of zeros included (no tolerance)."""
    from tisphi_gb300.simulation import Simulation
    a, b = (Simulation(cfg_of(small_column(2, corr=corr)), precision="fp32_mixed") for _ in range(2))
    a.solver.step(3)
    s = b.solver
    b.ps.initialize_particle_system()
    for _ in range(3):  # (no particle moves far enough for a rebuild)
        s.calc_kernel_corr()
        s.init_real2tmp()
        s.substep()
        s.advect_pos()
        s.advect_something()
    ia, ib = (np.argsort(q.ps.field("id0").cpu().numpy()) for q in (a, b))
    for nm in ("x", "v", "density", "stress"):
        x = a.ps.field(nm).cpu().numpy()[ia]
        y = b.ps.field(nm).cpu().numpy()[ib]
        np.testing.assert_array_equal(x.view(np.int64), y.view(np.int64), err_msg=nm)


def test_out_of_plane_shears_are_positive_zeros(native):
    """Sums of +-0 that start at +0 are +0; the CSV and VTK exports print the sign."""
    from tisphi_gb300.simulation import Simulation
    sim = Simulation(cfg_of(small_column(2)), precision="fp32_mixed")
    sim.solver.step(12)
    soil = sim.ps.field("mat_type").cpu().numpy() == 2
    st = sim.ps.field("stress").cpu().numpy()[soil].reshape(-1, 3, 3)
    assert np.any(st[:, 0, 0] < 0)  # compressed, where 0 times xx is -0
    for a, b in ((0, 2), (1, 2), (2, 0), (2, 1)):
        assert not st[:, a, b].any() and not np.signbit(st[:, a, b]).any()


def _column_3d():
    d = small_column(2, spacing=0.008, width=0.1, height=0.05, domain=(0.2, 0.08))
    d["Configuration"]["is2D"] = False
    d["Configuration"]["domainEnd"] = [0.2, 0.08, 0.048]
    d["Blocks"][0]["size"] = [0.1, 0.05, 0.048]
    return d


@pytest.mark.parametrize("skin", [0.05, 1e-6, 0.0])
@pytest.mark.parametrize("dim", [2, 3])
def test_steps_by_lists_and_by_enumeration(oracle_lib, native, dim, skin):
    """The neighbours from the lists; from the cells because every particle has moved too far for a
    tiny skin; and from the cells because there is no skin: the oracle's stress at the bound of the
    granular columns, 1e-4 of the largest entry."""
    from tisphi_gb300.simulation import Simulation
    d = _column_3d() if dim == 3 else small_column(2)
    d["Configuration"]["neighbourSkin"] = skin
    cfg = cfg_of(d)
    sim = Simulation(cfg, precision="fp32_mixed")
    orc = oracle_lib.OracleSim(cfg)
    sim.solver.step(12)
    orc.step(12)
    gid = sim.ps.field("id0").cpu().numpy()
    take = np.empty_like(gid)
    take[gid] = np.arange(gid.size)
    take = take[orc.get("id0").astype(np.int64)]
    f = orc.get("mat_type") == 2
    a = sim.ps.field("stress").cpu().numpy().astype(np.float64)[take][f].reshape(-1, 9)
    b = orc.get("stress")[f].reshape(-1, 9)
    assert np.max(np.abs(b)) > 0
    assert np.max(np.abs(a - b)) / np.max(np.abs(b)) < 1e-4
