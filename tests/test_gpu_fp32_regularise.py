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
