"""FP32-mixed scenes above the sizes up to which small scenes take kernels of their own: the rates
pass with two records per trip (more than 19,456 dynamic particles) and the list builds of larger
scenes (in 2D a thread per particle above 65,536 particles), against the f64 oracle at the bounds
of the small scenes (density 1e-5 relative, positions 1e-6 m), and the WCSPH adjoint with a thread
per particle (above 65,536) against central finite differences of the FP64 form."""
import numpy as np
import pytest
import torch

from helpers import cfg_of, small_dambreak_2d, small_dambreak_3d

pytestmark = pytest.mark.gpu

SCENES = {
    # name: (scene, least dynamic particles, least particles)
    "2d": (lambda: small_dambreak_2d(spacing=0.003), 19457, 0),
    "2d_cspm_cubic": (lambda: small_dambreak_2d(spacing=0.003, corr=1, kernel=0), 19457, 0),
    "2d_lists": (lambda: small_dambreak_2d(spacing=0.0019), 19457, 65537),
    "3d_cspm": (lambda: small_dambreak_3d(spacing=0.01, size=(0.4, 0.3, 0.2), domain=(0.6, 0.4, 0.2)), 19457, 0),
}


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_steps_of_larger_scenes(oracle_lib, native, scene):
    from tisphi_gb300.simulation import Simulation
    make, least_flow, least = SCENES[scene]
    cfg = cfg_of(make())
    sim = Simulation(cfg, precision="fp32_mixed")
    orc = oracle_lib.OracleSim(cfg)
    sim.solver.step(3)
    orc.step(3)
    gid = sim.ps.field("id0").cpu().numpy()
    take = np.empty_like(gid)
    take[gid] = np.arange(gid.size)
    take = take[orc.get("id0").astype(np.int64)]
    f = orc.get("mat_type") == 1
    assert f.sum() >= least_flow and f.size >= least
    rho, rho_o = (sim.ps.field("density").cpu().numpy().astype(np.float64)[take][f], orc.get("density")[f])
    x, x_o = sim.ps.field("x").cpu().numpy().astype(np.float64)[take][f], orc.get("x")[f]
    assert np.max(np.abs(rho - rho_o) / rho_o) < 1e-5
    assert np.max(np.abs(x - x_o)) < 1e-6


def test_wc_adjoint_of_a_larger_scene(native):
    """Gradient of the front's distance over 30 steps: 1e-3, the agreement the forms are held to."""
    from tisphi_gb300 import scenes
    from tisphi_gb300.adjoint import WCRollout, distal_loss, rollout_positions
    d = scenes.dambreak_2d(spacing=0.0033, width=1.2, height=0.6, integration=1)
    model = WCRollout(d, nsteps=30, checkpoint_every=10)
    assert model.n > 65536
    B0, nu0 = model.stiffness, model.viscosity
    params = torch.tensor([B0, nu0], dtype=torch.float64, requires_grad=True)
    loss, sel = distal_loss(model(params), target=1.3)
    loss.backward()
    fd = []
    for k, delta in ((0, 1e-3 * B0), (1, 1e-3 * nu0)):
        lo, hi = [B0, nu0], [B0, nu0]
        lo[k] -= delta
        hi[k] += delta
        l_hi, _ = distal_loss(rollout_positions(d, 30, *hi), target=1.3, sel=sel)
        l_lo, _ = distal_loss(rollout_positions(d, 30, *lo), target=1.3, sel=sel)
        fd.append((float(l_hi) - float(l_lo)) / (2 * delta))
    fd = torch.tensor(fd, dtype=torch.float64)
    rel = (params.grad.cpu() - fd).abs() / fd.abs()
    assert torch.all(rel < 1e-3), f"adjoint {params.grad.tolist()} central FD {fd.tolist()}"
