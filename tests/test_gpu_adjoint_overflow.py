"""tsg_adjoint_step on a state whose neighbour lists overflow: TSG_E_CAPACITY, with the state of
the handle and the caller's arrays as they were."""
import copy

import pytest
import torch

from tisphi_gb300 import scenes

pytestmark = pytest.mark.gpu


def _dense(method):
    """A second block over the first, offset by half a spacing: twice the neighbours."""
    d = (scenes.dambreak_2d(spacing=0.02, width=0.3, height=0.2, domain=(0.6, 0.4), integration=1) if method == 1
         else scenes.column_2d(method=2, spacing=0.004, dt=2e-5))
    h = d["Configuration"]["particleRadius"]
    b = copy.deepcopy(d["Blocks"][0])
    b["translation"] = [b["translation"][0] + h, b["translation"][1] + h, b["translation"][2]]
    b["velocity"] = [0.1, -0.05, 0.0]
    d["Blocks"].append(b)
    return d


@pytest.mark.parametrize("method", [1, 2])
def test_overflow_leaves_everything_as_it_was(native, method):
    from tisphi_gb300.adjoint import MuIRollout, WCRollout, _ptr
    from tisphi_gb300.particle_system import _stream
    model = (WCRollout if method == 1 else MuIRollout)(_dense(method), nsteps=4)
    model.load(model.initial)
    model.step(1)
    start = model.save()

    def state():
        ids = model.ps.field("id0").long()
        out = {}
        for nm in ["x", "v", "density", "pressure"] + (["stress"] if method == 2 else []):
            f = model.ps.field(nm)
            out[nm] = torch.empty_like(f)
            out[nm][ids] = f
        return out

    model.load(start)
    before = state()
    n = model.n
    g = torch.Generator(device="cuda").manual_seed(1)
    arrays = [torch.randn(s, dtype=torch.float64, device="cuda", generator=g) for s in ((n, 3), (n, 3), (n,), (n, 3), (2,))]
    kept = [a.clone() for a in arrays]
    for _ in range(2):
        rc = native.tsg_adjoint_step(model._h, *[_ptr(a) for a in arrays], _stream())
        assert rc == -7  # TSG_E_CAPACITY
        assert model.ps.list_stats()["overflowed"] > 100
        after = state()
        for nm in before:
            assert torch.equal(before[nm], after[nm]), nm
        assert all(torch.equal(a, b) for a, b in zip(arrays, kept))
    # and the handle steps on as from the state itself
    model.step(2)
    x1 = state()
    model.load(start)
    model.step(2)
    x2 = state()
    assert all(torch.equal(x1[nm], x2[nm]) for nm in x1)
