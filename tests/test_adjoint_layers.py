"""The 2D adjoint with d J / d psi kept on the CPML bands only: the eps gradient's own bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grad(pol, nx, ny, npml):
    from meep_torch_b200.core.coeffs import build_te_coeffs, build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor
    from meep_torch_b200.core.run import run_te, run_tm
    from meep_torch_b200.core.sources import GaussianPulse, LineSource, TESource
    from meep_torch_b200.core.stepper_te import init_te_state
    from meep_torch_b200.core.stepper_tm import init_tm_state
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    rng = np.random.default_rng(nx + ny)
    eps = torch.from_numpy((1 + 3 * rng.random((nx, ny))).astype(np.float32)).cuda()
    eps.requires_grad_(True)
    src = LineSource(g, ix=nx // 2, j0=1, j1=ny - 1, profile=GaussianPulse(0.6, 0.4))
    if pol == "tm":
        m, s = build_tm_coeffs(g, eps_inf=eps, npml=npml), init_tm_state(g)
        mon, run = DFTFieldsMonitor(g, [0.6], "Ez"), run_tm
    else:
        m, s = build_te_coeffs(g, eps_inf=eps, npml=npml), init_te_state(g)
        mon, run, src = DFTFieldsMonitor(g, [0.6], "Hz"), run_te, TESource(src)
    _, (acc,) = run(s, m, 90, source=src, monitors=[mon], checkpoint_every=40)
    acc.abs().square().sum().backward()
    return eps.grad


# no layers, layers that end inside a lane's four columns, layers that meet, one-row remainders
@pytest.mark.parametrize("pol", ["tm", "te"])
@pytest.mark.parametrize("nx, ny, npml", [(33, 40, 0), (41, 131, 7), (24, 30, 11), (65, 260, 10)])
def test_layers_only_gives_the_same_gradient(pol, nx, ny, npml, monkeypatch):
    from meep_torch_b200 import _lib as L
    part = _grad(pol, nx, ny, npml)
    monkeypatch.setattr(L.load(), "mtb_yee2d_adjoint_psi_layers", lambda p, on: 0)
    full = _grad(pol, nx, ny, npml)
    assert torch.isfinite(full).all() and full.abs().max() > 0
    assert torch.equal(part, full)
