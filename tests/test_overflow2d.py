"""Runs that overflow: conducting walls are never updated, so they keep their zeros in every
2D kernel while the fields beside them turn infinite or NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(pol, nx, ny, npml, variant):
    from meep_torch_b200.core.coeffs import build_te_coeffs, build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor
    from meep_torch_b200.core.sources import GaussianPulse, LineSource, TESource
    from meep_torch_b200.core.stepper_te import init_te_state
    from meep_torch_b200.core.stepper_tm import init_tm_state
    from meep_torch_b200.engine2d import Engine2D
    rng = np.random.default_rng(nx + ny)
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    # a wave speed of 7 against a step made for 1: every step multiplies the fields
    eps = torch.full((nx, ny), 0.02, device="cuda")
    src = LineSource(g, ix=nx // 2, j0=2, j1=ny - 2, profile=GaussianPulse(0.6, 0.4))
    if pol == "tm":
        s, c, f = init_tm_state(g), build_tm_coeffs(g, eps_inf=eps, npml=npml), "Hx"
    else:
        s, c, f = init_te_state(g), build_te_coeffs(g, eps_inf=eps, npml=npml), "Hz"
        src = TESource(src)
    s = s._replace(**{f: torch.from_numpy(rng.standard_normal(getattr(s, f).shape)
                                          .astype(np.float32)).cuda()})
    e = Engine2D([(s, c, src, [DFTFieldsMonitor(g, [0.5], "Ez" if pol == "tm" else "Ex")])],
                 variant=variant)
    e.run(0, 60)
    out = e.state(0)
    e.close()
    return out


@pytest.mark.parametrize("pol", ["tm", "te"])
@pytest.mark.parametrize("shape", [(60, 50, 0), (75, 250, 8), (300, 301, 10)])
def test_walls_keep_their_values(pol, shape):
    outs = {}
    for variant in (0, 3):
        o = outs[variant] = _run(pol, *shape, variant)
        walls = ([o.Dz[0], o.Dz[-1], o.Dz[:, 0], o.Dz[:, -1]] if pol == "tm"
                 else [o.Dx[:, 0], o.Dx[:, -1], o.Dy[0], o.Dy[-1]])
        inner = o.Dz[1:-1, 1:-1] if pol == "tm" else o.Hz
        assert not torch.isfinite(inner).any(), variant
        for q, w in enumerate(walls):
            assert bool((w == 0).all()), (variant, q)
    if pol == "te" or shape[1] == 301:      # not a plan that rounds as the cluster kernel does
        for k, v in outs[0]._asdict().items():
            if torch.is_tensor(v) and v.numel():
                torch.testing.assert_close(v, getattr(outs[3], k), rtol=0, atol=0,
                                           equal_nan=True, msg=k)
