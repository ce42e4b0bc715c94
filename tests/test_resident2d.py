"""The resident 2D kernel against the temporally blocked kernels it stands in for: the same
rounding, so the same bits, on plans whose tiles end in every way."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _item(pol, nx, ny, npml):
    from meep_torch_b200.core.coeffs import build_te_coeffs, build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import (DFTFieldsMonitor, FluxMonitorTE, FluxMonitorTEY,
                                               FluxMonitorTM)
    from meep_torch_b200.core.sources import GaussianPulse, LineSource, TESource
    from meep_torch_b200.core.stepper_te import init_te_state
    from meep_torch_b200.core.stepper_tm import init_tm_state
    rng = np.random.default_rng(nx * 31 + ny)
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    eps = torch.from_numpy((1 + 5 * rng.random((nx, ny))).astype(np.float32)).cuda()
    # the source line crosses tile columns; its row is the last or first of a tile's block
    src = LineSource(g, ix=nx // 2 // 24 * 24, j0=2, j1=ny - 2, profile=GaussianPulse(0.6, 0.4))
    f = [0.5, 0.7]
    if pol == "tm":
        m, s = build_tm_coeffs(g, eps_inf=eps, npml=npml), init_tm_state(g)
        mons = [FluxMonitorTM(g, f, x_normal=True, idx=min(24, nx - 2), lo=1, hi=ny - 1),
                FluxMonitorTM(g, f, x_normal=False, idx=min(120, ny - 2), lo=0, hi=nx),
                DFTFieldsMonitor(g, f, "Hx")]
        names = ("Hx", "Hy")
    else:
        m, s = build_te_coeffs(g, eps_inf=eps, npml=npml), init_te_state(g)
        mons = [FluxMonitorTE(g, f, ix=min(24, nx - 2), lo=1, hi=ny - 1),
                FluxMonitorTEY(g, f, iy=min(120, ny - 2), lo=0, hi=nx - 1),
                DFTFieldsMonitor(g, f, "Ey")]
        src, names = TESource(src), ("Hz",)
    s = s._replace(**{k: torch.from_numpy(rng.standard_normal(getattr(s, k).shape)
                                          .astype(np.float32)).cuda() for k in names})
    return s, m, src, mons


# one tile row and several, a last tile of one row, columns that end inside the first lane of
# a tile, no layers at all, the largest resident grid and one just past it (148 tiles of 24
# rows), a batch of both polarisations
@pytest.mark.parametrize("batch", [
    [("te", 20, 9, 2)], [("te", 25, 121, 4)], [("te", 73, 245, 0)], [("te", 97, 480, 10)],
    [("tm", 300, 301, 10)], [("tm", 241, 365, 0)], [("te", 888, 479, 20)],
    [("te", 889, 481, 20)], [("tm", 100, 700, 12), ("te", 50, 130, 5), ("te", 49, 127, 5)]])
@pytest.mark.parametrize("graph", [False, True])
def test_resident_equals_temporally_blocked(batch, graph):
    from meep_torch_b200.engine2d import Engine2D
    outs = []
    for variant in (3, 0):
        e = Engine2D([_item(*b) for b in batch], variant=variant, ring_slots=10, graph=graph)
        e.run(0, 27)
        e.run(27, 6)
        outs.append(([e.state(b) for b in range(len(batch))],
                     [[a.clone() for a in e.accumulators(b)] for b in range(len(batch))]))
        e.close()
    for b in range(len(batch)):
        for k, v in outs[0][0][b]._asdict().items():
            if torch.is_tensor(v) and v.numel():
                assert torch.equal(v, getattr(outs[1][0][b], k)), (b, k)
        for q, (x, y) in enumerate(zip(outs[0][1][b], outs[1][1][b])):
            assert torch.equal(x, y), (b, q)
