"""The cluster kernel (variant 4, and the default for batches of small TM structures that the
resident kernel cannot take) and the resident kernel that stands in for it: which of them
runs, and that they give the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _item(nx, ny, npml, seed=0):
    from meep_torch_b200.core.coeffs import build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor, FluxMonitorTM
    from meep_torch_b200.core.sources import GaussianPulse, LineSource
    from meep_torch_b200.core.stepper_tm import init_tm_state
    rng = np.random.default_rng(nx * 7 + ny + seed)
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    eps = torch.from_numpy((1 + 5 * rng.random((nx, ny))).astype(np.float32)).cuda()
    s = init_tm_state(g)
    s = s._replace(**{k: torch.from_numpy(0.1 * rng.standard_normal(getattr(s, k).shape)
                                          .astype(np.float32)).cuda() for k in ("Hx", "Hy")})
    f = [0.5, 0.6, 0.7]
    mons = [FluxMonitorTM(g, f, x_normal=True, idx=3 * nx // 4, lo=1, hi=ny - 1),
            FluxMonitorTM(g, f, x_normal=False, idx=ny // 3, lo=1, hi=nx - 1),
            DFTFieldsMonitor(g, f, "Ez")]
    src = LineSource(g, ix=nx // 4, j0=ny // 4, j1=ny - ny // 4, profile=GaussianPulse(0.6, 0.3))
    return s, build_tm_coeffs(g, eps_inf=eps, npml=npml), src, mons


def _run(batch, variant, graph):
    """Outputs of 81 steps and the names of the kernels that advanced all but the first."""
    from meep_torch_b200.engine2d import Engine2D
    e = Engine2D([_item(*b) for b in batch], variant=variant, ring_slots=16, graph=graph)
    e.run(0, 1)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        e.run(1, 47)
        e.run(48, 33)
        torch.cuda.synchronize()
    names = {k for k in ("k_cl_tm", "k_rb_resident", "k_tb_tm", "k_tile_tm")
             if any(k in ev.key for ev in prof.key_averages())}
    out = []
    for b in range(len(batch)):
        out += [v.clone() for v in e.state(b) if torch.is_tensor(v) and v.numel()]
        out += [a.clone() for a in e.accumulators(b)]
    e.close()
    return out, names


# the 320 x 160 cavity and shapes whose rows or columns do not split evenly
@pytest.mark.parametrize("shape", [(320, 160, 10), (77, 50, 10), (30, 301, 6), (200, 96, 0)])
@pytest.mark.parametrize("graph", [False, True])
def test_resident_equals_cluster(shape, graph):
    cl, k4 = _run([shape], 4, graph)
    rb, k0 = _run([shape], 0, graph)
    assert k4 == {"k_cl_tm"} and k0 == {"k_rb_resident"}, (k4, k0)
    for q, (x, y) in enumerate(zip(cl, rb)):
        assert torch.equal(x, y), q


@pytest.mark.parametrize("graph", [False, True])
def test_batch_past_the_resident_limit_runs_the_cluster_kernel(graph):
    # five structures of 33 tiles: more than an SM each, at most one cluster per 16 SMs
    batch = [(256, 256, 12, b) for b in range(5)]
    got, k0 = _run(batch, 0, graph)
    assert k0 == {"k_cl_tm"}, k0
    one = [v for b in batch for v in _run([b], 4, graph)[0]]
    for q, (x, y) in enumerate(zip(got, one)):
        assert torch.equal(x, y), q
