"""Reading a plan's accumulators while another thread captures a CUDA graph: neither notices
the other (a capture in the default mode forbids synchronising calls to every thread)."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("finished", [True, False])
def test_accumulators_during_another_threads_capture(finished):
    from meep_torch_b200.core.coeffs import build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor
    from meep_torch_b200.core.sources import GaussianPulse, LineSource
    from meep_torch_b200.core.stepper_tm import init_tm_state
    from meep_torch_b200.engine2d import Engine2D
    nx, ny = 200, 120
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    m = build_tm_coeffs(g, eps_inf=torch.full((nx, ny), 2.0, device="cuda"), npml=8)
    src = LineSource(g, ix=20, j0=10, j1=50, profile=GaussianPulse(0.6, 0.4))
    e = Engine2D([(init_tm_state(g), m, src, [DFTFieldsMonitor(g, [0.5], "Ez")])])
    x = torch.ones(8, device="cuda")
    inside, leave, errors, graphs = threading.Event(), threading.Event(), [], []

    def capture():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                y = x + 1
                inside.set()
                leave.wait(60)
                y = y + 1
            graphs.append((graph, y))
        except Exception as err:      # a thread's exception would go unseen
            errors.append(repr(err))
            inside.set()

    t = threading.Thread(target=capture)
    e.run(0, 64 if finished else 4000)
    if finished:
        torch.cuda.synchronize()
    t.start()
    assert inside.wait(60)
    try:
        accs = e.accumulators(0)
    finally:
        leave.set()
        t.join()
    assert not errors, errors
    graph, y = graphs[0]
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 3).all()) and bool(torch.isfinite(accs[0]).all())
    e.close()
