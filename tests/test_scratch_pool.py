"""Plan scratch is reused from one plan to the next: the same results whatever an earlier plan
left in it, from several threads at once, and given back on request."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(pol, nx, ny, steps):
    from meep_torch_b200.core.coeffs import build_te_coeffs, build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor, FluxMonitorTM
    from meep_torch_b200.core.sources import GaussianPulse, LineSource, TESource
    from meep_torch_b200.core.stepper_te import init_te_state
    from meep_torch_b200.core.stepper_tm import init_tm_state
    from meep_torch_b200.engine2d import Engine2D
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    eps = torch.full((nx, ny), 2.5, device="cuda")
    src = LineSource(g, ix=nx // 2, j0=9, j1=ny - 9, profile=GaussianPulse(0.6, 0.4))
    f = [0.5, 0.6, 0.7]
    if pol == "tm":
        item = (init_tm_state(g), build_tm_coeffs(g, eps_inf=eps, npml=8), src,
                [DFTFieldsMonitor(g, f, "Ez"),
                 FluxMonitorTM(g, f, x_normal=True, idx=nx // 3, lo=1, hi=ny - 1)])
    else:
        item = (init_te_state(g), build_te_coeffs(g, eps_inf=eps, npml=8), TESource(src),
                [DFTFieldsMonitor(g, f, "Hz")])
    e = Engine2D([item])
    e.run(0, steps)
    out = [a.clone() for a in e.accumulators(0)] + [e.state(0)[0].clone()]
    e.close()
    return out


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


def test_reused_scratch_gives_the_same_results():
    from meep_torch_b200 import _lib as L
    L.load().mtb_release_scratch()
    first = {k: _run(*k) for k in (("tm", 90, 70, 40), ("te", 200, 333, 70))}
    for k in (("tm", 400, 500, 33), *first, ("tm", 90, 70, 5), *first):
        out = _run(*k)
        assert k not in first or _same(out, first[k]), k


def test_threads_share_the_pool():
    want, bad = _run("tm", 120, 100, 64), []

    def work():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(12):
                    if not _same(_run("tm", 120, 100, 64), want):
                        bad.append("differs")
                torch.cuda.current_stream().synchronize()
        except Exception as e:      # a thread's exception would go unseen
            bad.append(repr(e))

    ts = [threading.Thread(target=work) for _ in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad


def test_kept_memory_is_bounded_and_given_back():
    from meep_torch_b200 import _lib as L
    lib = L.load()
    lib.mtb_release_scratch()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    for n in (300, 700, 1100, 1500):
        _run("tm", n, n, 3)
    torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info()[0] <= (256 << 20) + (64 << 20)
    lib.mtb_release_scratch()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20
