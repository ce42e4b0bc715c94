"""The component-parallel split 3D kernels at the sizes where their float4 walk can go
wrong, and recorded steps against single ones."""
import numpy as np
import pytest
import torch

from oracle import fdtd as O
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
POLES = [(1.1, 0.1, 0.6), (0.0, 0.2, 1.0, 0.8)]


def _problem(shape, poles):
    from meep_torch_b200.core.monitors_3d import PointSource3D
    from meep_torch_b200.core.sources import GaussianPulse
    from meep_torch_b200.core.stepper_3d import build_3d_coeffs, init_3d_state
    nx, ny, nz = shape
    dx, npml = 0.05, 1
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    eps = (1.0 + 3.0 * rng.random(shape)).astype(np.float32)
    masks = [(rng.random(shape) < 0.5).astype(np.float32) for _ in poles]
    kw = dict(poles=poles, pole_masks=[torch.from_numpy(m) for m in masks]) if poles else {}
    okw = dict(poles=poles, pole_masks=masks) if poles else {}
    c = build_3d_coeffs(nx, ny, nz, dx, eps=torch.from_numpy(eps), npml=npml, device="cuda", **kw)
    oc = O.coeffs_3d(nx, ny, nz, dx, eps=eps, npml=npml, dtype=np.float32, **okw)
    s0 = O.state_3d(oc)
    for k in FIELDS:
        s0[k] = rng.standard_normal(s0[k].shape).astype(np.float32)
    init = init_3d_state(nx, ny, nz, npml=npml, n_poles=len(poles), device="cuda")
    init = init._replace(**{k: torch.from_numpy(s0[k]).cuda() for k in FIELDS})
    src = PointSource3D(c.dt, "Ey", nx // 2, 0, nz // 2, GaussianPulse(1.0, 2.0))
    return c, oc, s0, init, src, ("Ey", nx // 2, 0, nz // 2)


# a plane smaller than a warp, rows that start mid-warp (zpitch 8, 12), a row of more than
# one block, a last block of one float4, padding columns in the last float4 of a row
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 5, 7), (5, 43, 12), (4, 3, 530), (3, 129, 4)])
@pytest.mark.parametrize("poles", [[], POLES])
def test_split_kernels_match_oracle(shape, poles):
    """12 float32 steps from random fields: each step rounds a value about a dozen times, so
    sqrt(12 * 12) * 2^-24 ~ 1e-6 relative; 1e-5 leaves a factor of ten."""
    from meep_torch_b200.core.monitors_3d import run_3d
    c, oc, s0, init, src, osrc = _problem(shape, poles)
    st, _ = run_3d(init, c, 12, source=src, variant=2)
    prof = O.gaussian_pulse(1.0, 2.0)
    os_, _ = O.run_3d(s0, oc, 12, amp_fn=lambda t: prof(O.src_time(t, oc["dt"])), src=osrc)
    bad = {}
    for k, v in st._asdict().items():
        if v is not None and v.numel() and k in os_:
            e = rel_l2(v.cpu().numpy(), os_[k])
            if not e < 1e-5:
                bad[k] = e
    assert not bad, bad


@pytest.mark.parametrize("shape,poles", [((5, 43, 12), []), ((6, 9, 70), POLES)])
def test_recorded_steps_equal_single_steps(shape, poles):
    """run_record keeps E before and after every step, bit for bit what runs of one step
    leave in the live buffers, and ends in the same state."""
    from meep_torch_b200.engine3d import Engine3D
    c, _, _, init, src, _ = _problem(shape, poles)
    a, b = Engine3D(init, c, src), Engine3D(init, c, src)
    k = 5
    rec = torch.full((k + 1, 3, a.nx, a.ny, a.zp), float("nan"), device="cuda")
    for t, v in enumerate(a.live_e()):
        assert torch.isfinite(v).all()
    want = [[v.clone() for v in b.live_e()]]
    a.run_record(3, k, rec)
    for q in range(k):
        b.run(3 + q, 1)
        want.append([v.clone() for v in b.live_e()])
    for q in range(k + 1):
        for cc in range(3):
            assert torch.equal(rec[q, cc], want[q][cc]), (q, cc)
    fa, fb = a.fields(), b.fields()
    for key in fa:
        assert torch.equal(fa[key], fb[key]), key
    a.close()
    b.close()


def test_default_kernel_choice_gives_the_same_results():
    """A grid on each side of the rule's lines (cells, row fill): the default equals the
    split kernels bit for bit."""
    from meep_torch_b200.core.monitors_3d import run_3d
    for shape in ((12, 20, 200), (160, 212, 250)):
        c, _, _, init, src, _ = _problem(shape, [])
        x, _ = run_3d(init, c, 3, source=src)
        y, _ = run_3d(init, c, 3, source=src, variant=2)
        for k, v in x._asdict().items():
            if v is not None:
                assert torch.equal(v, getattr(y, k)), (shape, k)
