"""The temporally blocked kernels' bounded wait, compiled for the host against scripted
copies and a scripted clock: no thread gives up without the error flag, and none gives up on
copies that have landed."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "meep_torch_b200", "csrc")

HOST = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
struct TbCtl { uint64_t bar; };
struct { unsigned x; } threadIdx;
constexpr unsigned long long WAIT_NS = 1000;
// polls before `lands` fail; the clock jumps by `jump` once, at its second reading
static long polls, lands, reads;
static unsigned long long now, jump;
static bool mbar_try_wait(uint64_t *, uint32_t) { return ++polls > lands; }
static unsigned long long gtimer() { now += 1 + (++reads == 2 ? jump : 0); return now; }
static int atomicExch(int *p, int v) { int o = *p; *p = v; return o; }
%s
int main(int argc, char **argv) {
    threadIdx.x = atoi(argv[1]);
    lands = atol(argv[2]);
    jump = atoll(argv[3]);
    TbCtl ctl{};
    int err = 0;
    const bool ok = tb_wait(ctl, 0, &err);
    printf("%%d %%d\n", (int)ok, err);
}
"""


@pytest.fixture(scope="module")
def wait(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src = open(os.path.join(CSRC, "yee2d_tb.cuh")).read()
    fn = re.search(r"__device__ __forceinline__ bool tb_wait\(.*?\n}\n", src, re.S).group(0)
    d = tmp_path_factory.mktemp("wait")
    (d / "w.cpp").write_text(HOST % fn)
    subprocess.run(["g++", "-O1", "-o", str(d / "w"), str(d / "w.cpp")], check=True)

    def run(thread, lands, jump):
        out = subprocess.run([str(d / "w"), str(thread), str(lands), str(jump)],
                             capture_output=True, text=True, check=True, timeout=60).stdout
        return tuple(int(v) for v in out.split())
    return run


@pytest.mark.parametrize("thread", [0, 1, 31, 1023])
def test_expired_wait_raises_the_flag_in_any_thread(wait, thread):
    assert wait(thread, 1 << 40, 0) == (0, 1)


@pytest.mark.parametrize("thread", [0, 7, 1023])
def test_landed_copies_are_taken(wait, thread):
    assert wait(thread, 0, 0) == (1, 0)          # at once
    assert wait(thread, 40, 0) == (1, 0)         # while waiting
    # between a poll and a reading of the clock that lies past the limit
    assert wait(thread, 2, 5000) == (1, 0)


# ------------------------------------------------------------------ who reads the flag
class _Lib:
    """Every entry point succeeds, but the plans named in ``timed_out`` report a timeout."""

    def __init__(self, timed_out=()):
        self.timed_out = set(timed_out)
        self.pending = False

    def mtb_yee2d_check(self, plan, stream):
        return 3 if plan in self.timed_out else 0

    def mtb_yee2d_poll(self, plan, stream, finished):
        finished._obj.value = not self.pending
        return 0 if self.pending else self.mtb_yee2d_check(plan, stream)

    def mtb_last_error(self):
        return b"a bounded wait expired"

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture
def fake(monkeypatch):
    from meep_torch_b200 import _lib as L
    lib = _Lib()
    monkeypatch.setattr(L, "load", lambda: lib)
    return lib


def _engine(lib, plan, nx=6, ny=8):
    import types

    import torch

    from meep_torch_b200 import _lib as L
    from meep_torch_b200.engine2d import Engine2D
    e = Engine2D.__new__(Engine2D)
    e.lib, e.plan, e.stream, e.device = lib, plan, None, torch.device("cpu")
    e._sptr = lambda: 0
    e.items = [types.SimpleNamespace(nx=nx, ny=ny, accs=[torch.zeros(3)])]
    e.structs = (L.Yee2DStruct * 1)()
    e.structs[0].pitch = ny
    e.regions, e.n_regions = None, 0
    e.groups, e.n_groups, e.ring_elems = None, 0, 0
    e._pack = lambda *a: torch.zeros(nx, ny)
    e._unpack = lambda *a: torch.zeros(nx, ny)
    e.run = lambda t0, k: setattr(e, "_checked", False)
    e.snapshot = lambda b: []
    e.restore = lambda b, snap: None
    e._checked = False
    return e


def test_accumulators_report_a_timeout(fake):
    from meep_torch_b200._lib import MtbError
    fake.timed_out = {"p"}
    e = _engine(fake, "p")
    with pytest.raises(MtbError, match="bounded wait"):
        e.accumulators(0)
    fake.pending = True                      # or captured: not waited for (NaN then)
    assert len(e.accumulators(0)) == 1 and not e._checked
    fake.pending, fake.timed_out = False, set()
    assert len(e.accumulators(0)) == 1 and e._checked
    e._checked, fake.timed_out = False, {"p", None}
    e.close()
    assert len(e.accumulators(0)) == 1       # a closed plan's are still there


@pytest.mark.parametrize("late", [None, "rec0", "rec1", "rec2"])
def test_gradient_reports_a_timeout_of_any_recording_plan(fake, monkeypatch, late):
    """The chunks are recorded anew by up to three plans, two of them closed on the way."""
    import collections
    import types

    import torch

    from meep_torch_b200 import adjoint2d
    from meep_torch_b200._lib import MtbError
    plans = []

    def recording(items, **kw):
        plans.append(f"rec{len(plans)}")
        return _engine(fake, plans[-1])
    monkeypatch.setattr(adjoint2d, "Engine2D", recording)
    monkeypatch.setattr(adjoint2d, "_record_monitors", lambda *a: [])
    fake.timed_out = {late}
    St = collections.namedtuple("St", adjoint2d.STATE_TM)
    st = St(*[torch.zeros(6, 8)] * len(St._fields))
    # 256-step chunks walked in pieces of 64, the first chunk from the imported state
    monkeypatch.setattr(adjoint2d, "_cuts", lambda c, te: ((0, 0), (0, 0)))
    g = adjoint2d.GradRun2D(st, types.SimpleNamespace(dt=0.1), 300, None, [], chunk=256)
    g.eng, g.out_state, g.accs, g.snaps = _engine(fake, "fwd"), st, [], [[], []]
    if late is None:
        g.backward([None] * len(g.names))
        assert plans == ["rec0", "rec1", "rec2"]
        return
    with pytest.raises(MtbError, match="bounded wait"):
        g.backward([None] * len(g.names))


# ------------------------------------------------------------------ what the flag does
@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 2, 3, 4])
@pytest.mark.parametrize("ring", [32, 7])
def test_raised_flag_turns_accumulators_into_nan(variant, ring):
    """The flag is raised by the test (no wait is made to expire): the sums of the run that
    follows are NaN and the run is reported."""
    import ctypes as C

    import torch

    from meep_torch_b200 import _lib as L
    from meep_torch_b200.core.coeffs import build_tm_coeffs
    from meep_torch_b200.core.grid import Grid
    from meep_torch_b200.core.monitors import DFTFieldsMonitor, FluxMonitorTM
    from meep_torch_b200.core.sources import GaussianPulse, LineSource
    from meep_torch_b200.core.stepper_tm import init_tm_state
    from meep_torch_b200.engine2d import Engine2D
    nx, ny = 70, 60
    g = Grid(nx=nx, ny=ny, dx=0.05, device="cuda")
    m = build_tm_coeffs(g, eps_inf=torch.full((nx, ny), 2.0, device="cuda"), npml=8)
    src = LineSource(g, ix=20, j0=10, j1=50, profile=GaussianPulse(0.6, 0.4))
    mons = [DFTFieldsMonitor(g, [0.5, 0.6, 0.7, 0.8, 0.9], "Ez"),
            FluxMonitorTM(g, [0.5], x_normal=True, idx=40, lo=10, hi=50)]
    e = Engine2D([(init_tm_state(g), m, src, mons)], variant=variant, ring_slots=ring)
    e.run(0, 40)
    torch.cuda.synchronize()
    assert all(torch.isfinite(a).all() for a in e.accumulators(0))
    flag, one = C.c_void_p(), torch.ones(1, device="cuda")
    L.check(e.lib.mtb_yee2d_error_flag(e.plan, C.byref(flag)))
    L.check(e.lib.mtb_pack(L.ptr(one), 1, 1, 1, 1, 1, flag, 1, 1, 1, 1, 1, 0, 0, 0, e._sptr()))
    e.run(40, 40)
    accs = list(e.items[0].accs)
    torch.cuda.synchronize()
    assert all(torch.isnan(a).all() for a in accs)
    with pytest.raises(L.MtbError):
        e.accumulators(0)
    e.close()
