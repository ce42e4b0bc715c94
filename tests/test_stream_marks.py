"""What a plan knows of the streams its work runs on (StreamMarks), compiled for the host
against a CUDA runtime whose streams are counters of queued work: scratch is called idle only
when all of it has run, and the bookkeeping leaves nothing behind for other calls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

HOST = r"""
#include "meep_torch_b200/csrc/mtb_common.cuh"
#include <cstdio>
#include <cstring>
#include <map>

// a stream: its id, work queued and work done; an event: the work of a stream it stands for
struct Work { unsigned long long id; long queued = 0, done = 0; bool capturing = false; };
struct Event { Work *w = nullptr; long upto = 0; };
static std::map<cudaStream_t, Work *> handles;     // what a handle means now
static unsigned long long next_id = 10;
static cudaError_t last = cudaSuccess, capture_query = cudaSuccess;
static int records = 0;
static Work *work_of(cudaStream_t st) {
    Work *&w = handles[st];
    if (!w) w = new Work{next_id++};
    return w;
}
static cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
extern "C" {
cudaError_t cudaStreamIsCapturing(cudaStream_t st, cudaStreamCaptureStatus *cs) {
    *cs = work_of(st)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return set(capture_query);
}
cudaError_t cudaStreamGetId(cudaStream_t st, unsigned long long *id) {
    *id = work_of(st)->id;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new Event);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    Work *w = work_of(st);
    *reinterpret_cast<Event *>(e) = {w, w->queued};
    ++records;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    Event *v = reinterpret_cast<Event *>(e);
    if (v->w && v->w->done < v->upto) v->w->done = v->upto;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<Event *>(e);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    Work *w = work_of(st);
    w->done = w->queued;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
}
namespace mtb { int fail(int code, const char *, ...) { return code; } }

static cudaStream_t stream(int k) { return reinterpret_cast<cudaStream_t>((size_t)(64 + k)); }
static bool idle(Work *w) { return w->done == w->queued; }

int main(int, char **argv) {
    const char *what = argv[1];
    mtb::StreamMarks m;
    if (!strcmp(what, "unfinished")) {           // set-up copies may still be landing
        printf("%d\n", (int)!m.wait());
        return 0;
    }
    work_of(cudaStreamLegacy)->queued += 2;      // set-up copies
    m.ready();
    bool ok = idle(work_of(cudaStreamLegacy));
    if (!ok) return 1;
    if (!strcmp(what, "use")) {                  // work on two streams is waited for
        for (int k = 0; k < 2; ++k) { work_of(stream(k))->queued += 3; m.mark(stream(k)); }
        ok = m.wait() && idle(work_of(stream(0))) && idle(work_of(stream(1)));
    } else if (!strcmp(what, "reused")) {        // a stream destroyed, its handle used again
        Work *gone = work_of(stream(0));
        gone->queued = 5;
        m.mark(stream(0));
        handles.erase(stream(0));
        work_of(stream(0))->queued = 2;
        m.mark(stream(0));
        ok = m.wait() && idle(gone) && idle(work_of(stream(0)));
    } else if (!strcmp(what, "halves")) {        // one record for a chunk of half steps
        for (int k = 0; k < 63; ++k) { ++work_of(stream(0))->queued; m.later(stream(0)); }
        ++work_of(stream(0))->queued;
        m.mark(stream(0));
        ok = records == 1 && m.wait() && idle(work_of(stream(0)));
    } else if (!strcmp(what, "halves_streams")) {   // a stream that may be gone by now
        m.later(stream(0));
        handles.clear();
        m.mark(stream(1));
        ok = handles.count(stream(0)) == 0 && !m.wait();
    } else if (!strcmp(what, "halves_left")) {   // a chunk that was not finished
        ++work_of(stream(0))->queued;
        m.later(stream(0));
        ok = !m.wait();
    } else if (!strcmp(what, "halves_capture")) {
        work_of(stream(0))->capturing = true;
        m.later(stream(0));
        work_of(stream(0))->capturing = false;
        m.mark(stream(0));
        ok = !m.wait();
    } else if (!strcmp(what, "unused")) {        // set up, never run
        ok = m.wait();
    } else if (!strcmp(what, "capture")) {       // captured work cannot be waited for
        work_of(stream(0))->capturing = true;
        m.mark(stream(0));
        ok = !m.wait();
    } else if (!strcmp(what, "last_error")) {    // a query that fails leaves no error behind
        capture_query = cudaErrorStreamCaptureImplicit;
        m.mark(stream(0));
        ok = cudaGetLastError() == cudaSuccess && !m.wait();
    }
    printf("%d\n", (int)ok);
}
"""


@pytest.fixture(scope="module")
def marks(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("marks")
    (d / "m.cpp").write_text(HOST)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", f"-I{ROOT}", f"-I{CUDA}", "-o",
                    str(d / "m"), str(d / "m.cpp")], check=True)
    return lambda what: subprocess.run([str(d / "m"), what], capture_output=True, text=True,
                                       check=True, timeout=60).stdout.strip()


@pytest.mark.parametrize("what", ["use", "capture", "last_error", "unfinished", "unused",
                                  "reused", "halves", "halves_streams", "halves_left",
                                  "halves_capture"])
def test_marks(marks, what):
    assert marks(what) == "1"
