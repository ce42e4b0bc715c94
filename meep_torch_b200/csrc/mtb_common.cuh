// Shared internals of the B200 FDTD library: error state, launch counting,
// vector helpers. Device code targets sm_100a only.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <string>
#include <utility>
#include <vector>

#include "../../include/meep_b200.h"

namespace mtb {

// Last error text, one per host thread (mtb_last_error()).
void set_error(const char *fmt, ...);
int fail(int code, const char *fmt, ...);
void count_launch(int64_t n = 1);

// CPML band of a 2D profile (device arrays of n nodes): nodes with a != 0 or b != 1 satisfy
// k < lo_end or k >= hi_start (s: structure number for messages)
int profile_band(const float *b_d, const float *a_d, int n, int32_t &lo_end, int32_t &hi_start,
                 int s);

#define MTB_CUDA_TRY(expr)                                                    \
    do {                                                                      \
        cudaError_t e_ = (expr);                                              \
        if (e_ != cudaSuccess)                                                \
            return ::mtb::fail(MTB_CUDA_ERROR, "%s failed: %s (%s:%d)", #expr, \
                               cudaGetErrorString(e_), __FILE__, __LINE__);   \
    } while (0)

#define MTB_CHECK_LAUNCH()                                                    \
    do {                                                                      \
        cudaError_t e_ = cudaGetLastError();                                  \
        if (e_ != cudaSuccess)                                                \
            return ::mtb::fail(MTB_CUDA_ERROR, "kernel launch failed: %s (%s:%d)", \
                               cudaGetErrorString(e_), __FILE__, __LINE__);   \
        ::mtb::count_launch();                                                \
    } while (0)

// Plan scratch comes from a bounded pool, so that building and closing a plan does not pay
// cudaMalloc / cudaFree (and their pinned forms) a dozen times: these took 1.3 of the 3.3 ms of
// a 200-step run of a small plan, and up to 10 ms where other programs use the driver too.
// A block goes back only when its plan's set-up and the work of every stream it ran on have
// finished (StreamMarks, ScratchIdle; not by a device-wide wait, which breaks graph captures
// of other threads), so any thread, stream or plan of that device may take it next; contents
// are not kept or cleared. Without that knowledge it is freed, as cudaFree waits by itself. At most
// SCRATCH_KEEP bytes stay (the oldest blocks are freed first), none are kept when an
// allocation fails, and mtb_release_scratch() frees all.
constexpr size_t SCRATCH_KEEP[2] = {(size_t)256 << 20, (size_t)16 << 20};   // device, pinned
int scratch_get(bool host, size_t n, void **p, size_t *bytes, int *dev);
void scratch_put(bool host, void *p, size_t bytes, int dev);

// A buffer owned by a plan: device memory, or pinned host staging (plan scratch only; fields,
// coefficients and accumulators always belong to the caller).
template <bool HOST>
struct ScratchBuf {
    void *p = nullptr;
    size_t bytes = 0;
    int dev = 0;
    int ensure(size_t n) {
        if (n <= bytes) return MTB_OK;
        release();
        return scratch_get(HOST, n, &p, &bytes, &dev);
    }
    void release() {
        if (p) scratch_put(HOST, p, bytes, dev);
        p = nullptr;
        bytes = 0;
    }
    template <class T> T *as() const { return reinterpret_cast<T *>(p); }
};
using DevBuf = ScratchBuf<false>;
using HostBuf = ScratchBuf<true>;

// While it lives, this thread's synchronising calls are allowed beside graph captures of other
// threads (in the default capture mode these forbid them to every thread, and end broken).
struct BesideCaptures {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
    BesideCaptures(const BesideCaptures &) = delete;
};

// The streams a plan has queued work on, each with an event behind its latest use. A stream
// is known by its id: its handle may name another one after it is destroyed, work pending.
struct StreamMarks {
    struct One {
        unsigned long long id;
        cudaEvent_t ev;
    };
    std::vector<One> uses;
    // cannot tell: set-up not finished, captured by a caller, or a call failed
    bool unknown = true;
    bool open = false;               // work on open_st whose mark is still to come
    cudaStream_t open_st = nullptr;
    // a call that fails here fails for no caller: its error is not left for the next check
    static bool did(cudaError_t e) noexcept {
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess;
    }
    // The end of the plan's creation: its copies (of pageable memory, on the legacy stream) may
    // land after the calls that made them have returned. Before it, nothing is known to be idle.
    void ready() noexcept { unknown = !did(cudaStreamSynchronize(cudaStreamLegacy)); }
    void mark(cudaStream_t st) noexcept {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        unsigned long long id = 0;
        if (open && open_st != st) unknown = true;
        open = false;
        if (unknown) return;
        unknown = true;
        if (!did(cudaStreamIsCapturing(st, &cs)) || cs != cudaStreamCaptureStatusNone) return;
        if (!did(cudaStreamGetId(st, &id))) return;
        cudaEvent_t ev = nullptr;
        for (const One &u : uses)
            if (u.id == id) ev = u.ev;
        if (!ev) {
            if (uses.size() >= 16) return;
            if (!did(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming))) return;
            try {
                uses.push_back({id, ev});
            } catch (...) {
                cudaEventDestroy(ev);
                return;
            }
        }
        unknown = !did(cudaEventRecord(ev, st));
    }
    // A use that the mark at the end of its chunk of steps will cover: an event for every half
    // step would be one per launch. A chunk left unfinished cannot be told, nor one that
    // changes streams (the first may be gone by then).
    void later(cudaStream_t st) noexcept {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (open && open_st != st) unknown = true;
        if (!did(cudaStreamIsCapturing(st, &cs)) || cs != cudaStreamCaptureStatusNone)
            unknown = true;
        open = true;
        open_st = st;
    }
    // waits for all of it; false if that cannot be told
    bool wait() noexcept {
        unknown = unknown || open;
        for (const One &u : uses) {
            if (!unknown && !did(cudaEventSynchronize(u.ev))) unknown = true;
            did(cudaEventDestroy(u.ev));
        }
        uses.clear();
        return !unknown;
    }
};
// marks the plan's use of a stream when an entry point returns, by any path
struct MarkUse {
    StreamMarks &m;
    cudaStream_t st;
    MarkUse(StreamMarks &marks, void *stream) : m(marks), st((cudaStream_t)stream) {}
    ~MarkUse() { m.mark(st); }
};
// the same for an entry point that makes one part of a chunk: marked when no part is left
template <class Plan>
struct MarkChunk {
    Plan &p;
    cudaStream_t st;
    MarkChunk(Plan &plan, void *stream) : p(plan), st((cudaStream_t)stream) {}
    ~MarkChunk() {
        if (p.c_s < p.c_k) p.marks.later(st);
        else p.marks.mark(st);
    }
};
// while it lives, buffers that this thread releases are known to be idle (if `idle`)
struct ScratchIdle {
    explicit ScratchIdle(bool idle);
    ~ScratchIdle();
};

// Programmatic dependent launch, for chains of short step kernels: a kernel launched by
// launch_pdl may start while its predecessor still runs, once every block of that one has
// started (pdl_next) and SM space is free, and waits in pdl_wait until it has finished and
// its writes are visible. So the launch latency and everything before pdl_wait overlap the
// previous kernel. Rules: every thread that goes on calls pdl_wait before it reads or writes
// what an earlier kernel of the chain wrote or reads, and at least one thread of every launch
// does (so that a kernel's end implies that of all before it); such data is not read through
// the read-only path (__ldg, const __restrict__), which the wait does not order. Behind anything
// but a kernel (a copy, an event) the launch is an ordinary one. Measured, whole runs:
// 400 x 301 TM with poles, 800 steps (one tile launch each, about 8 us) 11.4 -> 9.2 ms;
// 117 x 90 x 75, 240 steps of three launches 11.7 -> 9.8 ms; 128 x 112 x 100 with poles
// 12.4 -> 10.8 ms; 96 x 80 x 72 gradient 17.2 -> 15.9 ms.
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    MTB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
    count_launch();
    return MTB_OK;
}

// Opt-in per-launch device timing (event pairs around launches).
// Two pinned host staging buffers used alternately for host -> device
// uploads: a buffer is refilled only after its previous upload completed
// (an event), so back-to-back runs on one stream never wait for the GPU.
struct PinnedPair {
    HostBuf h[2];
    cudaEvent_t ev[2] = {nullptr, nullptr};
    bool pending[2] = {false, false};
    int next = 0;
    // a staging buffer of at least `bytes` that may be overwritten now
    int acquire(size_t bytes, void **out) {
        const int b = next;
        if (pending[b]) {
            MTB_CUDA_TRY(cudaEventSynchronize(ev[b]));
            pending[b] = false;
        }
        const int rc = h[b].ensure(bytes);
        if (rc) return rc;
        *out = h[b].p;
        return MTB_OK;
    }
    // the upload from the last acquired buffer has been queued on `st`
    int queued(cudaStream_t st) {
        const int b = next;
        if (!ev[b]) MTB_CUDA_TRY(cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming));
        MTB_CUDA_TRY(cudaEventRecord(ev[b], st));
        pending[b] = true;
        next ^= 1;
        return MTB_OK;
    }
    void release() {
        for (int b = 0; b < 2; ++b) {
            if (ev[b]) {
                cudaEventSynchronize(ev[b]);
                cudaEventDestroy(ev[b]);
            }
            ev[b] = nullptr;
            pending[b] = false;
            h[b].release();
        }
    }
};

struct LaunchTimer {
    bool on = false;
    std::vector<cudaEvent_t> pool;
    size_t used = 0;
    std::vector<int> kind;          // 0 = step kernel, 1 = DFT contraction
    double ms[2] = {0, 0};
    int64_t count[2] = {0, 0};
    int begin(cudaStream_t st, int k);   // record the start event of a launch
    int end(cudaStream_t st);            // record the end event
    int collect();                       // wait and sum; resets the pool cursor
    void release();
};

// ---------------------------------------------------------------- DFT
// Phase tables and the ring contraction shared by the 2D and 3D plans.
struct DftState {
    // host copies
    std::string err;
    int n_regions = 0, n_groups = 0;
    mtb_dft_region *regions_h = nullptr;   // host copy
    int *group_nf = nullptr;               // host
    int *group_mode = nullptr;
    double *group_dt = nullptr;
    double *freqs_h = nullptr;             // concatenated
    int *freq_off = nullptr;               // per group offset into freqs_h
    int total_nf = 0;                      // sum of nf
    // device
    DevBuf regions_d, blk_start_d, blk_region_d, phase_d, ring_d;
    DevBuf freq_dt_d;                      // {frequency, dt} of every phase column
    const int *wait_err = nullptr;         // the plan's flag of expired waits, if it has one
    PinnedPair phase_h;
    int64_t slot_elems = 0;
    int slots = 0;                         // ring depth K
    int64_t n_blocks = 0;                  // contraction blocks
    int *blk_start_h = nullptr;

    int init(const mtb_dft_region *regions, int n_regions, const mtb_phase_group *groups,
             int n_groups, int64_t slot_elems, int slots);
    // The phase table of steps [t0, t0+k), on `st`.
    int upload_phases(int64_t t0, int k, cudaStream_t st);
    // Fold ring slots [0, n) (steps t_first .. t_first+n-1, relative row
    // `row0` of the uploaded table, or of `phase_base` when given) into the
    // accumulators.
    int contract(int row0, int n, cudaStream_t st, LaunchTimer *tm = nullptr,
                 const float *phase_base = nullptr);
    // Transposed contraction: zero ring slots [0, n) and fill them with the
    // adjoint of the samples of the n staged steps (region acc = d J / d acc).
    int expand(int row0, int n, cudaStream_t st);
    void release();
};

}  // namespace mtb
