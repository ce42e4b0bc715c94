// Error state, launch counter, layout kernels and the DFT ring contraction.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "mtb_common.cuh"

namespace mtb {

static thread_local char g_err[1024] = "";
static std::atomic<int64_t> g_launches{0};

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

void count_launch(int64_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// ------------------------------------------------------------ launch timer

int LaunchTimer::begin(cudaStream_t st, int k) {
    if (!on) return MTB_OK;
    while (pool.size() < used + 2) {
        cudaEvent_t e;
        MTB_CUDA_TRY(cudaEventCreate(&e));
        pool.push_back(e);
    }
    kind.resize(pool.size() / 2 + 1);
    kind[used / 2] = k;
    MTB_CUDA_TRY(cudaEventRecord(pool[used], st));
    return MTB_OK;
}

int LaunchTimer::end(cudaStream_t st) {
    if (!on) return MTB_OK;
    MTB_CUDA_TRY(cudaEventRecord(pool[used + 1], st));
    used += 2;
    return MTB_OK;
}

int LaunchTimer::collect() {
    if (!on || used == 0) return MTB_OK;
    MTB_CUDA_TRY(cudaEventSynchronize(pool[used - 1]));
    for (size_t i = 0; i < used; i += 2) {
        float t = 0.f;
        MTB_CUDA_TRY(cudaEventElapsedTime(&t, pool[i], pool[i + 1]));
        ms[kind[i / 2]] += t;
        count[kind[i / 2]] += 1;
    }
    used = 0;
    return MTB_OK;
}

void LaunchTimer::release() {
    for (auto e : pool) cudaEventDestroy(e);
    pool.clear();
    used = 0;
}

// ------------------------------------------------------------ plan scratch

namespace {
struct Kept {
    void *p;
    size_t bytes;
    int dev;
};
struct ScratchPool {
    std::mutex mu;
    std::vector<Kept> kept;          // oldest first
    size_t held = 0;
};
// never destroyed: plans may be closed while the process exits
ScratchPool &scratch_pool(bool host) {
    static ScratchPool *pools = new ScratchPool[2];
    return pools[host];
}
cudaError_t raw_alloc(bool host, void **p, size_t n) {
    return host ? cudaMallocHost(p, n) : cudaMalloc(p, n);
}
void raw_free(bool host, void *p) {
    if (host) cudaFreeHost(p);
    else cudaFree(p);
}
// makes `dev` current for its lifetime
struct OnDevice {
    int before = 0;
    bool moved = false;
    explicit OnDevice(int dev) {
        moved = cudaGetDevice(&before) == cudaSuccess && before != dev &&
                cudaSetDevice(dev) == cudaSuccess;
    }
    ~OnDevice() {
        if (moved) cudaSetDevice(before);
    }
};
// frees the oldest kept blocks until at most `keep` bytes stay
void scratch_trim(bool host, size_t keep) {
    ScratchPool &P = scratch_pool(host);
    for (;;) {
        Kept k{};
        {
            std::lock_guard<std::mutex> lock(P.mu);
            if (P.held <= keep || P.kept.empty()) return;
            k = P.kept.front();
            P.kept.erase(P.kept.begin());
            P.held -= k.bytes;
        }
        OnDevice on(k.dev);
        raw_free(host, k.p);
    }
}
}  // namespace

int scratch_get(bool host, size_t n, void **p, size_t *bytes, int *dev) {
    *p = nullptr;
    *bytes = 0;
    MTB_CUDA_TRY(cudaGetDevice(dev));
    if (n == 0) return MTB_OK;
    const size_t unit = n < ((size_t)1 << 20) ? 512 : (size_t)1 << 16;
    n = (n + unit - 1) / unit * unit;
    {
        ScratchPool &P = scratch_pool(host);
        std::lock_guard<std::mutex> lock(P.mu);
        int best = -1;
        for (int k = 0; k < (int)P.kept.size(); ++k) {
            const Kept &b = P.kept[k];
            if (b.dev == *dev && b.bytes >= n && b.bytes <= 2 * n &&
                (best < 0 || b.bytes < P.kept[best].bytes))
                best = k;
        }
        if (best >= 0) {
            *p = P.kept[best].p;
            *bytes = P.kept[best].bytes;
            P.held -= *bytes;
            P.kept.erase(P.kept.begin() + best);
            return MTB_OK;
        }
    }
    cudaError_t e = raw_alloc(host, p, n);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        scratch_trim(host, 0);
        e = raw_alloc(host, p, n);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return fail(MTB_CUDA_ERROR, "%s(%zu) failed: %s", host ? "cudaMallocHost" : "cudaMalloc", n,
                    cudaGetErrorString(e));
    }
    *bytes = n;
    return MTB_OK;
}

static thread_local bool scratch_idle = false;
ScratchIdle::ScratchIdle(bool idle) { scratch_idle = idle; }
ScratchIdle::~ScratchIdle() { scratch_idle = false; }

void scratch_put(bool host, void *p, size_t bytes, int dev) {
    OnDevice on(dev);
    bool keep = scratch_idle && bytes <= SCRATCH_KEEP[host];
    if (keep) {
        ScratchPool &P = scratch_pool(host);
        std::lock_guard<std::mutex> lock(P.mu);
        try {
            P.kept.push_back({p, bytes, dev});
            P.held += bytes;
        } catch (...) {
            keep = false;
        }
    }
    if (keep) scratch_trim(host, SCRATCH_KEEP[host]);
    else raw_free(host, p);
}

// ------------------------------------------------------------ layout kernels

// Index arithmetic in T: 32-bit wherever the box has fewer than 2^31 elements (a 64-bit
// division per element and axis set the time: a 67 MB box took 53 us).
// Writes the whole box: the block [off, off+n) gets src, the rest zero.
template <class T>
__global__ void k_pack(const float *__restrict__ src, T n0, T n1, T n2, int64_t s0, int64_t s1,
                       float *__restrict__ box, T bn0, T bn1, T bn2, int64_t b0, int64_t b1,
                       T o0, T o1, T o2) {
    const T total = bn0 * bn1 * bn2, step = (T)gridDim.x * blockDim.x;
    for (T idx = blockIdx.x * (T)blockDim.x + threadIdx.x; idx < total; idx += step) {
        const T r = idx / bn2, k = idx - r * bn2;
        const T i = r / bn1, j = r - i * bn1;
        float v = 0.f;
        if (i >= o0 && i - o0 < n0 && j >= o1 && j - o1 < n1 && k >= o2 && k - o2 < n2)
            v = src[(i - o0) * s0 + (j - o1) * s1 + (k - o2)];
        box[i * b0 + j * b1 + k] = v;
    }
}

template <class T>
__global__ void k_unpack(const float *__restrict__ box, T n0, T n1, T n2, int64_t b0, int64_t b1,
                         T o0, T o1, T o2, float *__restrict__ dst, int64_t s0, int64_t s1) {
    const T total = n0 * n1 * n2, step = (T)gridDim.x * blockDim.x;
    for (T idx = blockIdx.x * (T)blockDim.x + threadIdx.x; idx < total; idx += step) {
        const T r = idx / n2, k = idx - r * n2;
        const T i = r / n1, j = r - i * n1;
        dst[i * s0 + j * s1 + k] = box[(i + o0) * b0 + (j + o1) * b1 + (k + o2)];
    }
}

// 1/eps and eps of a plan's box in one pass: the block gets src and 1/src, the pitch zeros.
template <class T>
__global__ void k_pack_eps(const float *__restrict__ src, T n0, T n1, T pitch,
                           float *__restrict__ eps, float *__restrict__ inv) {
    const T total = n0 * pitch, step = (T)gridDim.x * blockDim.x;
    for (T idx = blockIdx.x * (T)blockDim.x + threadIdx.x; idx < total; idx += step) {
        const T i = idx / pitch, j = idx - i * pitch;
        const float v = j < n1 ? src[i * n1 + j] : 0.f;
        eps[idx] = v;
        inv[idx] = j < n1 ? __frcp_rn(v) : 0.f;
    }
}

// Zero a list of buffers, one per block column, in one launch. What bounds it: the launches
// it replaces (a batch of 64 structures has 1088 buffers of about 100 kB: one launch each
// took 7.0 ms of host time and 2.35 ms on the GPU, 9 launches 0.2 ms), then store bandwidth
// (16-byte stores between the unaligned ends).
constexpr int ZL_N = 128;
struct ZeroList {
    float *p[ZL_N];
    int64_t n[ZL_N];
};
__global__ void k_zero_list(const __grid_constant__ ZeroList z) {
    float *p = z.p[blockIdx.y];
    const int64_t n = z.n[blockIdx.y];
    const int64_t head = min(n, (int64_t)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / 4);
    const int64_t n4 = (n - head) / 4, tail = head + 4 * n4;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    float4 *q = reinterpret_cast<float4 *>(p + head);
    for (int64_t k = t; k < n4; k += (int64_t)gridDim.x * blockDim.x)
        q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < head) p[t] = 0.f;
    if (t < n - tail) p[tail + t] = 0.f;
}

__global__ void k_unpack_ratio(const float *__restrict__ box, const float *__restrict__ den,
                               int64_t n0, int64_t n1, int64_t n2, int64_t b0, int64_t b1,
                               int64_t o0, int64_t o1, int64_t o2, float *__restrict__ dst,
                               int64_t s0, int64_t s1) {
    const int64_t total = n0 * n1 * n2;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = idx % n2;
        const int64_t r = idx / n2;
        const int64_t j = r % n1;
        const int64_t i = r / n1;
        const int64_t b = (i + o0) * b0 + (j + o1) * b1 + (k + o2);
        dst[i * s0 + j * s1 + k] = box[b] / den[b];
    }
}

__global__ void k_count_outside(const float *__restrict__ x, int64_t n0, int64_t n1, int64_t s0,
                                const uint8_t *__restrict__ a0, const uint8_t *__restrict__ a1,
                                unsigned long long *count) {
    const int64_t total = n0 * n1;
    unsigned long long c = 0;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = idx % n1, i = idx / n1;
        const bool act = (a0 && a0[i]) || (a1 && a1[j]);
        if (!act && x[i * s0 + j] != 0.f) ++c;
    }
    if (c) atomicAdd(count, c);
}

static int grid_for(int64_t total, int threads = 256) {
    int64_t b = (total + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (int)b;
}

// ------------------------------------------------------------ DFT contraction

constexpr int KMAX = 64;       // deepest ring supported by the contraction
constexpr int CT = 256;        // channels per contraction block

// A chunk is CT channels of one region (the region of a chunk from a per-chunk table); a
// block folds a contiguous range of chunks. Phase values of a region's (group, toff) are
// staged in shared memory, frequency by frequency (sP[(f - fa) * (n + 2) + s] = (Re, Im);
// the two spare columns spread the staging stores over the banks), and staged again only
// where the range enters a region of another group or time offset.
//
// What bounds it: memory, given enough loads in flight. A block per chunk spent its time in
// the chain table -> region -> phases -> samples -> accumulators, one frequency after the
// other (bends batch, 5.3 M channels: 285 us per 32-step flush, 3.2 TB/s). Now a block's
// first chain serves all of its chunks, and the accumulators of NFC frequencies are loaded
// with the samples, the next NFC before the last ones are stored; the region sits in shared
// memory, since in registers it spilled. Now 215 us (4.2 TB/s; 64 designs: 199 ->
// 152 us, 256^3 flux faces 59 -> 40 us, 50 frequencies of a flux line 6.5 -> 5.5 us).
constexpr int NFC = 4;
constexpr int KFULL = 32;      // ring depth with a fully unrolled contraction (the default)
constexpr int SB = 16;         // samples in flight at other depths
__global__ void __launch_bounds__(CT, 3) k_dft_contract(
    const mtb_dft_region *__restrict__ regions, const int *__restrict__ blk_region,
    const int64_t *__restrict__ blk_start, const int *__restrict__ group_nf,
    const int *__restrict__ group_off, int total_nf, const float *__restrict__ phase, int row0,
    int n, const float *__restrict__ ring, int64_t slot_elems, int64_t n_chunks,
    const int *__restrict__ err) {
    extern __shared__ float4 sP4[];
    float2 *sP = reinterpret_cast<float2 *>(sP4);
    const int64_t per = (n_chunks + gridDim.x - 1) / gridDim.x;
    const int64_t c0 = blockIdx.x * per, c1 = min(n_chunks, c0 + per);
    __shared__ mtb_dft_region R;             // (in registers it spills)
    int rg = -1, staged = -1, fa = 0, fb = 0;
    int64_t first = 0;
    for (int64_t b = c0; b < c1; ++b) {
        const int q = blk_region[b];
        if (q != rg) {
            rg = q;
            first = blk_start[rg];
            __syncthreads();                 // the last chunk's readers are done
            for (int e = threadIdx.x; e < (int)(sizeof(R) / 4); e += CT)
                reinterpret_cast<int *>(&R)[e] = reinterpret_cast<const int *>(regions + rg)[e];
            __syncthreads();
            const int nf = group_nf[R.group];
            // frequencies [fa, fb) of this block row (small channel counts split the
            // frequency loop over gridDim.y block rows; each sum is formed as without it)
            const int pf = (nf + gridDim.y - 1) / gridDim.y;
            fa = blockIdx.y * pf;
            fb = min(nf, fa + pf);
            const int sel = (R.toff == 2) ? 2 : 0;
            if (staged != 2 * R.group + (sel >> 1)) {
                staged = 2 * R.group + (sel >> 1);
                const float *p0 = phase + ((int64_t)row0 * total_nf + group_off[R.group]) * 4 + sel;
                // after an expired wait the samples are incomplete: NaN phases, so NaN sums
                const bool bad = err && *err;
                for (int e = threadIdx.x; e < n * (fb - fa); e += CT) {
                    const int s = e / (fb - fa), f = e - s * (fb - fa);
                    const float *p = p0 + ((int64_t)s * total_nf + fa + f) * 4;
                    sP[f * (n + 2) + s] = bad ? make_float2(NAN, NAN) : make_float2(p[0], p[1]);
                }
                __syncthreads();
            }
        }
        const int64_t ch = (b - first) * CT + threadIdx.x;
        if (fa >= fb || ch >= (int64_t)R.rows * R.cols) continue;
        const int r = (int)(ch / R.cols), c = (int)(ch - (int64_t)r * R.cols);
        const float *xa = ring + R.ring_a + (int64_t)r * R.ring_pitch + c;
        const float *xb = (R.ring_b >= 0) ? ring + R.ring_b + (int64_t)r * R.ring_pitch + c : nullptr;
        float *pre = R.acc + R.re_off + (int64_t)r * R.acc_pitch + c;
        float *pim = R.acc + R.im_off + (int64_t)r * R.acc_pitch + c;
        const int64_t fs = R.f_stride;
        if (n == KFULL) {
            // a whole ring: every sample of the channel in flight at once
            float x[KFULL], ore[NFC], oim[NFC];
#pragma unroll
            for (int s = 0; s < KFULL; ++s) x[s] = __ldg(xa + s * slot_elems);
#pragma unroll
            for (int k = 0; k < NFC; ++k) {
                const int64_t o = min(fa + k, fb - 1) * fs;
                ore[k] = pre[o];
                oim[k] = pim[o];
            }
            if (xb) {
#pragma unroll
                for (int s = 0; s < KFULL; ++s) x[s] = 0.5f * (x[s] + __ldg(xb + s * slot_elems));
            }
            for (int f0 = fa; f0 < fb; f0 += NFC) {
                float re[NFC], im[NFC];
#pragma unroll
                for (int k = 0; k < NFC; ++k) {
                    re[k] = 0.f;
                    im[k] = 0.f;
                    if (f0 + k < fb) {
                        const float4 *pf = sP4 + (f0 - fa + k) * (KFULL / 2 + 1);
#pragma unroll
                        for (int s = 0; s < KFULL; s += 2) {
                            const float4 p = pf[s / 2];
                            re[k] = fmaf(p.x, x[s], re[k]);
                            im[k] = fmaf(p.y, x[s], im[k]);
                            re[k] = fmaf(p.z, x[s + 1], re[k]);
                            im[k] = fmaf(p.w, x[s + 1], im[k]);
                        }
                        re[k] += ore[k];
                        im[k] += oim[k];
                    }
                }
                if (f0 + NFC < fb) {
#pragma unroll
                    for (int k = 0; k < NFC; ++k) {
                        const int64_t o = min(f0 + NFC + k, fb - 1) * fs;
                        ore[k] = pre[o];
                        oim[k] = pim[o];
                    }
                }
#pragma unroll
                for (int k = 0; k < NFC; ++k) {
                    if (f0 + k < fb) {
                        pre[(f0 + k) * fs] = re[k];
                        pim[(f0 + k) * fs] = im[k];
                    }
                }
            }
            continue;
        }
        for (int f0 = fa; f0 < fb; f0 += NFC) {
            float *pr[NFC], *pi[NFC];
            float re[NFC], im[NFC];
#pragma unroll
            for (int k = 0; k < NFC; ++k) {
                const int64_t o = min(f0 + k, fb - 1) * fs;
                pr[k] = pre + o;
                pi[k] = pim + o;
                re[k] = 0.f;
                im[k] = 0.f;
            }
            // blocks of SB samples in flight at once (even n: the phases as float4), the rest
            // one by one
            const int nb = (n & 1) ? 0 : n / SB * SB;
            for (int s0 = 0; s0 < nb; s0 += SB) {
                float x[SB];
#pragma unroll
                for (int i = 0; i < SB; ++i) x[i] = xa[(s0 + i) * slot_elems];
                if (xb) {
#pragma unroll
                    for (int i = 0; i < SB; ++i) x[i] = 0.5f * (x[i] + xb[(s0 + i) * slot_elems]);
                }
#pragma unroll
                for (int k = 0; k < NFC; ++k) {
                    if (f0 + k < fb) {
                        const float4 *pf = reinterpret_cast<const float4 *>(
                            sP + (f0 - fa + k) * (n + 2) + s0);
#pragma unroll
                        for (int i = 0; i < SB; i += 2) {
                            const float4 p = pf[i / 2];
                            re[k] = fmaf(p.x, x[i], re[k]);
                            im[k] = fmaf(p.y, x[i], im[k]);
                            re[k] = fmaf(p.z, x[i + 1], re[k]);
                            im[k] = fmaf(p.w, x[i + 1], im[k]);
                        }
                    }
                }
            }
#pragma unroll 4
            for (int s = nb; s < n; ++s) {
                float x = xa[s * slot_elems];
                if (xb) x = 0.5f * (x + xb[s * slot_elems]);
                const float2 *ps = sP + (f0 - fa) * (n + 2) + s;
#pragma unroll
                for (int k = 0; k < NFC; ++k) {
                    if (f0 + k < fb) {
                        const float2 p = ps[k * (n + 2)];
                        re[k] = fmaf(p.x, x, re[k]);
                        im[k] = fmaf(p.y, x, im[k]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < NFC; ++k) {
                if (f0 + k < fb) {
                    *pr[k] += re[k];
                    *pi[k] += im[k];
                }
            }
        }
    }
}

// Transpose of k_dft_contract (the adjoint of DFT sampling): for ring slot
// s of the n staged steps, every channel of a region receives
//   sum_f Re P(s, f) acc_re[f, ch] + Im P(s, f) acc_im[f, ch]
// (acc = d J / d accumulator), split 1/2 : 1/2 onto ring_a / ring_b where
// the forward averaged two samples. Regions may share ring elements, so the
// ring (zeroed by the caller) is accumulated atomically.
__global__ void __launch_bounds__(CT) k_dft_expand(
    const mtb_dft_region *__restrict__ regions, const int *__restrict__ blk_region,
    const int64_t *__restrict__ blk_start, const int *__restrict__ group_nf,
    const int *__restrict__ group_off, int total_nf, const float *__restrict__ phase, int row0,
    int n, float *__restrict__ ring, int64_t slot_elems) {
    extern __shared__ float2 sP[];
    const int64_t b = blockIdx.x;
    const int rg = blk_region[b];
    const mtb_dft_region R = regions[rg];
    const int nf = group_nf[R.group];
    const int foff = group_off[R.group];
    const int sel = (R.toff == 2) ? 2 : 0;
    for (int e = threadIdx.x; e < n * nf; e += CT) {
        const int s = e / nf, f = e - s * nf;
        const float *p = phase + ((int64_t)(row0 + s) * total_nf + foff + f) * 4 + sel;
        sP[e] = make_float2(p[0], p[1]);
    }
    __syncthreads();
    const int64_t ch = (b - blk_start[rg]) * CT + threadIdx.x;
    const int64_t nch = (int64_t)R.rows * R.cols;
    if (ch >= nch) return;
    const int r = (int)(ch / R.cols), c = (int)(ch - (int64_t)r * R.cols);
    float *xa = ring + R.ring_a + (int64_t)r * R.ring_pitch + c;
    float *xb = (R.ring_b >= 0) ? ring + R.ring_b + (int64_t)r * R.ring_pitch + c : nullptr;
    const float *acc = R.acc;
    const int64_t base = (int64_t)r * R.acc_pitch + c;
    for (int s = 0; s < n; ++s) {
        float g = 0.f;
        for (int f = 0; f < nf; ++f) {
            const float2 p = sP[s * nf + f];
            g = fmaf(p.x, __ldg(acc + R.re_off + f * R.f_stride + base), g);
            g = fmaf(p.y, __ldg(acc + R.im_off + f * R.f_stride + base), g);
        }
        if (xb) {
            atomicAdd(xa + s * slot_elems, 0.5f * g);
            atomicAdd(xb + s * slot_elems, 0.5f * g);
        } else {
            atomicAdd(xa + s * slot_elems, g);
        }
    }
}

int DftState::init(const mtb_dft_region *regions, int nreg, const mtb_phase_group *groups,
                   int ngrp, int64_t selems, int nslots) {
    n_regions = nreg;
    n_groups = ngrp;
    slot_elems = selems;
    slots = nslots;
    if (nslots < 1 || nslots > KMAX)
        return fail(MTB_INVALID_ARG, "ring_slots must be in [1, %d], got %d", KMAX, nslots);
    if (nreg < 0 || ngrp < 0) return fail(MTB_INVALID_ARG, "negative region/group count");
    if (nreg > 0 && (!regions || !groups)) return fail(MTB_INVALID_ARG, "null regions/groups");
    group_nf = (int *)calloc(ngrp + 1, sizeof(int));
    group_mode = (int *)calloc(ngrp + 1, sizeof(int));
    group_dt = (double *)calloc(ngrp + 1, sizeof(double));
    freq_off = (int *)calloc(ngrp + 1, sizeof(int));
    total_nf = 0;
    for (int g = 0; g < ngrp; ++g) {
        if (groups[g].nf < 1 || groups[g].nf > 256 || !groups[g].freqs)
            return fail(MTB_INVALID_ARG, "phase group %d: nf=%d out of [1,256] or null freqs", g,
                        groups[g].nf);
        if (groups[g].mode != 0 && groups[g].mode != 1)
            return fail(MTB_INVALID_ARG, "phase group %d: mode must be 0 or 1", g);
        group_nf[g] = groups[g].nf;
        group_mode[g] = groups[g].mode;
        group_dt[g] = groups[g].dt;
        freq_off[g] = total_nf;
        total_nf += groups[g].nf;
    }
    freqs_h = (double *)calloc(total_nf + 1, sizeof(double));
    for (int g = 0; g < ngrp; ++g)
        memcpy(freqs_h + freq_off[g], groups[g].freqs, sizeof(double) * groups[g].nf);
    regions_h = (mtb_dft_region *)calloc(nreg + 1, sizeof(mtb_dft_region));
    if (nreg) memcpy(regions_h, regions, sizeof(mtb_dft_region) * nreg);
    blk_start_h = (int *)calloc(nreg + 1, sizeof(int));
    std::vector<int64_t> bs(nreg + 1, 0);
    int64_t nb = 0;
    for (int r = 0; r < nreg; ++r) {
        const mtb_dft_region &R = regions[r];
        if (R.group < 0 || R.group >= ngrp)
            return fail(MTB_INVALID_ARG, "region %d: bad group %d", r, R.group);
        if (R.toff != 1 && R.toff != 2)
            return fail(MTB_INVALID_ARG, "region %d: toff must be 1 or 2", r);
        if (R.rows < 0 || R.cols < 0 || !R.acc)
            return fail(MTB_INVALID_ARG, "region %d: bad extent or null accumulator", r);
        if (R.ring_a < 0 || R.ring_a + (int64_t)(R.rows - 1) * R.ring_pitch + R.cols > selems ||
            (R.ring_b >= 0 && R.ring_b + (int64_t)(R.rows - 1) * R.ring_pitch + R.cols > selems))
            return fail(MTB_INVALID_ARG, "region %d: ring window outside the slot (%lld elems)", r,
                        (long long)selems);
        bs[r] = nb;
        nb += ((int64_t)R.rows * R.cols + CT - 1) / CT;
    }
    bs[nreg] = nb;
    n_blocks = nb;
    if (nb > 0x7fffffffLL) return fail(MTB_INVALID_ARG, "too many DFT channels");
    std::vector<int> br((size_t)nb + 1, 0);
    for (int r = 0; r < nreg; ++r)
        for (int64_t q = bs[r]; q < bs[r + 1]; ++q) br[q] = r;
    int rc;
    if ((rc = blk_region_d.ensure(sizeof(int) * (br.size())))) return rc;
    MTB_CUDA_TRY(cudaMemcpy(blk_region_d.p, br.data(), sizeof(int) * br.size(),
                            cudaMemcpyHostToDevice));
    if ((rc = regions_d.ensure(sizeof(mtb_dft_region) * (nreg + 1)))) return rc;
    if ((rc = blk_start_d.ensure(sizeof(int64_t) * (nreg + 1) + 2 * sizeof(int) * (ngrp + 1))))
        return rc;
    std::vector<double2> fd(total_nf);
    for (int g = 0; g < ngrp; ++g)
        for (int f = 0; f < group_nf[g]; ++f)
            fd[freq_off[g] + f] = make_double2(groups[g].freqs[f], groups[g].dt);
    if ((rc = freq_dt_d.ensure(sizeof(double2) * fd.size()))) return rc;
    if (total_nf) MTB_CUDA_TRY(cudaMemcpy(freq_dt_d.p, fd.data(), sizeof(double2) * fd.size(),
                                          cudaMemcpyHostToDevice));
    if (nreg) MTB_CUDA_TRY(cudaMemcpy(regions_d.p, regions, sizeof(mtb_dft_region) * nreg,
                                      cudaMemcpyHostToDevice));
    MTB_CUDA_TRY(cudaMemcpy(blk_start_d.p, bs.data(), sizeof(int64_t) * (nreg + 1),
                            cudaMemcpyHostToDevice));
    int *gd = reinterpret_cast<int *>(blk_start_d.as<int64_t>() + (nreg + 1));
    MTB_CUDA_TRY(cudaMemcpy(gd, group_nf, sizeof(int) * (ngrp + 1), cudaMemcpyHostToDevice));
    MTB_CUDA_TRY(cudaMemcpy(gd + (ngrp + 1), freq_off, sizeof(int) * (ngrp + 1),
                            cudaMemcpyHostToDevice));
    // the ring exists whenever samples are written (DFT regions or stacked probes)
    if (selems > 0 && (rc = ring_d.ensure(sizeof(float) * (size_t)selems * nslots))) return rc;
    return MTB_OK;
}

// Phase rows of steps t0 .. t0+k-1 in FP64 (mode 0), one sample time of one frequency per
// thread. What bounds it: the FP64 sine and cosine; on the host they held up the first launch
// (4000 steps x 50 frequencies: 10-16 ms against about 0.03 ms here).
__global__ void __launch_bounds__(256) k_phase_rows(float2 *__restrict__ phase,
                                                    const double2 *__restrict__ freq_dt,
                                                    uint32_t total_nf, int64_t t0, int64_t n) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int64_t row = e >> 1, s = row / total_nf;
    const double2 q = freq_dt[row - s * total_nf];
    const double two_pi = 2.0 * M_PI;
    const double tt = ((double)(t0 + s) + 0.5 * (double)((e & 1) + 1)) * q.y;
    double sn, c;
    sincos(two_pi * q.x * tt, &sn, &c);
    phase[e] = make_float2((float)(q.y * c), (float)(-q.y * sn));
}

int DftState::upload_phases(int64_t t0, int k, cudaStream_t st) {
    if (n_regions == 0) return MTB_OK;
    const size_t n = (size_t)k * total_nf * 4;
    int rc;
    if (std::all_of(group_mode, group_mode + n_groups, [](int m) { return m == 0; })) {
        // all in FP64: on the GPU. The float32 mode restates another program's float32
        // sines and stays with the host's.
        if ((rc = phase_d.ensure(n * sizeof(float)))) return rc;
        if (n == 0) return MTB_OK;
        const int64_t m = (int64_t)n / 2;
        k_phase_rows<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(
            phase_d.as<float2>(), freq_dt_d.as<double2>(), total_nf, t0, m);
        MTB_CHECK_LAUNCH();
        return MTB_OK;
    }
    void *hp = nullptr;
    if ((rc = phase_h.acquire(n * sizeof(float), &hp))) return rc;
    if ((rc = phase_d.ensure(n * sizeof(float)))) return rc;
    float *P = static_cast<float *>(hp);
    const double two_pi = 2.0 * M_PI;
    for (int g = 0; g < n_groups; ++g) {
        const double dt = group_dt[g];
        const float dtf = (float)dt;
        for (int f = 0; f < group_nf[g]; ++f) {
            const double fr = freqs_h[freq_off[g] + f];
            const float wf = (float)two_pi * (float)fr;   // reference float32 w
            for (int s = 0; s < k; ++s) {
                float *p = P + ((size_t)s * total_nf + freq_off[g] + f) * 4;
                for (int h = 0; h < 2; ++h) {
                    const double tt = ((double)(t0 + s) + 0.5 * (h + 1)) * dt;
                    float c, sn;
                    if (group_mode[g] == 0) {
                        const double arg = two_pi * fr * tt;
                        c = (float)(dt * cos(arg));
                        sn = (float)(-dt * sin(arg));
                    } else {
                        const float arg = wf * (float)tt;
                        c = dtf * cosf(arg);
                        sn = dtf * -sinf(arg);
                    }
                    p[2 * h] = c;
                    p[2 * h + 1] = sn;
                }
            }
        }
    }
    MTB_CUDA_TRY(cudaMemcpyAsync(phase_d.p, P, n * sizeof(float), cudaMemcpyHostToDevice, st));
    return phase_h.queued(st);
}

int DftState::contract(int row0, int n, cudaStream_t st, LaunchTimer *tm,
                       const float *phase_base) {
    if (n_regions == 0 || n <= 0 || n_blocks == 0) return MTB_OK;
    int maxnf = 1;
    for (int g = 0; g < n_groups; ++g) maxnf = std::max(maxnf, group_nf[g]);
    static bool attr_set = false;
    if (!attr_set) {
        MTB_CUDA_TRY(cudaFuncSetAttribute(k_dft_contract,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          sizeof(float2) * (KMAX + 2) * 256));
        attr_set = true;
    }
    const int *gd = reinterpret_cast<const int *>(blk_start_d.as<int64_t>() + (n_regions + 1));
    if (n_blocks > 0x7fffffffLL) return fail(MTB_INVALID_ARG, "too many contraction blocks");
    int rc;
    if (tm && (rc = tm->begin(st, 1))) return rc;
    // few channels: split every channel's frequencies over block rows (four or more
    // frequencies each) until the launch has about 2^17 threads
    const int64_t want = ((int64_t)1 << 17) / std::max<int64_t>(n_blocks * CT, 1);
    const int fsplit = (int)std::max<int64_t>(1, std::min<int64_t>(want, (maxnf + 3) / 4));
    const size_t smem = sizeof(float2) * (size_t)(n + 2) * ((maxnf + fsplit - 1) / fsplit);
    // enough blocks for 16 per SM, then more chunks per block
    const int64_t nb = std::min<int64_t>(n_blocks, 148 * 16);
    k_dft_contract<<<dim3((unsigned)nb, fsplit), CT, smem, st>>>(
        regions_d.as<mtb_dft_region>(), blk_region_d.as<int>(), blk_start_d.as<int64_t>(), gd,
        gd + (n_groups + 1), total_nf, phase_base ? phase_base : phase_d.as<float>(), row0, n,
        ring_d.as<float>(), slot_elems, n_blocks, wait_err);
    MTB_CHECK_LAUNCH();
    if (tm && (rc = tm->end(st))) return rc;
    return MTB_OK;
}

int DftState::expand(int row0, int n, cudaStream_t st) {
    if (n <= 0) return MTB_OK;
    MTB_CUDA_TRY(cudaMemsetAsync(ring_d.p, 0, sizeof(float) * (size_t)slot_elems * n, st));
    if (n_regions == 0 || n_blocks == 0) return MTB_OK;
    int maxnf = 1;
    for (int g = 0; g < n_groups; ++g) maxnf = std::max(maxnf, group_nf[g]);
    const size_t smem = sizeof(float2) * (size_t)n * maxnf;
    static bool attr_set = false;
    if (!attr_set) {
        MTB_CUDA_TRY(cudaFuncSetAttribute(k_dft_expand, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          sizeof(float2) * KMAX * 256));
        attr_set = true;
    }
    const int *gd = reinterpret_cast<const int *>(blk_start_d.as<int64_t>() + (n_regions + 1));
    k_dft_expand<<<(unsigned)n_blocks, CT, smem, st>>>(
        regions_d.as<mtb_dft_region>(), blk_region_d.as<int>(), blk_start_d.as<int64_t>(), gd,
        gd + (n_groups + 1), total_nf, phase_d.as<float>(), row0, n, ring_d.as<float>(),
        slot_elems);
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

void DftState::release() {
    regions_d.release();
    blk_start_d.release();
    blk_region_d.release();
    phase_d.release();
    freq_dt_d.release();
    ring_d.release();
    phase_h.release();
    free(regions_h);
    free(group_nf);
    free(group_mode);
    free(group_dt);
    free(freqs_h);
    free(freq_off);
    free(blk_start_h);
    regions_h = nullptr;
    group_nf = group_mode = freq_off = blk_start_h = nullptr;
    group_dt = freqs_h = nullptr;
}

}  // namespace mtb

using namespace mtb;

extern "C" {

const char *mtb_last_error(void) { return g_err; }

int32_t mtb_abi_version(void) { return MTB_ABI_VERSION; }

int64_t mtb_launch_count(void) { return g_launches.load(); }

int64_t mtb_struct_size(int32_t which) {
    switch (which) {
        case 0: return sizeof(mtb_cells);
        case 1: return sizeof(mtb_line_sample);
        case 2: return sizeof(mtb_yee2d_struct);
        case 3: return sizeof(mtb_phase_group);
        case 4: return sizeof(mtb_dft_region);
        case 5: return sizeof(mtb_tuning);
        case 6: return sizeof(mtb_yee3d_struct);
        case 7: return sizeof(mtb_adj2d_buffers);
        case 8: return sizeof(mtb_adj3d_buffers);
        default: return -1;
    }
}

void mtb_release_scratch(void) {
    scratch_trim(false, 0);
    scratch_trim(true, 0);
}

int mtb_pack(const float *src, int64_t n0, int64_t n1, int64_t n2, int64_t s0, int64_t s1,
             float *box, int64_t bn0, int64_t bn1, int64_t bn2, int64_t b0, int64_t b1,
             int64_t o0, int64_t o1, int64_t o2, void *stream) {
    if (!box || (!src && n0 * n1 * n2 > 0)) return fail(MTB_INVALID_ARG, "mtb_pack: null pointer");
    if (n0 < 0 || n1 < 0 || n2 < 0 || o0 < 0 || o1 < 0 || o2 < 0 || o0 + n0 > bn0 ||
        o1 + n1 > bn1 || o2 + n2 > bn2 || bn2 > b1 || bn1 * b1 > b0)
        return fail(MTB_INVALID_ARG, "mtb_pack: block (%lld,%lld,%lld)+(%lld,%lld,%lld) outside box "
                    "(%lld,%lld,%lld)", (long long)n0, (long long)n1, (long long)n2, (long long)o0,
                    (long long)o1, (long long)o2, (long long)bn0, (long long)bn1, (long long)bn2);
    const int64_t total = bn0 * bn1 * bn2;
    if (total == 0) return MTB_OK;
    // the grid's stride stays within 32 bits too
    if (total < INT32_MAX && n0 < INT32_MAX && n1 < INT32_MAX && n2 < INT32_MAX)
        k_pack<uint32_t><<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
            src, n0, n1, n2, s0, s1, box, bn0, bn1, bn2, b0, b1, o0, o1, o2);
    else
        k_pack<int64_t><<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
            src, n0, n1, n2, s0, s1, box, bn0, bn1, bn2, b0, b1, o0, o1, o2);
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

int mtb_pack_eps(const float *src, int64_t n0, int64_t n1, int64_t pitch, float *eps, float *inv,
                 void *stream) {
    if (!src || !eps || !inv) return fail(MTB_INVALID_ARG, "mtb_pack_eps: null pointer");
    if (n0 < 1 || n1 < 1 || pitch < n1)
        return fail(MTB_INVALID_ARG, "mtb_pack_eps: %lld x %lld of pitch %lld", (long long)n0,
                    (long long)n1, (long long)pitch);
    if (n0 * pitch < INT32_MAX)
        k_pack_eps<uint32_t><<<grid_for(n0 * pitch), 256, 0, (cudaStream_t)stream>>>(
            src, n0, n1, pitch, eps, inv);
    else
        k_pack_eps<int64_t><<<grid_for(n0 * pitch), 256, 0, (cudaStream_t)stream>>>(
            src, n0, n1, pitch, eps, inv);
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

int mtb_zero(const uint64_t *bufs, const int64_t *n, int32_t count, void *stream) {
    if (count < 0 || (count && (!bufs || !n)))
        return fail(MTB_INVALID_ARG, "mtb_zero: null list");
    for (int32_t k = 0; k < count; ++k)
        if (n[k] < 0 || (n[k] && (!bufs[k] || bufs[k] % sizeof(float))))
            return fail(MTB_INVALID_ARG, "mtb_zero: buffer %d", k);
    for (int32_t k = 0; k < count;) {
        ZeroList z;
        int m = 0;
        int64_t most = 0;
        for (; k < count && m < ZL_N; ++k) {
            if (!n[k]) continue;
            z.p[m] = reinterpret_cast<float *>(bufs[k]);
            z.n[m++] = n[k];
            most = std::max(most, n[k]);
        }
        if (!m) break;
        for (int i = m; i < ZL_N; ++i) z.p[i] = nullptr, z.n[i] = 0;
        // at most eight 16-byte stores per thread in the largest buffer, 32 blocks per SM
        const int64_t bx = std::min<int64_t>((most + 8191) / 8192, (148 * 32 + m - 1) / m);
        k_zero_list<<<dim3((unsigned)bx, m), 256, 0, (cudaStream_t)stream>>>(z);
        MTB_CHECK_LAUNCH();
    }
    return MTB_OK;
}

int mtb_unpack(const float *box, int64_t n0, int64_t n1, int64_t n2, int64_t b0, int64_t b1,
               int64_t o0, int64_t o1, int64_t o2, float *dst, int64_t s0, int64_t s1,
               void *stream) {
    const int64_t total = n0 * n1 * n2;
    if (total == 0) return MTB_OK;
    if (!box || !dst) return fail(MTB_INVALID_ARG, "mtb_unpack: null pointer");
    if (n0 < 0 || n1 < 0 || n2 < 0 || o0 < 0 || o1 < 0 || o2 < 0)
        return fail(MTB_INVALID_ARG, "mtb_unpack: negative extent");
    if (total < INT32_MAX && o0 < INT32_MAX && o1 < INT32_MAX && o2 < INT32_MAX)
        k_unpack<uint32_t><<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
            box, n0, n1, n2, b0, b1, o0, o1, o2, dst, s0, s1);
    else
        k_unpack<int64_t><<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
            box, n0, n1, n2, b0, b1, o0, o1, o2, dst, s0, s1);
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

int mtb_unpack_ratio(const float *box, const float *den, int64_t n0, int64_t n1, int64_t n2,
                     int64_t b0, int64_t b1, int64_t o0, int64_t o1, int64_t o2, float *dst,
                     int64_t s0, int64_t s1, void *stream) {
    const int64_t total = n0 * n1 * n2;
    if (total == 0) return MTB_OK;
    if (!box || !den || !dst) return fail(MTB_INVALID_ARG, "mtb_unpack_ratio: null pointer");
    if (n0 < 0 || n1 < 0 || n2 < 0 || o0 < 0 || o1 < 0 || o2 < 0)
        return fail(MTB_INVALID_ARG, "mtb_unpack_ratio: negative extent");
    k_unpack_ratio<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(box, den, n0, n1, n2, b0, b1,
                                                                       o0, o1, o2, dst, s0, s1);
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

int mtb_count_outside(const float *x, int64_t n0, int64_t n1, int64_t s0, const uint8_t *a0,
                      const uint8_t *a1, int64_t *count_dev, void *stream) {
    if (!x || !count_dev) return fail(MTB_INVALID_ARG, "mtb_count_outside: null pointer");
    const int64_t total = n0 * n1;
    MTB_CUDA_TRY(cudaMemsetAsync(count_dev, 0, sizeof(int64_t), (cudaStream_t)stream));
    if (total == 0) return MTB_OK;
    k_count_outside<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(
        x, n0, n1, s0, a0, a1, reinterpret_cast<unsigned long long *>(count_dev));
    MTB_CHECK_LAUNCH();
    return MTB_OK;
}

}  // extern "C"
