// Resident 2D Yee steps (TM and TE) for sm_100a: the reference's step (TM
// core/stepper_tm.py:234-254, TE core/stepper_te.py:178-190, with CPML, soft sources and
// the monitor samples) for a ring's worth of steps per launch, for plans whose tiles all
// fit on the GPU at once. One cooperative launch, one block per tile; a tile stays in its
// block's registers for the whole launch.
//
// Tile. W warps of RW rows x RB_C = 128 columns: lane L of warp w keeps rows w RW ..
// w RW + RW - 1, columns 4L .. 4L+3 of every field and of 1/eps in registers. The output
// block has a halo of RB_T = 4 rows above and below and 4 columns left and right: a step
// reads one neighbour on each side, so after RB_T sub-steps the output block is exact.
// Then the blocks store their rims (4 cells deep) to the plan's arrays, publish an epoch
// flag, wait for their eight neighbours' flags and load their halos from L2.
//
// One barrier per sub-step: a warp repeats the update of one extra row (TM: Hy of the row
// above its first; TE: Dy of the row below its last), so that the H and the E half need
// one exchange between warps together: the top and bottom rows of Ez (TM) / Hz (TE)
// through shared memory, double-buffered by sub-step parity.
//
// What bounds it, and why this split: small plans are chains of short dependent steps.
// Launches of one or four steps (5.8-16.6 us each) or two cluster barriers a step (3.3 us)
// set their time, not bytes. Per step, profiler, before -> with this kernel: 64 x 48 TM
// 3.28 -> 1.46 us (cluster kernel before), 320 x 160 TM 4.16 -> 2.14 us (cluster kernel),
// 501 x 389 TE 4.11 -> 2.58 us (temporally blocked kernel). About 0.25 us of each step is
// the exchange between blocks every RB_T steps, the rest the warps' dependent updates and
// the one barrier (issue slots 22-34 % active, the barrier the largest stall). The rounding
// of every sub-step is that of the kernel it stands in for (CL: the cluster kernel; else the
// temporally blocked tile around it): same bits, but for a source cell listed more than
// once, which is subtracted once with the summed weight.
//
// CPML memory sits in shared memory, each thread's own slots (no exchange), and only in
// tiles that reach a layer; tiles that reach no x / no y layer run sub-steps without the
// terms of that axis. Waits are bounded by %globaltimer: an expired one raises the plan's
// error flag and the block leaves.
#pragma once

namespace mtb {

constexpr int RB_T = 4;                      // sub-steps between halo refreshes
constexpr int RB_C = 128;                    // tile columns (a float4 per lane)
constexpr int RB_OUTC = RB_C - 8;            // output columns per tile
constexpr int RB_WARPS = 16;                 // most warps of a block
constexpr int RB_SLOTS = 64;                 // deepest ring (steps per resident launch)

// A tile: {structure, first output row, first output column, flags}, {output rows, 0, 0, 0}
constexpr int RB_WORK = 2;                   // int4 per tile
constexpr int RBF_XL = 1, RBF_YL = 2;        // the tile reaches an x / y layer
constexpr int RBF_LEAN = 4;                  // the temporally blocked tile around it is lean
constexpr int RBF_SRC = 8;                   // a row with source cells
constexpr int RBF_LINES = 16;                // a line sample crosses the output block

struct __align__(16) RbMeta {
    mtb_yee2d_struct s;
    mtb_line_sample lines[MAXL];
};
static_assert(sizeof(mtb_yee2d_struct) % 16 == 0, "descriptor copies are 16-byte multiples");

struct RbCtx {
    const RbMeta *meta;      // per structure
    const float *amp_e;      // coefficient row of sub-step 0; sub-step s at + s * ncols
    const float *amp_h;
    int ncols;
    int nsub;                // steps of this launch
    float *ring;             // ring slot of sub-step 0; sub-step s at + s * slot_elems
    int64_t slot_elems;
    int *err;
    int par;                 // buffer holding the old state
    const int4 *work;
    int *flags;              // epoch per tile
    const int *nb;           // eight neighbours per tile, -1 where there is none
    int hits;                // room for line hits per warp
};

// ------------------------------------------------------------------ tile state
// Per-thread state of a tile. m, x, y: Dz, Hx, Hy (TM) / Hz, Dx, Dy (TE); ia, ib: 1/eps.
// yh: Hy of row -1 (TM) / Dy of row RW (TE), the extra row, with its 1/eps (TE) and
// x-layer memory.
template <bool TE, int RW>
struct RbTile {
    float m[RW][4], x[RW][4], y[RW][4], ia[RW][4], ib[TE ? RW : 1][4];
    float yh[4], ph[4], ibh[TE ? 4 : 1];
    float iah[4];                            // TM, CL: 1/eps of row -1
    float e[RW][4];                          // TM: Ez (also the sampled value)
};

// Where a thread's tile lies and what is valid there; rows are bit r + 1 of the masks
// (bit 0: row -1, bit RW + 1: row RW). A difference is set to +0 in a row or column that
// is not updated (an and with its bits: a factor of 0 would give NaN beside a field that has
// overflowed). Rows and columns off the arrays hold zeros with 1/eps = 0 and stay zero.
template <int RW>
struct RbPos {
    int nx, ny, P;
    int iw;                  // structure row of this warp's row 0
    int jb;                  // structure column of this lane's first cell
    int w, lane, W;
    unsigned ca[4], cb[4];   // ~0 where the column is updated, else 0: TM Hx, Dz; TE Dx, Hz
    unsigned ty[RW + 1];     // the same of rows: TM Hy of rows -1 .. RW-1; TE Dy of 0 .. RW
    unsigned tm[RW];         // TM Dz; TE Hz
    unsigned rout;           // rows of the output block inside the grid (bit r)
    bool outc;               // columns of the output block inside the array
    bool act;                // columns inside the array
    unsigned xb;             // rows inside the x layer (bit r): TM of Dz, TE of Hz
    unsigned se, s1, s2;     // rows with source cells: electric, first / second magnetic
    unsigned lines[(3 * RW + 3) / 4];   // end of each (component, row) bucket of RbHit, 8 bits
    float dt, rdx;
};

// shared memory of a tile
struct RbShared {
    float *xch;              // [2 parities][top, bottom][W][RB_C]
    float *psi;              // 4 planes [rows][RB_C] of CPML memory
    int plane;               // floats per plane
    const float *yp;         // y profiles [4][RB_C]: H b, a; E b, a
    const float *xp;         // x profiles [4][xs]: row r of warp w at w RW + r + 1
    int xs;
    float *ws;               // source weight planes (E, H1, H2), tiles with source rows
    const float *amp;        // [3][RB_SLOTS] amplitudes
    const struct RbHit *hits;// this warp's line sample hits
};

// The cells of one line sample on one row: those with column - lo in [0, len) go to
// ring[base + column].
struct __align__(16) RbHit {
    int64_t base;
    int lo, len;
};

template <int RW>
__device__ __forceinline__ unsigned rb_rows_in(int iw, int lo, int hi) {   // bits of lo..hi
    unsigned m = 0;
#pragma unroll
    for (int r = -1; r <= RW; ++r)
        if (iw + r >= lo && iw + r <= hi) m |= 1u << (r + 1);
    return m;
}

template <bool TE, int RW>
__device__ __forceinline__ RbPos<RW> rb_pos(const RbMeta &M, const int4 a, int rows_out, int w,
                                        int lane, int W) {
    const mtb_yee2d_struct &S = M.s;
    RbPos<RW> p;
    p.nx = S.nx; p.ny = S.ny; p.P = S.pitch;
    p.w = w; p.lane = lane; p.W = W;
    p.iw = a.y - RB_T + w * RW;
    p.jb = a.z - 4 + 4 * lane;
    p.dt = S.dt;
    p.rdx = 1.0f / S.dx;
    p.act = p.jb >= 0 && p.jb < p.P;
    p.outc = p.act && lane >= 1 && lane <= 30;
    const int nx = p.nx, ny = p.ny;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int j = p.jb + q;
        const bool h = j >= 0 && j <= ny - 2, in = j >= 1 && j <= ny - 2;
        p.ca[q] = (TE ? in : h) ? ~0u : 0u;
        p.cb[q] = (TE ? h : in) ? ~0u : 0u;
    }
#pragma unroll
    for (int r = 0; r <= RW; ++r) {
        const int i = p.iw + r - (TE ? 0 : 1);
        p.ty[r] = (TE ? (i >= 1 && i <= nx - 2) : (i >= 0 && i <= nx - 2)) ? ~0u : 0u;
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int i = p.iw + r;
        p.tm[r] = (TE ? (i >= 0 && i <= nx - 2) : (i >= 1 && i <= nx - 2)) ? ~0u : 0u;
    }
    p.rout = (rb_rows_in<RW>(p.iw, a.y, min(a.y + rows_out, nx) - 1) >> 1) & ((1u << RW) - 1);
    p.xb = 0;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int i = p.iw + r;
        if (TE ? (i >= 0 && i <= nx - 2 && in_band(i, S.xband[0], S.xband[1]))
               : (i >= 1 && i <= nx - 2 && in_band(i, S.xband[2], S.xband[3])))
            p.xb |= 1u << r;
    }
    p.se = p.s1 = p.s2 = 0;
    if (a.w & RBF_SRC) {
        if (S.src_e.n > 0) p.se = rb_rows_in<RW>(p.iw, S.src_e.row_lo, S.src_e.row_hi);
        if (S.src_h1.n > 0) p.s1 = rb_rows_in<RW>(p.iw, S.src_h1.row_lo, S.src_h1.row_hi);
        if (S.src_h2.n > 0) p.s2 = rb_rows_in<RW>(p.iw, S.src_h2.row_lo, S.src_h2.row_hi);
    }
    return p;
}

// The line samples of this warp's output rows as hits in shared memory, sorted by
// (component, row); bucket ends packed into p.lines. Done once per launch: a sub-step then
// spends a shared load and four predicated stores per hit instead of a scan of the
// descriptors (1.2 us of a 2.9 us step with two flux lines).
template <int RW>
__device__ __forceinline__ void rb_hits(const RbMeta &M, const int4 a, RbPos<RW> &p, RbHit *h) {
    int n = 0;
#pragma unroll
    for (int k = 0; k < (3 * RW + 3) / 4; ++k) p.lines[k] = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int i = p.iw + r;
            if ((a.w & RBF_LINES) && ((p.rout >> r) & 1u))
                for (int l = 0; l < M.s.n_lines; ++l) {
                    const mtb_line_sample &s = M.lines[l];
                    if (s.comp != c) continue;
                    RbHit q;
                    if (s.kind == 0) {
                        if (s.index != i) continue;
                        q.base = (int64_t)s.ring_off - s.lo;
                        q.lo = s.lo;
                        q.len = s.hi - s.lo;
                    } else {
                        if (i < s.lo || i >= s.hi) continue;
                        q.base = (int64_t)s.ring_off + (i - s.lo) - s.index;
                        q.lo = s.index;
                        q.len = 1;
                    }
                    // columns of the output block only
                    const int lo = max(q.lo, a.z), hi = min(q.lo + q.len, a.z + RB_OUTC);
                    if (lo >= hi) continue;
                    q.lo = lo;
                    q.len = hi - lo;
                    if (p.lane == 0) h[n] = q;
                    ++n;
                }
            const int k = c * RW + r;
            p.lines[k >> 2] |= (unsigned)n << (8 * (k & 3));
        }
}

// Subtract the source cells of tile row r (-1 .. RW) from v.
template <int RW>
__device__ __forceinline__ void rb_source(int which, const RbPos<RW> &p, const RbShared &sh, int r,
                                          int s, float (&v)[4]) {
    const int row = p.w * RW + r;
    if (row < 0 || row >= p.W * RW) return;
    const float a = sh.amp[which * RB_SLOTS + s];
    float wv[4];
    lds4(sh.ws + which * sh.plane + row * RB_C + 4 * p.lane, wv);
#pragma unroll
    for (int q = 0; q < 4; ++q)              // (an infinite amplitude leaves other cells alone)
        v[q] = wv[q] != 0.f ? __fsub_rn(v[q], __fmul_rn(a, wv[q])) : v[q];
}

template <int RW>
__device__ __forceinline__ void rb_sample(const RbMeta &M, const RbPos<RW> &p, const RbShared &sh,
                                          const float (&m)[RW][4], const float (&x)[RW][4],
                                          const float (&y)[RW][4], float *ring) {
    const mtb_yee2d_struct &S = M.s;
    if (p.outc) {
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            if (!((p.rout >> r) & 1u)) continue;
            const uint32_t ro = (uint32_t)((p.iw + r) * p.P + p.jb);
            if (S.ring_full[0] >= 0) st4(ring + S.ring_full[0] + ro, m[r]);
            if (S.ring_full[1] >= 0) st4(ring + S.ring_full[1] + ro, x[r]);
            if (S.ring_full[2] >= 0) st4(ring + S.ring_full[2] + ro, y[r]);
        }
    }
    if (p.lines[(3 * RW - 1) >> 2] >> (8 * ((3 * RW - 1) & 3)) == 0) return;   // no hits
    int k0 = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int k = c * RW + r;
            const int k1 = (p.lines[k >> 2] >> (8 * (k & 3))) & 0xff;
            const float(&v)[4] = c == 0 ? m[r] : c == 1 ? x[r] : y[r];
            for (; k0 < k1; ++k0) {
                const RbHit h = sh.hits[k0];
                float *o = ring + h.base + p.jb;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if ((unsigned)(p.jb + q - h.lo) < (unsigned)h.len) o[q] = v[q];
            }
        }
}

// The rows of the warps above and below: publish the warp's top and bottom rows, one
// barrier, read the neighbours' (zero beyond the tile).
template <int RW>
__device__ __forceinline__ void rb_exchange(const RbShared &sh, const RbPos<RW> &p, int par,
                                            const float (&top)[4], const float (&bot)[4],
                                            float (&above)[4], float (&below)[4]) {
    float *t = sh.xch + par * 2 * p.W * RB_C + p.w * RB_C + 4 * p.lane;
    float *b = t + p.W * RB_C;
    st4(t, top);
    st4(b, bot);
    __syncthreads();
    if (p.w > 0) lds4(b - RB_C, above);
    else zero4(above);
    if (p.w + 1 < p.W) lds4(t + RB_C, below);
    else zero4(below);
}

// The update's rounding is written out (no contraction is left to the compiler) and is that
// of the kernel which would run the same plan launch by launch, so that results are the same
// bit for bit whichever of the two advances it (a term with psi = 0 adds 0 exactly):
//  - the temporally blocked kernels: tiles here never straddle one of their 24 x 120 output
//    blocks; where a row has no term of a layer (no y layer in the tile, the row outside the
//    x layer) the curl is one fma, else a difference of the two rounded terms; their lean TE
//    tiles form E = D / eps of a cell's own, or of its right neighbour's, inside the
//    difference (LEAN);
//  - CL: the cluster kernel, which forms Ez = Dz / eps of the own cell inside the
//    difference (one rounding less) where its neighbour's comes from memory.
__device__ __forceinline__ float rb_d(float a, float b, float rdx) {       // (a - b) / dx
    return __fmul_rn(__fsub_rn(a, b), rdx);
}
__device__ __forceinline__ float rb_and(float v, unsigned mask) {
    return __uint_as_float(__float_as_uint(v) & mask);
}
// CPML term: t = d + q with q = b psi + a d (kappa = 1), psi <- q
__device__ __forceinline__ float rb_cpml(float d, float b, float a, float &psi) {
    psi = __fmaf_rn(b, psi, __fmul_rn(a, d));
    return __fadd_rn(d, psi);
}

// ------------------------------------------------------------------ TM sub-step
// Hx, Hy(n+1/2) from Ez(n) (core/stepper_tm.py:85-128) with the magnetic sheets; Dz(n+1)
// with PEC walls (:130-166); the electric source (:197-200); Ez = Dz / eps (:224-231).
// Straight-line code between the exchange and the (rare) sources and samples, one
// instance per kind of tile: with the layer and source tests inside the row loops the
// update falls into dozens of short blocks, each with its own exposed latencies.
template <int RW, bool XL, bool YL, bool LEAN, bool CL>
__device__ __forceinline__ void rb_step(RbTile<false, RW> &T, const RbMeta &M,
                                        const RbPos<RW> &p, const RbShared &sh, int s, int par,
                                        const RbCtx &C) {
    const float rdx = p.rdx, dt = p.dt;
    float *psi = sh.psi + (p.w * RW) * RB_C + 4 * p.lane;
    const float *xp = sh.xp + p.w * RW + 1;
    float ea[4], eb[4];
    rb_exchange(sh, p, par, T.e[0], CL ? T.m[RW - 1] : T.e[RW - 1], ea, eb);   // CL: Dz above
    // ---- Hy of the row above (yh) and of the own rows
#pragma unroll
    for (int r = -1; r < RW; ++r) {
        float(&h)[4] = r < 0 ? T.yh : T.y[r < 0 ? 0 : r];
        float ps[4], b = 1.f, a = 0.f;
        if (XL) {
            b = xp[r]; a = xp[sh.xs + r];
            if (r < 0) copy4(ps, T.ph);
            else lds4(psi + sh.plane + r * RB_C, ps);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float e0 = r < 0 ? ea[q] : T.e[r < 0 ? 0 : r][q];
            const float e1 = r + 1 < RW ? T.e[r + 1 < RW ? r + 1 : 0][q] : eb[q];
            // CL: e1 - Dz / eps of the row itself
            const float d = CL ? __fmul_rn(__fmaf_rn(r < 0 ? -ea[q] : -T.m[r < 0 ? 0 : r][q],
                                                     r < 0 ? T.iah[q] : T.ia[r < 0 ? 0 : r][q],
                                                     e1), rdx)
                               : rb_d(e1, e0, rdx);
            const float t = rb_and(d, p.ty[r + 1]);
            h[q] = __fmaf_rn(dt, XL ? rb_cpml(t, b, a, ps[q]) : t, h[q]);
        }
        if (XL) {
            if (r < 0) copy4(T.ph, ps);
            else st4(psi + sh.plane + r * RB_C, ps);
        }
    }
    // ---- Hx
    float yb[4], ya[4];
    if (YL) { lds4(sh.yp + 4 * p.lane, yb); lds4(sh.yp + RB_C + 4 * p.lane, ya); }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float er4 = __shfl_down_sync(0xffffffffu, T.e[r][0], 1);    // lane 31: halo
        float ps[4];
        if (YL) lds4(psi + r * RB_C, ps);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float er = q < 3 ? T.e[r][q < 3 ? q + 1 : 3] : er4;
            constexpr int q1[4] = {1, 2, 3, 3};
            const float d =
                !CL ? rb_d(er, T.e[r][q], rdx)
                : (q == 0 || q == 3)
                    ? __fmul_rn(__fmaf_rn(-T.m[r][q], T.ia[r][q], er), rdx)
                    : __fmul_rn(__fmaf_rn(T.m[r][q1[q]], T.ia[r][q1[q]], -T.e[r][q]), rdx);
            const float c = rb_and(d, p.ca[q]);
            T.x[r][q] = __fmaf_rn(-dt, YL ? rb_cpml(c, yb[q], ya[q], ps[q]) : c, T.x[r][q]);
        }
        if (YL) st4(psi + r * RB_C, ps);
    }
    if (p.s1 | p.s2) {
        if (p.s1 & 1u) rb_source(1, p, sh, -1, s, T.yh);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            if ((p.s1 >> (r + 1)) & 1u) rb_source(1, p, sh, r, s, T.y[r]);
            if ((p.s2 >> (r + 1)) & 1u) rb_source(2, p, sh, r, s, T.x[r]);
        }
    }
    // ---- Dz, source, Ez
    if (YL) { lds4(sh.yp + 2 * RB_C + 4 * p.lane, yb); lds4(sh.yp + 3 * RB_C + 4 * p.lane, ya); }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float hm4 = __shfl_up_sync(0xffffffffu, T.x[r][3], 1);      // lane 0: halo
        float p2[4], p3[4], b = 1.f, a = 0.f;
        if (XL) {
            b = xp[2 * sh.xs + r]; a = xp[3 * sh.xs + r];
            lds4(psi + 2 * sh.plane + r * RB_C, p2);
        }
        if (YL) lds4(psi + 3 * sh.plane + r * RB_C, p3);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float ha = r > 0 ? T.y[r > 0 ? r - 1 : 0][q] : T.yh[q];
            const float hm = q > 0 ? T.x[r][q > 0 ? q - 1 : 0] : hm4;
            const unsigned v = p.cb[q] & p.tm[r];
            const float fy = rb_and(__fsub_rn(T.y[r][q], ha), v);
            const float dhy = __fmul_rn(fy, rdx);
            const float dhx = rb_and(rb_d(T.x[r][q], hm, rdx), v);
            const float ty = XL ? rb_cpml(dhy, b, a, p2[q]) : dhy;
            const float tx = YL ? rb_cpml(dhx, yb[q], ya[q], p3[q]) : dhx;
            const float c0 = __fsub_rn(ty, tx);
            const float c1 = __fmaf_rn(fy, rdx, -tx);
            const float curl = (CL || YL) ? c0 : !XL ? c1 : ((p.xb >> r) & 1u) ? c0 : c1;
            T.m[r][q] = __fmaf_rn(dt, curl, T.m[r][q]);
        }
        if (XL) st4(psi + 2 * sh.plane + r * RB_C, p2);
        if (YL) st4(psi + 3 * sh.plane + r * RB_C, p3);
    }
    if (p.se) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
            if ((p.se >> (r + 1)) & 1u)
                rb_source(0, p, sh, r, s, T.m[r]);
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) T.e[r][q] = __fmul_rn(T.m[r][q], T.ia[r][q]);
    rb_sample<RW>(M, p, sh, T.e, T.x, T.y, C.ring + (int64_t)s * C.slot_elems);
}

// ------------------------------------------------------------------ TE sub-step
// Dx, Dy(n+1/2) from Hz(n) with CPML (core/stepper_te.py:73-111), the source into Dy
// (:120-134), E = D / eps (:150-175); Hz(n+1) from E(n+1/2) (:113-117) with the sheet.
template <int RW, bool XL, bool YL, bool LEAN, bool CL>
__device__ __forceinline__ void rb_step(RbTile<true, RW> &T, const RbMeta &M,
                                        const RbPos<RW> &p, const RbShared &sh, int s, int par,
                                        const RbCtx &C) {
    const float rdx = p.rdx, dt = p.dt;
    float *psi = sh.psi + (p.w * RW) * RB_C + 4 * p.lane;
    const float *xp = sh.xp + p.w * RW + 1;
    float ha[4], hb[4];
    rb_exchange(sh, p, par, T.m[0], T.m[RW - 1], ha, hb);
    // ---- Dy of the own rows and of the row below (yh)
#pragma unroll
    for (int r = 0; r <= RW; ++r) {
        float(&h)[4] = r == RW ? T.yh : T.y[r < RW ? r : 0];
        float ps[4], b = 1.f, a = 0.f;
        if (XL) {
            b = xp[2 * sh.xs + r]; a = xp[3 * sh.xs + r];
            if (r == RW) copy4(ps, T.ph);
            else lds4(psi + sh.plane + r * RB_C, ps);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float h1 = r == RW ? hb[q] : T.m[r < RW ? r : 0][q];
            const float h0 = r == 0 ? ha[q] : T.m[r > 0 ? r - 1 : 0][q];
            const float d = rb_and(rb_d(h1, h0, rdx), p.ty[r]);
            h[q] = __fmaf_rn(-dt, XL ? rb_cpml(d, b, a, ps[q]) : d, h[q]);
        }
        if (XL) {
            if (r == RW) copy4(T.ph, ps);
            else st4(psi + sh.plane + r * RB_C, ps);
        }
    }
    // ---- Dx / Ex
    float ex[RW][4], ey[RW][4], eyb[4], yb[4], ya[4];
    if (YL) { lds4(sh.yp + 2 * RB_C + 4 * p.lane, yb); lds4(sh.yp + 3 * RB_C + 4 * p.lane, ya); }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float hm4 = __shfl_up_sync(0xffffffffu, T.m[r][3], 1);      // lane 0: halo
        float ps[4];
        if (YL) lds4(psi + r * RB_C, ps);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float hm = q > 0 ? T.m[r][q > 0 ? q - 1 : 0] : hm4;
            const float d = rb_and(rb_d(T.m[r][q], hm, rdx), p.ca[q]);
            T.x[r][q] = __fmaf_rn(dt, YL ? rb_cpml(d, yb[q], ya[q], ps[q]) : d, T.x[r][q]);
            ex[r][q] = __fmul_rn(T.x[r][q], T.ia[r][q]);
        }
        if (YL) st4(psi + r * RB_C, ps);
    }
    if (p.se) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
            if ((p.se >> (r + 1)) & 1u) rb_source(0, p, sh, r, s, T.y[r]);
        if ((p.se >> (RW + 1)) & 1u) rb_source(0, p, sh, RW, s, T.yh);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) eyb[q] = __fmul_rn(T.yh[q], T.ibh[q]);
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) ey[r][q] = __fmul_rn(T.y[r][q], T.ib[r][q]);
    // ---- Hz, sheet
    if (YL) { lds4(sh.yp + 4 * p.lane, yb); lds4(sh.yp + RB_C + 4 * p.lane, ya); }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const float ex4 = __shfl_down_sync(0xffffffffu, ex[r][0], 1);     // lane 31: halo
        float p2[4], p3[4], b = 1.f, a = 0.f;
        if (XL) {
            b = xp[r]; a = xp[sh.xs + r];
            lds4(psi + 2 * sh.plane + r * RB_C, p2);
        }
        if (YL) lds4(psi + 3 * sh.plane + r * RB_C, p3);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float en = r + 1 < RW ? ey[r + 1 < RW ? r + 1 : 0][q] : eyb[q];
            const float exn = q < 3 ? ex[r][q < 3 ? q + 1 : 3] : ex4;
            constexpr int q1[4] = {1, 2, 3, 3};
            const unsigned v = p.cb[q] & p.tm[r];
            const float fy = LEAN ? __fmaf_rn(-T.y[r][q], T.ib[r][q], en)
                                  : rb_and(__fsub_rn(en, ey[r][q]), v);
            const float fx = !LEAN    ? rb_and(__fsub_rn(exn, ex[r][q]), v)
                             : q == 3 ? __fmaf_rn(-T.x[r][q], T.ia[r][q], exn)
                                      : __fmaf_rn(T.x[r][q1[q]], T.ia[r][q1[q]], -ex[r][q]);
            const float dey = __fmul_rn(fy, rdx);
            const float dex = __fmul_rn(fx, rdx);
            const float ty = XL ? rb_cpml(dey, b, a, p2[q]) : dey;
            const float tx = YL ? rb_cpml(dex, yb[q], ya[q], p3[q]) : dex;
            const float c0 = __fsub_rn(ty, tx);
            const float c1 = __fmaf_rn(fy, rdx, -tx);
            const float curl = YL ? c0 : !XL ? c1 : ((p.xb >> r) & 1u) ? c0 : c1;
            T.m[r][q] = __fmaf_rn(-dt, curl, T.m[r][q]);
        }
        if (XL) st4(psi + 2 * sh.plane + r * RB_C, p2);
        if (YL) st4(psi + 3 * sh.plane + r * RB_C, p3);
    }
    if (p.s1) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
            if ((p.s1 >> (r + 1)) & 1u)
                rb_source(1, p, sh, r, s, T.m[r]);
    }
    rb_sample<RW>(M, p, sh, T.m, ex, ey, C.ring + (int64_t)s * C.slot_elems);
}

// Sub-steps s0 .. s1-1 of a tile.
template <bool TE, int RW, bool CL>
__device__ __forceinline__ void rb_steps(RbTile<TE, RW> &T, const RbMeta &M, const RbPos<RW> &p,
                                         const RbShared &sh, int fl, int s0, int s1,
                                         const RbCtx &C) {
    switch (fl & (RBF_XL | RBF_YL)) {
        case 0:
            if (TE && (fl & RBF_LEAN))
                for (int s = s0; s < s1; ++s)
                    rb_step<RW, false, false, TE, CL>(T, M, p, sh, s, s & 1, C);
            else
                for (int s = s0; s < s1; ++s)
                    rb_step<RW, false, false, false, CL>(T, M, p, sh, s, s & 1, C);
            break;
        case RBF_XL:
            for (int s = s0; s < s1; ++s)
                rb_step<RW, true, false, false, CL>(T, M, p, sh, s, s & 1, C);
            break;
        case RBF_YL:
            for (int s = s0; s < s1; ++s)
                rb_step<RW, false, true, false, CL>(T, M, p, sh, s, s & 1, C);
            break;
        default:
            for (int s = s0; s < s1; ++s)
                rb_step<RW, true, true, false, CL>(T, M, p, sh, s, s & 1, C);
    }
}

// ------------------------------------------------------------------ loads and stores
// The x layer memory (psi 1, 2) lives on rows of the x bands, the y layer memory (psi 0,
// 3) on float4s that touch the y bands; row / column sets as the one-step kernels use them.
template <bool TE>
struct RbBand {
    bool y0, y3;             // this lane's columns
    template <int RW>
    __device__ RbBand(const mtb_yee2d_struct &S, const RbPos<RW> &p) {
        // TM: psi 0 on the H side, psi 3 on the E side; TE the other way round
        const bool h = p.act && band4(p.jb, S.yband[0], S.yband[1]);
        const bool e = p.act && band4(p.jb, S.yband[2], S.yband[3]);
        y0 = TE ? e : h;
        y3 = TE ? h : e;
    }
    // psi 0, 1, 2, 3 of structure row i
    __device__ __forceinline__ void rows(const mtb_yee2d_struct &S, int nx, int i, bool (&on)[4]) const {
        const bool hr = i >= 0 && i <= nx - 2, er = i >= 1 && i <= nx - 2;
        const bool xh = hr && in_band(i, S.xband[0], S.xband[1]);
        const bool xe = er && in_band(i, S.xband[2], S.xband[3]);
        const bool in = i >= 0 && i < nx;
        on[0] = y0 && (TE ? hr : in);
        on[1] = TE ? xe : xh;
        on[2] = TE ? xh : xe;
        on[3] = y3 && (TE ? hr : er);
    }
};

__device__ __forceinline__ void rb_ldcg(const float *p, float (&v)[4]) {   // L2 (not L1)
    const float4 x = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}

// CPML memory of tile row r (structure row i) from buffer b into the thread's slots; zero
// where there is none
template <bool TE, bool CG, int RW>
__device__ __forceinline__ void rb_load_psi(const mtb_yee2d_struct &S, const RbPos<RW> &p,
                                            const RbBand<TE> &B, float *psi, int plane, int i,
                                            bool in, int b, int flags) {
    bool on[4];
    B.rows(S, p.nx, i, on);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!(flags & ((k == 0 || k == 3) ? RBF_YL : RBF_XL))) continue;
        float v[4];
        zero4(v);
        if (in && on[k]) {
            const float *src = S.psi[k][b] + (uint32_t)(i * p.P + p.jb);
            if (CG) rb_ldcg(src, v);
            else ld4(src, v);
        }
        st4(psi + k * plane, v);
    }
}

// Store this thread's cells of row r (fields and CPML memory) to buffer b.
template <bool TE, int RW>
__device__ __forceinline__ void rb_store_row(const RbTile<TE, RW> &T, const mtb_yee2d_struct &S,
                                             const RbPos<RW> &p, const RbBand<TE> &B,
                                             const RbShared &sh, int r, const float (&m)[4],
                                             const float (&x)[4], const float (&y)[4], int b,
                                             int flags) {
    const int i = p.iw + r;
    const uint32_t ro = (uint32_t)(i * p.P + p.jb);
    st4(S.f_main[b] + ro, m);
    st4(S.f_x[b] + ro, x);
    st4(S.f_y[b] + ro, y);
    if (flags & (RBF_XL | RBF_YL)) {
        bool on[4];
        B.rows(S, p.nx, i, on);
        const float *psi = sh.psi + (p.w * RW + r) * RB_C + 4 * p.lane;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (on[k]) {
                float v[4];
                lds4(psi + k * sh.plane, v);
                st4(S.psi[k][b] + ro, v);
            }
    }
}

// Profiles of the tile: y profiles of its columns, x profiles of its rows and the row
// before and after, (1, 0) off the arrays and outside the bands.
template <bool TE>
__device__ __forceinline__ void rb_profiles(const mtb_yee2d_struct &S, int r0, int c0, int rows,
                                            float *yp, float *xp, int xs, int flags, int tid,
                                            int nt) {
    const int nx = S.nx, ny = S.ny;
    if (flags & RBF_YL)
        for (int e = tid; e < RB_C; e += nt) {
            const int j = c0 - 4 + e;
            const bool oh = j >= 0 && j <= ny - 2 && in_band(j, S.yband[0], S.yband[1]);
            const bool oe = j >= 1 && j <= ny - 2 && in_band(j, S.yband[2], S.yband[3]);
            yp[e] = oh ? __ldg(S.hy_b + j) : 1.f;
            yp[RB_C + e] = oh ? __ldg(S.hy_a + j) : 0.f;
            yp[2 * RB_C + e] = oe ? __ldg(S.ey_b + j) : 1.f;
            yp[3 * RB_C + e] = oe ? __ldg(S.ey_a + j) : 0.f;
        }
    if (flags & RBF_XL)
        for (int e = tid; e < rows + 2; e += nt) {
            const int i = r0 - RB_T - 1 + e;
            const bool oh = i >= 0 && i <= nx - 2 && in_band(i, S.xband[0], S.xband[1]);
            const bool oe = i >= 1 && i <= nx - 2 && in_band(i, S.xband[2], S.xband[3]);
            xp[e] = oh ? __ldg(S.hx_b + i) : 1.f;
            xp[xs + e] = oh ? __ldg(S.hx_a + i) : 0.f;
            xp[2 * xs + e] = oe ? __ldg(S.ex_b + i) : 1.f;
            xp[3 * xs + e] = oe ? __ldg(S.ex_a + i) : 0.f;
        }
}

// ------------------------------------------------------------------ resident kernel
// exchange rows (two parities and the extra row), CPML planes, weight planes, y and x
// profiles, amplitudes, line hits (hits per warp), record; at least more than half an SM's
// shared memory, so that the blocks spread over the SMs
__host__ __device__ constexpr size_t rb_res_smem(int W, int RW, int hits) {
    const size_t b = sizeof(float) * (6 * (size_t)W * RB_C + 7 * (size_t)W * RW * RB_C + 4 * RB_C +
                                      4 * ((size_t)W * RW + 4) + 3 * RB_SLOTS) +
                     sizeof(RbHit) * (size_t)W * hits + sizeof(RbMeta) + 16;
    return b > 120 * 1024 ? b : 120 * 1024;
}

__device__ __forceinline__ int rb_ld_relaxed(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void rb_st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <bool TE, int RW, bool CL>
__global__ void __launch_bounds__(32 * RB_WARPS, 1) k_rb_resident(const __grid_constant__ RbCtx C) {
    extern __shared__ __align__(1024) unsigned char rb_raw[];
    const int W = blockDim.x >> 5, ROWS = W * RW, PL = ROWS * RB_C;
    RbShared sh;
    sh.xch = reinterpret_cast<float *>(rb_raw);
    float *xx = sh.xch + 4 * W * RB_C;       // extra row: [top, bottom][W][RB_C]
    sh.psi = xx + 2 * W * RB_C;
    sh.plane = PL;
    sh.ws = sh.psi + 4 * PL;
    float *yp = sh.ws + 3 * PL, *xp = yp + 4 * RB_C;
    sh.xs = ROWS + 4;
    sh.yp = yp;
    sh.xp = xp;
    float *amp = xp + 4 * (ROWS + 4);
    sh.amp = amp;
    RbHit *hits = reinterpret_cast<RbHit *>(amp + 3 * RB_SLOTS);
    RbMeta &M = *reinterpret_cast<RbMeta *>(hits + (size_t)W * C.hits);
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, w = tid >> 5;
    const int4 wk = __ldg(C.work + (size_t)RB_WORK * blockIdx.x);
    const int rout = __ldg(&C.work[(size_t)RB_WORK * blockIdx.x + 1].x);
    const int fl = wk.w;
    for (int b = tid; b < (int)(sizeof(RbMeta) / 4); b += nt)
        reinterpret_cast<int *>(&M)[b] = __ldg(reinterpret_cast<const int *>(C.meta + wk.x) + b);
    const int epoch0 = *reinterpret_cast<volatile int *>(C.flags + blockIdx.x);
    const int nbr = tid < 8 ? __ldg(C.nb + 8 * blockIdx.x + tid) : -1;
    __syncthreads();
    const mtb_yee2d_struct &S = M.s;
    RbPos<RW> p = rb_pos<TE, RW>(M, wk, rout, w, lane, W);
    sh.hits = hits + (size_t)w * C.hits;
    rb_hits<RW>(M, wk, p, hits + (size_t)w * C.hits);
    const RbBand<TE> B(S, p);
    const int cell = w * RW * RB_C + 4 * lane;
    if (fl & (RBF_XL | RBF_YL)) rb_profiles<TE>(S, wk.y, wk.z, ROWS, yp, xp, sh.xs, fl, tid, nt);
    if (fl & RBF_SRC) {
        for (int s = tid; s < C.nsub; s += nt) {
            const size_t o = (size_t)s * C.ncols;
            amp[s] = S.src_e.n > 0 ? C.amp_e[o + S.src_e.amp_col] : 0.f;
            amp[RB_SLOTS + s] = S.src_h1.n > 0 ? C.amp_h[o + S.src_h1.amp_col] : 0.f;
            amp[2 * RB_SLOTS + s] = S.src_h2.n > 0 ? C.amp_h[o + S.src_h2.amp_col] : 0.f;
        }
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int i = p.iw + r;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const mtb_cells &cl = k == 0 ? S.src_e : k == 1 ? S.src_h1 : S.src_h2;
                float v[4];
                zero4(v);
                if (p.act && i >= 0 && i < p.nx && cl.n > 0) apply_cells_a(cl, i, -1.f, p.jb, v);
                st4(sh.ws + k * PL + cell + r * RB_C, v);
            }
        }
    }
    // rows of the output block and of its halo (a tile may have spare rows below)
    const unsigned rin = (rb_rows_in<RW>(p.iw, max(wk.y - RB_T, 0),
                                         min(wk.y + rout + RB_T, p.nx) - 1) >> 1) &
                         ((1u << RW) - 1);
    RbTile<TE, RW> T;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int i = p.iw + r;
        const bool in = p.act && ((rin >> r) & 1u);
        zero4(T.m[r]); zero4(T.x[r]); zero4(T.y[r]); zero4(T.ia[r]);
        if (TE) zero4(T.ib[TE ? r : 0]);
        if (in) {
            const uint32_t g = (uint32_t)(i * p.P + p.jb);
            ld4(S.f_main[C.par] + g, T.m[r]);
            ld4(S.f_x[C.par] + g, T.x[r]);
            ld4(S.f_y[C.par] + g, T.y[r]);
            ld4(S.inv_eps_a + g, T.ia[r]);
            if (TE) ld4(S.inv_eps_b + g, T.ib[TE ? r : 0]);
        }
        if (fl & (RBF_XL | RBF_YL))
            rb_load_psi<TE, false>(S, p, B, sh.psi + cell + r * RB_C, PL, i, in, C.par, fl);
    }
    // the extra row: its owner's values through rows of their own, so that neither the
    // sub-step before nor the one after needs another barrier
    auto extra_row = [&](const float (&top)[4], const float (&bot)[4], float (&v)[4]) {
        float *t = xx + w * RB_C + 4 * lane, *b = t + W * RB_C;
        st4(t, top);
        st4(b, bot);
        __syncthreads();
        zero4(v);
        if (TE && w + 1 < W) lds4(t + RB_C, v);
        if (!TE && w > 0) lds4(b - RB_C, v);
    };
    // its x-layer memory (the owner updates it only after the next barrier)
    auto extra_psi = [&]() {
        zero4(T.ph);
        if (fl & RBF_XL) {
            if (TE && w + 1 < W) lds4(sh.psi + PL + cell + RW * RB_C, T.ph);
            if (!TE && w > 0) lds4(sh.psi + PL + cell - RB_C, T.ph);
        }
    };
    auto form_e = [&]() {
        if (!TE)
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) T.e[r][q] = __fmul_rn(T.m[r][q], T.ia[r][q]);
    };
    zero4(T.iah);
    if (TE) {
        float v[4];
        extra_row(T.ib[0], T.ib[TE ? RW - 1 : 0], v);
#pragma unroll
        for (int q = 0; q < 4; ++q) T.ibh[TE ? q : 0] = v[q];
        __syncthreads();
    } else if (CL) {
        extra_row(T.ia[0], T.ia[RW - 1], T.iah);
        __syncthreads();
    }
    extra_row(T.y[0], T.y[RW - 1], T.yh);
    extra_psi();
    form_e();
    int ex = 0;
    for (int s0 = 0; s0 < C.nsub; s0 += RB_T) {
        const int s1 = min(s0 + RB_T, C.nsub);
        rb_steps<TE, RW, CL>(T, M, p, sh, fl, s0, s1, C);
        ++ex;
        const int b = C.par ^ (ex & 1);
        const bool last = s1 == C.nsub;
        // ---- the output block (at the end), else its rim
        if (p.outc) {
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int d = w * RW + r - RB_T;               // row of the output block
                const bool rim = last || d < RB_T || d >= rout - RB_T || lane == 1 || lane == 30;
                if (((p.rout >> r) & 1u) && rim)
                    rb_store_row<TE, RW>(T, S, p, B, sh, r, T.m[r], T.x[r], T.y[r], b, fl);
            }
        }
        if (last) break;
        __syncthreads();
        if (tid == 0) rb_st_release(C.flags + blockIdx.x, epoch0 + ex);
        bool ok = true;
        if (nbr >= 0) {
            if (rb_ld_relaxed(C.flags + nbr) - (epoch0 + ex) < 0) {
                const unsigned long long t0 = gtimer();
                while (rb_ld_relaxed(C.flags + nbr) - (epoch0 + ex) < 0)
                    if (gtimer() - t0 > WAIT_NS) {
                        atomicExch(C.err, 1);
                        ok = false;
                        break;
                    }
            }
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
        }
        if (!__syncthreads_and(ok)) return;
        // ---- the halo from the neighbours' rims
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            if (p.outc && ((p.rout >> r) & 1u)) continue;
            const int i = p.iw + r;
            const bool in = p.act && ((rin >> r) & 1u);
            zero4(T.m[r]); zero4(T.x[r]); zero4(T.y[r]);
            if (in) {
                const uint32_t g = (uint32_t)(i * p.P + p.jb);
                rb_ldcg(S.f_main[b] + g, T.m[r]);
                rb_ldcg(S.f_x[b] + g, T.x[r]);
                rb_ldcg(S.f_y[b] + g, T.y[r]);
            }
            if (fl & (RBF_XL | RBF_YL))
                rb_load_psi<TE, true>(S, p, B, sh.psi + cell + r * RB_C, PL, i, in, b, fl);
        }
        extra_row(T.y[0], T.y[RW - 1], T.yh);
        extra_psi();
        form_e();
    }
    // the epoch of a launch without refreshes stays; every block ends on the same one
}

}  // namespace mtb
