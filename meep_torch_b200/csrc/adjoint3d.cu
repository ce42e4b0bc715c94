// Discrete adjoint of the 3D CPML step for sm_100a (with conductive damping:
// H' = d1 H - d2 curl, E' = d1 E + d2 curl / eps, dispersive poles, whose
// recurrence is linear with eps-free coefficients, and PMC walls): the exact transpose of
// the split H / E update (core/stepper_3d.py:363-437, the same arithmetic as
// k_yee3d_h / k_yee3d_e) and of the plane sampling (core/monitors_3d.py:70-189)
// -- the reverse sweep of the reference's run_3d_adjoint
// (core/adjoint3d.py:56-115). Sources are additive constants; their only
// derivative is through eps (E += s / eps_c), which the E-increment form below
// carries.
//
// Reverse of forward step t, adjoint state A = d J / d state_{t+1} on entry:
//   inject  monitor plane samples of state_{t+1} -> gE, gH (scatter)
//   E part  E' = E + (dt curl + s) / eps_c:
//             d J / d eps_c = -gE' (E' - E) / eps_c, its numerator summed over the
//             steps of a run                               -> tmp6..8
//             g_curl = dt gE' / eps_c on the curl interior
//             E-side psi transposes -> g_psi6..11, adjoints of the six
//             H differences -> tmp0..5; gE passes through (identity)
//   H part  gH += transposed differences of tmp0..5; H' = H - dt curl E:
//             H-side psi transposes -> g_psi0..5, adjoints of the six E
//             differences -> tmp9..14
//   fin     gE += transposed differences of tmp9..14
// After the steps of a run, k_adj3_eps divides tmp6..8 by the averages and gathers the
// two cells of each Yee average into g_eps: the average is linear, so one gather of the
// sum replaces one per step.
// tmp index: 0 Ex:dy(Hz) 1 Ex:dz(Hy) 2 Ey:dz(Hx) 3 Ey:dx(Hz) 4 Ez:dx(Hy)
// 5 Ez:dy(Hx) 6 eps_x 7 eps_y 8 eps_z 9 Hx:dy(Ez) 10 Hx:dz(Ey) 11 Hy:dz(Ex)
// 12 Hy:dx(Ez) 13 Hz:dx(Ey) 14 Hz:dy(Ex); tmp0..5 and 9..14 are zero outside the
// cells where their term exists.
// Launches per step: H part, inject, and fin of the step with the E part of the one
// before it (k_adj3_fe): both touch only their own node, so gE makes one round trip.
#include <algorithm>
#include <vector>

#include "mtb_common.cuh"

namespace mtb {

constexpr int A3_T = 128;         // float4s per block, three components each

struct Adj3 {
    mtb_adj3d_buffers b;
    const float *eps;
    const float *pb[3][2];
    const float *pa[3][2];
    const float *dmp[6][2];       // conductive damping (d1, d2) per component, or null
    const float *c3[3];           // pole drives per E component (np box planes each)
    float c1[MTB_MAX_POLES], c2[MTB_MAX_POLES];
    int np;                       // dispersive poles (0: none)
    int pmc;                      // PMC walls: bit 0 x, 1 y, 2 z
    int psi_all;                  // 1: g_psi outside the layers too (adjoint_psi_layers)
    int nx, ny, nz, zp;
    float dt, rdx;
};

__device__ __forceinline__ void l4(const float *p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void s4(float *p, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void zz(float (&v)[4]) { v[0] = v[1] = v[2] = v[3] = 0.f; }
__device__ __forceinline__ float prof(const float *p, bool on, float dflt, int k) {
    return on ? __ldg(p + k) : dflt;
}

// gF[cell] += adjoint ring value, for every plane sample of the step.
__global__ void k_adj3_inject(const mtb_yee3d_struct *__restrict__ SS,
                              const int64_t *__restrict__ pstart, int n_planes,
                              const float *__restrict__ radj, mtb_adj3d_buffers B) {
    const mtb_yee3d_struct &S = *SS;
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    pdl_next();
    if (e >= pstart[n_planes]) {
        pdl_wait();
        return;
    }
    int lo = 0, hi = n_planes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pstart[mid] <= e) lo = mid; else hi = mid - 1;
    }
    const int *pl = S.planes + 8 * lo;
    const int comp = pl[0], axis = pl[1], index = pl[2];
    const int w1 = pl[6] - pl[5];
    const int64_t p = e - pstart[lo];
    const int a = pl[3] + (int)(p / w1), b = pl[5] + (int)(p % w1);
    int i, j, k;
    if (axis == 0) { i = index; j = a; k = b; }
    else if (axis == 1) { i = a; j = index; k = b; }
    else { i = a; j = b; k = index; }
    pdl_wait();                          // the descriptor and plane tables are constant
    atomicAdd(B.g[comp] + ((int64_t)i * S.ny + j) * S.zpitch + k,
              radj[S.plane_ring_off[lo] + p]);
}

// The adjoint kernels take a float4 of z of one component per thread (threadIdx.y the
// component, blockIdx.y the x plane, threadIdx.x counting float4s through the plane's
// rows). All three components in one thread took 158 (E) and 128 (H) registers and one
// or two blocks an SM, with the loads' latency exposed: E 52.3 us, H 12.4 us on
// 96 x 80 x 72.
struct A3Cell {
    int i, j, kb, lane;
    uint32_t g;
    bool act;
    __device__ __forceinline__ A3Cell(const Adj3 &P) {
        const uint32_t zq = (uint32_t)P.zp >> 2;
        const uint32_t q = blockIdx.x * (uint32_t)A3_T + threadIdx.x;
        act = q < (uint32_t)P.ny * zq;
        i = blockIdx.y;
        j = (int)(q / zq);
        kb = 4 * (int)(q - (uint32_t)j * zq);
        lane = threadIdx.x & 31;
        g = (uint32_t)i * ((uint32_t)P.ny * P.zp) + 4u * q;
    }
};

// CPML profile (b, a) of one node, (1, 0) where it is not applied
__device__ __forceinline__ void a3_prof(const Adj3 &P, int ax, int h, bool on, int k, float &b,
                                        float &a) {
    b = prof(P.pb[ax][h], on, 1.f, k);
    a = prof(P.pa[ax][h], on, 0.f, k);
}

// gE of component C: += the transposed differences of the H part's adjoints (fin).
template <int C>
__device__ __forceinline__ void a3_fin(const Adj3 &P, const A3Cell &c, float (&ge)[4]) {
    // Ex: dz(Ex) of Hy (11), dy(Ex) of Hz (14); Ey: dz(Ey) of Hx (10), dx(Ey) of Hz (13);
    // Ez: dy(Ez) of Hx (9), dx(Ez) of Hy (12)
    constexpr int UA = C == 0 ? 11 : C == 1 ? 10 : 9, UB = C == 0 ? 14 : C == 1 ? 13 : 12;
    const int ZP = P.zp;
    const uint32_t g = c.g, NYZ = (uint32_t)P.ny * ZP;
    float ua[4], uap[4], ub[4], ubp[4], zk = 0.f;
    zz(ua); zz(uap); zz(ub); zz(ubp);
    if (c.act) {
        l4(P.b.tmp[UA] + g, ua);
        l4(P.b.tmp[UB] + g, ub);
        if (C == 2 && c.j >= 1) l4(P.b.tmp[UA] + g - ZP, uap);
        if (C == 0 && c.j >= 1) l4(P.b.tmp[UB] + g - ZP, ubp);
        if (C != 0 && c.i >= 1) l4(P.b.tmp[UB] + g - NYZ, ubp);
        if (C != 2 && c.lane == 0 && c.kb >= 1) zk = P.b.tmp[UA][g - 1];
    }
    if (C != 2) {
        const float t = __shfl_up_sync(0xffffffffu, ua[3], 1);
        if (c.lane != 0) zk = t;
        if (c.kb == 0) zk = 0.f;
        uap[0] = zk; uap[1] = ua[0]; uap[2] = ua[1]; uap[3] = ua[2];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
        ge[q] += (uap[q] - ua[q]) * P.rdx + (ubp[q] - ub[q]) * P.rdx;
}

// E part of component C. FIN: the fin of the later step first (gE then carries it).
// ADD: tmp6..8 accumulate (clear: this step starts the run's sum). MODE bit 0: damping,
// bit 1: poles.
template <int C, bool FIN, bool ADD, int MODE>
__device__ __forceinline__ void a3_e(const Adj3 &P, const A3Cell &c, const float *en_,
                                     const float *eo_, int64_t rec_comp) {
    constexpr bool DAMP = (MODE & 1) != 0, PL = (MODE & 2) != 0;
    const int nx = P.nx, ny = P.ny, nz = P.nz, ZP = P.zp;
    const int i = c.i, j = c.j, kb = c.kb;
    const uint32_t g = c.g, NYZ = (uint32_t)ny * ZP;
    const mtb_adj3d_buffers &B = P.b;
    const float dt = P.dt;
    const bool act = c.act;
    const bool iin = i >= 1 && i <= nx - 2, jin = j >= 1 && j <= ny - 2;
    const bool xok = i <= nx - 2, vyH = j <= ny - 2;
    // first term (psi 6 + 2C, tmp 2C) and second (psi 7 + 2C, tmp 2C + 1) and their axes:
    // Ex: y, z; Ey: z, x; Ez: x, y
    float b0, a0, b1 = 1.f, a1 = 0.f, zb[4], za[4];
    if (C == 0) a3_prof(P, 1, 1, act && jin, j, b0, a0);
    else a3_prof(P, 0, 1, act && iin, i, b0, a0);
    if (C == 2) a3_prof(P, 1, 1, act && jin, j, b1, a1);
    bool zon = false;
    if (C != 2)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = kb + q;
            a3_prof(P, 2, 1, act && k >= 1 && k <= nz - 2, k, zb[q], za[q]);
            zon |= za[q] != 0.f;
        }
    // the psi adjoint feeds back only through a: outside the layers it is not needed
    const bool pA = act && (P.psi_all || (C == 0 ? a0 != 0.f : C == 1 ? zon : a0 != 0.f));
    const bool pB = act && (P.psi_all || (C == 0 ? zon : C == 1 ? a0 != 0.f : a1 != 0.f));
    float ep[4], epn[4], ge[4], en[4], eo[4], gs[4], g6[4], g7[4], epk = 1.f;
    ep[0] = ep[1] = ep[2] = ep[3] = 1.f;
    epn[0] = epn[1] = epn[2] = epn[3] = 1.f;
    zz(ge); zz(en); zz(eo); zz(gs); zz(g6); zz(g7);
    float d1[4] = {1.f, 1.f, 1.f, 1.f}, d2[4] = {dt, dt, dt, dt};
    if (act) {
        l4(P.eps + g, ep);
        if (C == 0 && i + 1 < nx) l4(P.eps + g + NYZ, epn);
        if (C == 1 && j + 1 < ny) l4(P.eps + g + ZP, epn);
        if (C == 2 && c.lane == 31 && kb + 4 < ZP) epk = P.eps[g + 4];
        l4(B.g[C] + g, ge);
        l4(en_ + C * rec_comp + g, en);
        l4(eo_ + C * rec_comp + g, eo);
        if (ADD) l4(B.tmp[6 + C] + g, gs);
        if (pA) l4(B.g_psi[6 + 2 * C] + g, g6);
        if (pB) l4(B.g_psi[7 + 2 * C] + g, g7);
        // conductive damping: E' = d1 E + (d2 curl + s) / eps_c (core/stepper_3d.py:405-437)
        if (DAMP) { l4(P.dmp[C][0] + g, d1); l4(P.dmp[C][1] + g, d2); }
    }
    if (C == 2) {
        const float t = __shfl_down_sync(0xffffffffu, ep[0], 1);
        if (c.lane != 31) epk = t;
        if (kb + 4 >= ZP) epk = 1.f;
        epn[0] = ep[1]; epn[1] = ep[2]; epn[2] = ep[3]; epn[3] = epk;
    }
    if (FIN) a3_fin<C>(P, c, ge);
    if (!act) return;
    // dispersive poles (core/stepper_3d.py:295-300, :311-322): P(n+1) = c1 P(n) +
    // c2 P(n-1) + c3 E(n), E' = (d1 (E eps_c + sum P(n)) + d2 curl + s - sum P(n+1)) / eps_c.
    // P(n+1) is the next state's P(n), so gN = d J / d P(n+1) = gPc' - gE' / eps_c, and
    //   d J / d E(n) gains sum c3 gN,  gPc = d1 gE' / eps_c + c1 gN + gPp',  gPp = c2 gN.
    float pe[4];
    zz(pe);
    if (PL) {
        const size_t plane = (size_t)nx * NYZ;
#pragma unroll 1
        for (int p = 0; p < P.np; ++p) {
            float *gc_ = B.g_pol[C][0] + p * plane + g;
            float *gq_ = B.g_pol[C][1] + p * plane + g;
            float gpc[4], gpp[4], c3[4];
            l4(gc_, gpc); l4(gq_, gpp); l4(P.c3[C] + p * plane + g, c3);
            const float c1 = P.c1[p], c2 = P.c2[p];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = kb + q;
                if (!(C == 0 ? (xok && k < nz) : C == 1 ? (vyH && k < nz) : (k <= nz - 2)))
                    continue;
                const float ec = 0.5f * (ep[q] + epn[q]);
                const float gE = ge[q];
                const float gN = gpc[q] - gE / ec;
                pe[q] += c3[q] * gN;
                gpc[q] = d1[q] * gE / ec + c1 * gN + gpp[q];
                gpp[q] = c2 * gN;
            }
            s4(gc_, gpc); s4(gq_, gpp);
        }
    }
    // PMC walls (core/stepper_3d.py _term_pmc :99-121): the tangential E on the wall is
    // live, and there the term differentiating along the wall's axis is zero
    const bool iL = iin || (P.pmc & 1), jL = jin || (P.pmc & 2);
    float t0[4], t1[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = kb + q;
        const bool kin = k >= 1 && k <= nz - 2, kL = kin || (P.pmc & 4);
        const bool v = C == 0 ? (xok && k < nz) : C == 1 ? (vyH && k < nz) : (k <= nz - 2);
        const bool in = v && (C == 0 ? jL && kL : C == 1 ? iL && kL : iL && jL);
        const float ec = 0.5f * (ep[q] + epn[q]);
        const float gE = ge[q];
        gs[q] = v ? gs[q] - gE * (en[q] - d1[q] * eo[q]) : gs[q];
        const float gc = in ? d2[q] * gE / ec : 0.f;
        if (DAMP || PL) ge[q] = v ? d1[q] * gE + pe[q] : gE;   // d1 gE (+ poles) to E
        const bool uA = v && (C == 0 ? jin : C == 1 ? kin : iin);
        const bool uB = v && (C == 0 ? kin : C == 1 ? iin : jin);
        const float bA = C == 1 ? zb[q] : b0, aA = C == 1 ? za[q] : a0;
        const float bB = C == 0 ? zb[q] : C == 1 ? b0 : b1;
        const float aB = C == 0 ? za[q] : C == 1 ? a0 : a1;
        const float gA = g6[q] + gc, gB = g7[q] - gc;
        g6[q] = uA ? bA * gA : g6[q];
        g7[q] = uB ? bB * gB : g7[q];
        t0[q] = uA ? gc + aA * gA : 0.f;
        t1[q] = uB ? -gc + aB * gB : 0.f;
    }
    if (FIN || DAMP || PL) s4(B.g[C] + g, ge);
    s4(B.tmp[6 + C] + g, gs);
    s4(B.tmp[2 * C] + g, t0);
    s4(B.tmp[2 * C + 1] + g, t1);
    if (pA) s4(B.g_psi[6 + 2 * C] + g, g6);
    if (pB) s4(B.g_psi[7 + 2 * C] + g, g7);
}

// The E part of one step, after the fin of the step that follows it when FIN. What
// bounds it: the latency of its 18 floats a cell (96 x 80 x 72: 28 % of the DRAM peak, issue
// 46 % active, waiting for loads first of all, at 18 warps an SM and 72 registers). With
// damping and poles together the 80 registers of two blocks an SM spill (208 bytes of stores
// with the fin, 96 without).
template <bool FIN, int MODE>
__global__ void __launch_bounds__(3 * A3_T, 2) k_adj3_fe(const __grid_constant__ Adj3 P,
                                                        const float *__restrict__ en,
                                                        const float *__restrict__ eo,
                                                        int64_t rec_comp) {
    pdl_next();
    const A3Cell c(P);
    pdl_wait();
    if (threadIdx.y == 0) a3_e<0, FIN, FIN, MODE>(P, c, en, eo, rec_comp);
    else if (threadIdx.y == 1) a3_e<1, FIN, FIN, MODE>(P, c, en, eo, rec_comp);
    else a3_e<2, FIN, FIN, MODE>(P, c, en, eo, rec_comp);
}

// H part of component C.
template <int C>
__device__ __forceinline__ void a3_h(const Adj3 &P, const A3Cell &c) {
    // transposed differences of the E part's H derivatives, in the order
    // Hx: 2 (z), 5 (y); Hy: 1 (z), 4 (x); Hz: 0 (y), 3 (x)
    constexpr int TA = C == 0 ? 2 : C == 1 ? 1 : 0, TB = C == 0 ? 5 : C == 1 ? 4 : 3;
    const int nx = P.nx, ny = P.ny, nz = P.nz, ZP = P.zp;
    const int i = c.i, j = c.j, kb = c.kb;
    const uint32_t g = c.g, NYZ = (uint32_t)ny * ZP;
    const mtb_adj3d_buffers &B = P.b;
    const float dt = P.dt, rdx = P.rdx;
    const bool act = c.act, xok = i <= nx - 2, vyH = j <= ny - 2;
    // psi 2C (tmp 9 + 2C) and psi 2C + 1 (tmp 10 + 2C): Hx: y, z; Hy: z, x; Hz: x, y
    float b0, a0, b1 = 1.f, a1 = 0.f, zb[4], za[4];
    if (C == 0) a3_prof(P, 1, 0, act && vyH, j, b0, a0);
    else a3_prof(P, 0, 0, act && xok, i, b0, a0);
    if (C == 2) a3_prof(P, 1, 0, act && vyH, j, b1, a1);
    bool zon = false;
    if (C != 2)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            a3_prof(P, 2, 0, act && kb + q <= nz - 2, kb + q, zb[q], za[q]);
            zon |= za[q] != 0.f;
        }
    const bool pA = act && (P.psi_all || (C == 0 ? a0 != 0.f : C == 1 ? zon : a0 != 0.f));
    const bool pB = act && (P.psi_all || (C == 0 ? zon : C == 1 ? a0 != 0.f : a1 != 0.f));
    float ta[4], tan_[4], tb[4], tbn[4], gh[4], g0[4], g1[4], zk = 0.f;
    zz(ta); zz(tan_); zz(tb); zz(tbn); zz(gh); zz(g0); zz(g1);
    float h1[4] = {1.f, 1.f, 1.f, 1.f}, h2[4] = {dt, dt, dt, dt};
    const bool damp = P.dmp[3][0] != nullptr;
    if (act) {
        l4(B.tmp[TA] + g, ta);
        l4(B.tmp[TB] + g, tb);
        if (C == 2 && j + 1 < ny) l4(B.tmp[TA] + g + ZP, tan_);
        if (C == 0 && j + 1 < ny) l4(B.tmp[TB] + g + ZP, tbn);
        if (C != 0 && i + 1 < nx) l4(B.tmp[TB] + g + NYZ, tbn);
        if (C != 2 && c.lane == 31 && kb + 4 < ZP) zk = B.tmp[TA][g + 4];
        l4(B.g[3 + C] + g, gh);
        if (pA) l4(B.g_psi[2 * C] + g, g0);
        if (pB) l4(B.g_psi[2 * C + 1] + g, g1);
        // conductive damping: H' = d1 H - d2 curl (core/stepper_3d.py:375-393)
        if (damp) { l4(P.dmp[3 + C][0] + g, h1); l4(P.dmp[3 + C][1] + g, h2); }
    }
    if (C != 2) {
        const float t = __shfl_down_sync(0xffffffffu, ta[0], 1);
        if (c.lane != 31) zk = t;
        if (kb + 4 >= ZP) zk = 0.f;
        tan_[0] = ta[1]; tan_[1] = ta[2]; tan_[2] = ta[3]; tan_[3] = zk;
    }
    if (!act) return;
    float u0[4], u1[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = kb + q;
        const bool vz = k <= nz - 2;
        const bool v = C == 0 ? (vyH && vz) : C == 1 ? (xok && vz) : (xok && vyH && k < nz);
        const float gx = gh[q] + (ta[q] - tan_[q]) * rdx + (tb[q] - tbn[q]) * rdx;
        // H -= dt ((A + psi A') - (B + psi B'))
        const float bA = C == 1 ? zb[q] : b0, aA = C == 1 ? za[q] : a0;
        const float bB = C == 0 ? zb[q] : C == 1 ? b0 : b1;
        const float aB = C == 0 ? za[q] : C == 1 ? a0 : a1;
        const float cA = -h2[q] * gx, cB = h2[q] * gx;
        const float gA = g0[q] + cA, gB = g1[q] + cB;
        u0[q] = v ? cA + aA * gA : 0.f;
        u1[q] = v ? cB + aB * gB : 0.f;
        g0[q] = v ? bA * gA : g0[q];
        g1[q] = v ? bB * gB : g1[q];
        gh[q] = v ? h1[q] * gx : gx;
    }
    s4(B.g[3 + C] + g, gh);
    s4(B.tmp[9 + 2 * C] + g, u0);
    s4(B.tmp[10 + 2 * C] + g, u1);
    if (pA) s4(B.g_psi[2 * C] + g, g0);
    if (pB) s4(B.g_psi[2 * C + 1] + g, g1);
}

__global__ void __launch_bounds__(3 * A3_T, 2) k_adj3_h(const __grid_constant__ Adj3 P) {
    pdl_next();
    const A3Cell c(P);
    pdl_wait();
    if (threadIdx.y == 0) a3_h<0>(P, c);
    else if (threadIdx.y == 1) a3_h<1>(P, c);
    else a3_h<2>(P, c);
}

// The last step's fin (gE only).
__global__ void __launch_bounds__(3 * A3_T) k_adj3_fin(const __grid_constant__ Adj3 P) {
    pdl_next();
    const A3Cell c(P);
    pdl_wait();
    const int C = threadIdx.y;
    float ge[4];
    zz(ge);
    if (c.act) l4(P.b.g[C] + c.g, ge);
    if (C == 0) a3_fin<0>(P, c, ge);
    else if (C == 1) a3_fin<1>(P, c, ge);
    else a3_fin<2>(P, c, ge);
    if (c.act) s4(P.b.g[C] + c.g, ge);
}

// g_eps += the run's sums of each component's eps_c adjoint, divided by eps_c, at the two
// cells of its Yee average.
__global__ void __launch_bounds__(A3_T) k_adj3_eps(const __grid_constant__ Adj3 P) {
    pdl_next();
    const A3Cell c(P);
    pdl_wait();
    if (!c.act) return;
    const int i = c.i, j = c.j, ZP = P.zp;
    const uint32_t g = c.g, NYZ = (uint32_t)P.ny * ZP;
    const mtb_adj3d_buffers &B = P.b;
    float e[4], ei[4], eim[4], ej[4], ejm[4], t6[4], t6i[4], t7[4], t7j[4], t8[4], ge[4];
    zz(t6i); zz(t7j);
    l4(P.eps + g, e);
#pragma unroll
    for (int q = 0; q < 4; ++q) ei[q] = eim[q] = ej[q] = ejm[q] = e[q];
    l4(B.tmp[6] + g, t6); l4(B.tmp[7] + g, t7); l4(B.tmp[8] + g, t8);
    if (i + 1 < P.nx) l4(P.eps + g + NYZ, ei);
    if (j + 1 < P.ny) l4(P.eps + g + ZP, ej);
    if (i >= 1) { l4(P.eps + g - NYZ, eim); l4(B.tmp[6] + g - NYZ, t6i); }
    if (j >= 1) { l4(P.eps + g - ZP, ejm); l4(B.tmp[7] + g - ZP, t7j); }
    const float em = c.kb >= 1 ? P.eps[g - 1] : 1.f, t8m = c.kb >= 1 ? B.tmp[8][g - 1] : 0.f;
    const float ekp = c.kb + 4 < ZP ? P.eps[g + 4] : 1.f;
    l4(B.g_eps + g, ge);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = c.kb + q;
        if (k >= P.nz) continue;
        const float ek = q < 3 ? e[q + 1] : ekp, ekm = q > 0 ? e[q - 1] : em;
        const float tk = q > 0 ? t8[q - 1] : t8m;
        // a sum is zero outside its component's cells; the average there may be with padding
        const float x = t6[q] / (0.5f * (e[q] + ei[q])) + t6i[q] / (0.5f * (eim[q] + e[q]));
        const float y = t7[q] / (0.5f * (e[q] + ej[q])) + t7j[q] / (0.5f * (ejm[q] + e[q]));
        const float z = (k <= P.nz - 2 ? t8[q] / (0.5f * (e[q] + ek)) : 0.f) +
                        (k >= 1 ? tk / (0.5f * (ekm + e[q])) : 0.f);
        ge[q] += 0.5f * x + 0.5f * y + 0.5f * z;
    }
    s4(B.g_eps + g, ge);
}

}  // namespace mtb

using namespace mtb;

struct mtb_yee3d_adjoint {
    StreamMarks marks;             // streams its work runs on
    mtb_yee3d_struct s{};
    Adj3 a{};
    DftState dft;
    DevBuf s_d, pstart_d;
    int n_planes = 0;
    int64_t n_samples = 0;
    int64_t last_launches = 0;
};

extern "C" {

int mtb_yee3d_adjoint_create(const mtb_yee3d_struct *s, const mtb_adj3d_buffers *bufs,
                             const mtb_dft_region *regions, int32_t n_regions,
                             const mtb_phase_group *groups, int32_t n_groups,
                             int64_t ring_slot_elems, int32_t ring_slots,
                             mtb_yee3d_adjoint **out) {
    if (!out || !s || !bufs) return fail(MTB_INVALID_ARG, "null argument");
    *out = nullptr;
    const mtb_yee3d_struct &S = *s;
    const bool dmp = S.damp[0][0] != nullptr;
    for (int c = 0; c < 6; ++c)
        for (int h = 0; h < 2; ++h)
            if ((S.damp[c][h] != nullptr) != dmp ||
                (S.damp[c][h] && (reinterpret_cast<uintptr_t>(S.damp[c][h]) & 15)))
                return fail(MTB_INVALID_ARG, "3D adjoint: damping needs all twelve arrays, "
                            "16-byte aligned");
    if (S.n_poles < 0 || S.n_poles > MTB_MAX_POLES)
        return fail(MTB_INVALID_ARG, "3D adjoint: n_poles %d", S.n_poles);
    if (S.pmc_axes & ~7) return fail(MTB_INVALID_ARG, "3D adjoint: pmc_axes %d", S.pmc_axes);
    if (S.nx < 3 || S.ny < 3 || S.nz < 3 || S.zpitch < S.nz || (S.zpitch & 3))
        return fail(MTB_INVALID_ARG, "3D adjoint: bad grid");
    if ((int64_t)S.nx * S.ny * S.zpitch >= (1LL << 31) || S.nx > 65535 || S.ny > 65535 * 8)
        return fail(MTB_UNSUPPORTED, "3D adjoint: grid too large");
    auto bad = [](const void *p) { return !p || (reinterpret_cast<uintptr_t>(p) & 15); };
    for (int c = 0; c < 6; ++c)
        if (bad(bufs->g[c])) return fail(MTB_INVALID_ARG, "3D adjoint: bad g buffer");
    for (int c = 0; c < 12; ++c)
        if (bad(bufs->g_psi[c])) return fail(MTB_INVALID_ARG, "3D adjoint: bad g_psi buffer");
    for (int c = 0; c < 15; ++c)
        if (bad(bufs->tmp[c])) return fail(MTB_INVALID_ARG, "3D adjoint: bad tmp buffer");
    if (bad(bufs->g_eps) || bad(S.eps)) return fail(MTB_INVALID_ARG, "3D adjoint: bad eps");
    if (S.n_poles > 0)
        for (int c = 0; c < 3; ++c)
            if (bad(S.pol_c3[c]) || bad(bufs->g_pol[c][0]) || bad(bufs->g_pol[c][1]))
                return fail(MTB_INVALID_ARG, "3D adjoint: poles need c3 and both g_pol stacks "
                            "per component, 16-byte aligned");
    for (int a = 0; a < 3; ++a)
        for (int h = 0; h < 2; ++h)
            if (!S.prof_b[a][h] || !S.prof_a[a][h])
                return fail(MTB_INVALID_ARG, "3D adjoint: null CPML profile");
    if (S.n_planes < 0 || (S.n_planes > 0 && (!S.planes || !S.plane_ring_off)))
        return fail(MTB_INVALID_ARG, "3D adjoint: bad plane list");
    mtb_yee3d_adjoint *p = new mtb_yee3d_adjoint();
    p->s = S;
    Adj3 &A = p->a;
    A.b = *bufs;
    A.eps = S.eps;
    for (int a = 0; a < 3; ++a)
        for (int h = 0; h < 2; ++h) {
            A.pb[a][h] = S.prof_b[a][h];
            A.pa[a][h] = S.prof_a[a][h];
        }
    for (int c = 0; c < 6; ++c)
        for (int h = 0; h < 2; ++h) A.dmp[c][h] = S.damp[c][h];
    A.np = S.n_poles;
    A.pmc = S.pmc_axes;
    A.psi_all = 1;
    for (int c = 0; c < 3; ++c) A.c3[c] = S.n_poles ? S.pol_c3[c] : nullptr;
    for (int p = 0; p < MTB_MAX_POLES; ++p) {
        A.c1[p] = p < S.n_poles ? S.pol_c1[p] : 0.f;
        A.c2[p] = p < S.n_poles ? S.pol_c2[p] : 0.f;
    }
    A.nx = S.nx; A.ny = S.ny; A.nz = S.nz; A.zp = S.zpitch;
    A.dt = S.dt;
    A.rdx = 1.0f / S.dx;
    int rc = p->dft.init(regions, n_regions, groups, n_groups, ring_slot_elems,
                         ring_slots > 0 ? ring_slots : 32);
    if (!rc) rc = p->s_d.ensure(sizeof(mtb_yee3d_struct));
    if (!rc) rc = p->pstart_d.ensure(sizeof(int64_t) * (S.n_planes + 1));
    if (!rc && n_regions == 0)
        rc = p->dft.ring_d.ensure(sizeof(float) * (size_t)std::max<int64_t>(ring_slot_elems, 4) *
                                  p->dft.slots);
    if (rc) { p->dft.release(); delete p; return rc; }
    std::vector<int64_t> ps(S.n_planes + 1, 0);
    if (S.n_planes > 0) {
        std::vector<int32_t> pl(8 * S.n_planes);
        cudaError_t e = cudaMemcpy(pl.data(), S.planes, sizeof(int32_t) * 8 * S.n_planes,
                                   cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            p->dft.release(); delete p;
            return fail(MTB_CUDA_ERROR, "reading plane list: %s", cudaGetErrorString(e));
        }
        for (int q = 0; q < S.n_planes; ++q)
            ps[q + 1] = ps[q] + (int64_t)(pl[8 * q + 4] - pl[8 * q + 3]) *
                                    (pl[8 * q + 6] - pl[8 * q + 5]);
    }
    p->n_planes = S.n_planes;
    p->n_samples = ps[S.n_planes];
    cudaError_t e = cudaMemcpy(p->s_d.p, &S, sizeof(S), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(p->pstart_d.p, ps.data(), sizeof(int64_t) * ps.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        p->dft.release(); delete p;
        return fail(MTB_CUDA_ERROR, "3D adjoint upload: %s", cudaGetErrorString(e));
    }
    p->marks.ready();
    *out = p;
    return MTB_OK;
}

int mtb_yee3d_adjoint_run(mtb_yee3d_adjoint *p, int64_t t0, int32_t k, const float *rec,
                          int64_t rec_comp_stride, int64_t rec_slot_stride, void *stream) {
    if (!p) return fail(MTB_INVALID_ARG, "3D adjoint plan is null");
    p->last_launches = 0;
    if (k <= 0) return MTB_OK;
    const MarkUse use(p->marks, stream);
    if (k > p->dft.slots) return fail(MTB_INVALID_ARG, "k %d > ring slots %d", k, p->dft.slots);
    if (!rec || (reinterpret_cast<uintptr_t>(rec) & 15) || (rec_comp_stride & 3) ||
        (rec_slot_stride & 3))
        return fail(MTB_INVALID_ARG, "3D adjoint: bad forward record");
    cudaStream_t st = (cudaStream_t)stream;
    int rc;
    if ((rc = p->dft.upload_phases(t0, k, st))) return rc;
    if (p->dft.n_regions > 0) {
        if ((rc = p->dft.expand(0, k, st))) return rc;
        ++p->last_launches;
    } else {
        MTB_CUDA_TRY(cudaMemsetAsync(p->dft.ring_d.p, 0,
                                     sizeof(float) * (size_t)p->dft.slot_elems * k, st));
    }
    const Adj3 &A = p->a;
    const dim3 blk(A3_T, 3);
    const dim3 grid((unsigned)(((int64_t)A.ny * (A.zp / 4) + A3_T - 1) / A3_T), A.nx);
    const int mode = (A.dmp[0][0] ? 1 : 0) | (A.np > 0 ? 2 : 0);
    // The first launch of the chunk is an ordinary one: the chunk's sample adjoints, which the
    // kernels read through the read-only path, are complete behind it.
    bool first = true;
    auto go = [&](auto kernel, dim3 g, dim3 b, auto... args) -> int {
        if (!first) return launch_pdl(kernel, g, b, st, args...);
        first = false;
        kernel<<<g, b, 0, st>>>(args...);
        MTB_CHECK_LAUNCH();
        return MTB_OK;
    };
    auto inject = [&](int q) -> int {
        if (p->n_samples == 0) return MTB_OK;
        const float *radj = p->dft.ring_d.as<float>() + (size_t)q * p->dft.slot_elems;
        ++p->last_launches;
        return go(k_adj3_inject, (unsigned)((p->n_samples + 255) / 256), 256,
                  p->s_d.as<mtb_yee3d_struct>(), p->pstart_d.as<int64_t>(), p->n_planes, radj, A.b);
    };
    if ((rc = inject(k - 1))) return rc;
    for (int q = k - 1; q >= 0; --q) {
        const float *en = rec + (size_t)(q + 1) * rec_slot_stride;
        const float *eo = rec + (size_t)q * rec_slot_stride;
        decltype(&k_adj3_fe<false, 0>) fe[8] = {
            k_adj3_fe<false, 0>, k_adj3_fe<false, 1>, k_adj3_fe<false, 2>, k_adj3_fe<false, 3>,
            k_adj3_fe<true, 0>,  k_adj3_fe<true, 1>,  k_adj3_fe<true, 2>,  k_adj3_fe<true, 3>};
        const bool fin = q < k - 1;
        if ((rc = go(fe[mode + (fin ? 4 : 0)], grid, blk, A, en, eo, rec_comp_stride))) return rc;
        if ((rc = go(k_adj3_h, grid, blk, A))) return rc;
        p->last_launches += 2;
        if (q > 0 && (rc = inject(q - 1))) return rc;    // before the fin + E launch of q - 1
    }
    if ((rc = go(k_adj3_fin, grid, blk, A)) || (rc = go(k_adj3_eps, grid, A3_T, A))) return rc;
    p->last_launches += 2;
    return MTB_OK;
}

int mtb_yee3d_adjoint_psi_layers(mtb_yee3d_adjoint *p, int32_t only_layers) {
    if (!p) return fail(MTB_INVALID_ARG, "3D adjoint plan is null");
    p->a.psi_all = only_layers ? 0 : 1;
    return MTB_OK;
}

int64_t mtb_yee3d_adjoint_last_launches(const mtb_yee3d_adjoint *p) {
    return p ? p->last_launches : -1;
}

void mtb_yee3d_adjoint_destroy(mtb_yee3d_adjoint *p) {
    if (!p) return;
    const ScratchIdle scratch(p->marks.wait());
    p->dft.release();
    p->s_d.release();
    p->pstart_d.release();
    delete p;
}

}  // extern "C"
