// Gradients of recorded membrane potentials with respect to channel
// conductivities and cell axial resistivities (include/eden_gpu.h,
// edenGpuGrad*).  The reference has no gradient path; this file has no
// counterpart there.
//
// The forward step is the one the reference runs per compartment and the
// plain GPU path reproduces: HH gates by exponential Euler with clamp
// (eden/Eden.cpp:5126-5259), channel currents (5805-5898), the V pre-update
// (6057-6107) and the backward-Euler Hines solve (6114-6225).  The gradient
// is the discrete adjoint of that step (reverse mode, exact for the
// arithmetic of the step up to rounding):
//
//   state (V^n, q^n) -> q^{n+1} = Q(V^n, q^n)            (gates, old V)
//                       g_c = gbase_c fopen_c(q^n) 1e-5 A  (channel conductance)
//                       d = G/C + s irc,  x = V + dt (I + V G)/C
//                       M V^{n+1} = x,  M = 1 + dt d on the diagonal,
//                                      s U (row child), s L (row parent)
//   with s = Ra_ref / Ra the cell's axial scale.  Given the adjoints
//   (lV, lq) of (V^{n+1}, q^{n+1}):  mu = M^-T lV (the same elimination with
//   U and L exchanged), x_bar = mu, d_bar = -dt mu V^{n+1};
//   g_bar_c = (d_bar + mu dt E_c) / C; Ra_bar += (1/Ra) mu^T A_ax V^{n+1}
//   (A_ax the axial part of M); V_bar = x_bar + sum lq dQ/dV; q_bar = lq
//   dQ/dq + g_bar gbase 1e-5 A dfopen/dq.  dQ/dq = b and dQ/dV = b'(q - inf)
//   + (1 - b) inf' where the gate did not clamp, 0 where it did.
//
// Synaptic drive with event steps fixed in advance -- timedSynapticInput
// inputs and connection synapses whose presynaptic cell is a spike source
// (spike lists, generators, event-set readers) -- enters each step as
// conductances g_k = sum_s w_s g^_s(n) per group k (one compartment, one
// synapse type, inputs or connections), with g^_s the unit-weight exposure
// of synapse s at step n (expTwo gbase (B - A), expOne G;
// LEMS_CoreComponents.inc.xml:145-180, eden/Eden.cpp:3424-3466): forward
// Euler between events, the event's jump instead of the decay in its step.
// g^_s does not depend on V or on the weights, so a k_grad_drive launch
// tabulates g_k(n) for the run before the forward, and the adjoint gives
// g_bar_k(n) = (d_bar + mu dt E_k) / C like a channel's; a weight's gradient
// is then sum_n g_bar_k(n) g^_s(n) (eden/Eden.cpp:3708-3710 multiplies the
// synapse's current and conductance by its weight), summed per synapse in
// double by k_grad_weights.
//
// Cells are independent, and a run of one is a chain of steps, so what a step
// must do one thing after another decides its time.  The forward kernel gives a
// cell a block: a few warps compute the currents and one of them solves the
// cable, while the others update the gates, which the next step is the first to
// need.  It writes the trace, a checkpoint of (V, q) every S steps and, where
// they fit the trajectory buffer, every step's V, q and pivots; where they do
// not, the backward recomputes as many segments as fit at a time from their
// checkpoints, all at once.  Of the adjoint, only the recurrence
//   mu = M^-T lV,  lV' = mu + sum lq cv,  lq' = lq b + mu kq
// goes back step by step; its coefficients (the factors of M^T from the
// forward's pivots, b, cv = dQ/dV, kq = dt (E - V^{n+1}) / C gbase 1e-5 A
// dfopen/dq) come from a kernel parallel over all steps, and the parameters'
// terms, sums over steps of mu times known factors, from another.  They
// accumulate in double in a fixed order, so gradients are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/eden_gpu.h"
#include "eden_math.cuh"

using namespace eden;

namespace eden_grad {

constexpr int kMaxSlots = 32;  // distinct parameters one cell may use

// A synapse type as the drive needs it: kind, gbase (uS), time constants
// (us) and expTwo's jump weight_prop * waveform_factor.
struct GradSyn {
    int32_t kind;
    float gbase, tau_decay, tau_rise, wf_w;
};

struct GradDev {
    int n_cells = 0, n_rec = 0, S = 100, n_types = 0;
    int64_t N = 0, n_comp = 0, n_gate = 0;
    float dt = 0.0f;
    // per cell: compartments, gates, channels, depth table, parameter slots, recorded columns
    const int32_t *cell_c0, *cell_g0, *cell_ch0, *cell_l0, *cell_s0, *cell_r0;
    const int32_t *cell_ra_slot, *cell_ra_param, *cell_chain;
    const float *cell_ra;
    const int32_t *lev;  // each cell's depth boundaries (local indices), nlev + 1 entries
    // per compartment, breadth-first within the cell
    const float *C, *A, *IRC, *U, *L, *V0;
    const int32_t *P, *CB, *CE, *comp_ch0, *comp_pu0;  // local indices; comp_ch0 local to the cell
    // per channel instance
    const int32_t *ch_type, *ch_g0, *ch_param, *ch_slot;
    const float *ch_gbase, *ch_erev;
    const EdenGpuChannelType *types;
    // pulses
    const float *pu_start, *pu_dur, *pu_aw;
    // recorded compartments (local index) and their trace columns
    const int32_t *rec_local, *rec_col;
    const float *tk;  // [N + 1]: tk[n] = time of step n
    // synaptic drive: groups of each compartment (breadth-first order),
    // each group's reversal potential, kind (0 inputs, 1 connections) and
    // items; each item's synapse type, weight (or parameter) and event steps
    int32_t n_grp = 0;
    int64_t n_item = 0;
    const int32_t *comp_gr0, *gr_kind, *gr_it0, *it_grp, *it_type, *it_param, *it_ev;
    const int64_t *it_ev0;
    const float *gr_erev, *it_w;
    const GradSyn *syn;
    float *it_a, *it_b;      // unit-weight synapse state while tabulating
    int64_t *it_cur;         // its next event
    float *ex;               // [ex_rows][n_item] unit-weight exposures of some steps
    float *gtab;             // [N + 1][n_grp] group conductance at step n (weights applied)
    float *gbar;             // [N + 1][n_grp] its adjoint
    double *item_grad;       // [n_item] d loss / d weight
    const float *params;
    float *ck_v, *ck_q;  // checkpoints [n_ck][n_comp], [n_ck][n_gate]
    // trajectory of the steps from tr_n0 on: V and q at their starts (and after
    // the last), and the reciprocal pivots of their solves
    float *tr_v, *tr_q, *tr_d;
    int64_t tr_n0 = 1;
    // adjoint coefficients of the steps from co_n0 on: a row of co_len floats a
    // step, a cell's [factor up, factor down, reciprocal pivot][nc], [b, cv, kq][ng]
    // from cell_k0; mu, the solved adjoints of the same steps; the adjoints of
    // the state between launches
    const int32_t *cell_k0, *comp_cell, *gate_map, *comp_g0, *comp_rc0;
    int32_t co_len = 0;
    float *co, *mu;
    int64_t co_n0 = 1;
    float *lv, *lq;
    double *part;        // [slots][chunks of kSumSteps steps]
    int32_t n_part = 0;
    float *trace;        // [N][n_rec]
    const float *trace_grad;
    double *slot_grad;   // per cell and slot
};

constexpr int kSumSteps = 32;  // steps whose parameter terms one block sums
constexpr int kRing = 4;       // steps of coefficients in flight
constexpr int kFwdWarps = 16;  // most warps of a forward block
constexpr int kBlock = 4;      // nodes of a chain loaded at a time, and the padding of its arrays

// Largest cell, for the shared-memory layout.
struct Dims {
    int slots, c, g, ch;
};

// A block's shared memory in the forward kernel: the channel types, the cell's
// state and solve arrays, and its constants staged once per launch (axial
// terms already scaled by the cell's resistivity parameter).
struct Cell {
    // the solve's pairs, kBlock before and after the cell's: pre-updated V and
    // 1 + dt d, by the solve the eliminated V and the reciprocal pivot; U and L
    float2 *XD, *UL;
    EdenGpuChannelType *types;
    float *Va, *Vb, *qa, *qb;  // V (kBlock after) and q: two buffers each, by turns
    float *Cc, *Ac, *IRCs;
    int32_t *P, *CB, *CE, *ch0;
    int32_t *ctype, *cg0;
    const int32_t *gmap;  // per gate: compartment | (channel type << 2 | gate of it) << 16
    float *cgb, *cerev;
    int c0, g0, nc, ng, nch, nlev;
    const int32_t *lev;
    bool serial;  // solve by one lane (cells with few compartments per depth)
    bool chain;   // an unbranched cable: node j's only child is j + 1
};

// A cell's axial scale Ra_ref / Ra.
__device__ __forceinline__ float axial_scale(const GradDev &m, int cell) {
    const int rp = m.cell_ra_param[cell];
    return rp >= 0 ? m.cell_ra[cell] / m.params[rp] : 1.0f;
}

// NEAR: the gates' map is staged too (a cell that has no room for it reads it
// where it is).
template <bool NEAR>
__device__ __forceinline__ Cell stage_cell(const GradDev &m, int cell, const Dims &dm) {
    extern __shared__ __align__(16) double smem_d[];
    const int tid = threadIdx.x, nt = blockDim.x;
    Cell c;
    c.XD = reinterpret_cast<float2 *>(smem_d) + kBlock;
    c.UL = c.XD + dm.c + 2 * kBlock;
    c.types = reinterpret_cast<EdenGpuChannelType *>(c.UL + dm.c + kBlock);
    float *f = reinterpret_cast<float *>(c.types + m.n_types);
    c.Va = f; f += dm.c + kBlock;
    c.Vb = f; f += dm.c + kBlock;
    c.Cc = f; f += dm.c;
    c.Ac = f; f += dm.c;
    c.IRCs = f; f += dm.c;
    c.qa = f; f += dm.g;
    c.qb = f; f += dm.g;
    c.cgb = f; f += dm.ch;
    c.cerev = f; f += dm.ch;
    int32_t *i = reinterpret_cast<int32_t *>(f);
    c.P = i; i += dm.c;
    c.CB = i; i += dm.c;
    c.CE = i; i += dm.c;
    c.ch0 = i; i += dm.c + 1;
    c.ctype = i; i += dm.ch;
    c.cg0 = i; i += dm.ch;
    int32_t *gmap = i;
    c.c0 = m.cell_c0[cell];
    c.nc = m.cell_c0[cell + 1] - c.c0;
    c.g0 = m.cell_g0[cell];
    c.ng = m.cell_g0[cell + 1] - c.g0;
    const int h0 = m.cell_ch0[cell];
    c.nch = m.cell_ch0[cell + 1] - h0;
    c.lev = m.lev + m.cell_l0[cell];
    c.nlev = m.cell_l0[cell + 1] - m.cell_l0[cell] - 1;
    c.serial = c.nc <= 6 * c.nlev;
    c.chain = m.cell_chain[cell] != 0;
    const float s = axial_scale(m, cell);
    const int words = (int)(sizeof(EdenGpuChannelType) / 4) * m.n_types;
    for (int k = tid; k < words; k += nt)
        reinterpret_cast<int32_t *>(c.types)[k] = reinterpret_cast<const int32_t *>(m.types)[k];
    for (int j = tid; j < c.nc; j += nt) {
        const int gc = c.c0 + j;
        c.UL[j] = make_float2(m.U[gc] * s, m.L[gc] * s);
        c.IRCs[j] = m.IRC[gc] * s;
        c.Cc[j] = m.C[gc];
        c.Ac[j] = m.A[gc];
        c.P[j] = m.P[gc];
        c.CB[j] = m.CB[gc];
        c.CE[j] = m.CE[gc];
        c.ch0[j] = m.comp_ch0[gc];
    }
    // (what the padding holds is computed with, and not used)
    if (tid < kBlock) {
        c.XD[-1 - tid] = c.XD[c.nc + tid] = make_float2(0.0f, 1.0f);
        c.UL[-1 - tid] = c.UL[c.nc + tid] = make_float2(0.0f, 0.0f);
    }
    if (tid == 0) c.ch0[c.nc] = c.nch;
    for (int k = tid; k < c.nch; k += nt) {
        const int ch = h0 + k;
        const int p = m.ch_param[ch];
        c.ctype[k] = m.ch_type[ch];
        c.cg0[k] = m.ch_g0[ch];
        c.cgb[k] = p >= 0 ? m.params[p] : m.ch_gbase[ch];
        c.cerev[k] = m.ch_erev[ch];
    }
    c.gmap = NEAR ? gmap : m.gate_map + c.g0;
    if (NEAR)
        for (int k = tid; k < c.ng; k += nt) gmap[k] = m.gate_map[c.g0 + k];
    __syncthreads();
    return c;
}

// d(rate)/dV of the HH rate forms of rate_value, from the mathematics of
// each form: EXP r e^x -> val / s; SIGMOID r / (1 + e^-x) -> val (e^-x / (1 +
// e^-x)) / s; EXPLINEAR r f(x), f = x / (1 - e^-x) -> r f'(x) / s with
// f'(x) = (1 - e^-x (1 + x)) / (1 - e^-x)^2, by its Taylor series
// 1/2 + x/6 - x^3/180 near x = 0 (where the closed form cancels).
__device__ __forceinline__ float rate_slope(int kind, float r, float mid, float s, float v, float val) {
    const float x = (v - mid) / s;
    if (kind == EDEN_RATE_EXP) return val / s;
    if (kind == EDEN_RATE_SIGMOID) {
        const float e = expf(-x);
        return val * (1.0f / (1.0f + 1.0f / e)) / s;
    }
    float fp;
    if (fabsf(x) < 1e-2f) {
        fp = 0.5f + x * (1.0f / 6.0f) - x * x * x * (1.0f / 180.0f);
    } else if (x < -60.0f) {
        fp = 0.0f;
    } else {
        const float em = expm1f(-x);  // e^-x - 1
        fp = (-em - x * (1.0f + em)) / (em * em);
    }
    return r * fp / s;
}

// A gate's next value (gate_relax, as the plain path's target_step).
__device__ __forceinline__ float gate_step(const GradDev &m, const Cell &c, int k, float v, float qo, bool init) {
    const EdenGpuChannelType &ct = c.types[(uint32_t)c.gmap[k] >> 18];
    const int g = (c.gmap[k] >> 16) & 3;
    const float al = rate_value(ct.fwd_kind[g], ct.fwd_rate[g], ct.fwd_mid[g], ct.fwd_scale[g], v);
    const float be = rate_value(ct.rev_kind[g], ct.rev_rate[g], ct.rev_mid[g], ct.rev_scale[g], v);
    return gate_relax(al, be, ct.q10[g], init, m.dt, qo);
}

// Channel currents and V pre-update of compartment j at time t, from the gates
// at the step's start: the pre-updated V (x) and the diagonal term d, with the
// plain path's operations (target_step).
struct CompInputs {  // of a compartment: its pulses, its synaptic groups, RN(1 / C) for div_known
    int pu0, pu1, gr0, gr1;
    float rC;
};
__device__ __forceinline__ CompInputs comp_inputs(const GradDev &m, const Cell &c, int j) {
    const int gc = c.c0 + j;
    return {m.comp_pu0[gc], m.comp_pu0[gc + 1], m.comp_gr0[gc], m.comp_gr0[gc + 1], known_reciprocal(c.Cc[j])};
}
__device__ __forceinline__ void comp_pre(const GradDev &m, const Cell &c, const float *q, int j, const CompInputs &ci,
                                         int64_t n, float t, float v, float &x, float &d) {
    const float A = c.Ac[j];
    float Ich = 0.0f, Gch = 0.0f;
    for (int k = c.ch0[j]; k < c.ch0[j + 1]; k++) {
        const EdenGpuChannelType &ct = c.types[c.ctype[k]];
        const float *qq = q + c.cg0[k];
        float fopen = 1.0f;
        for (int g = 0; g < ct.n_gates; g++) {
            const float qo = qq[g];
            for (int r = 0; r < ct.gate_instances[g]; r++) fopen = fopen * qo;
        }
        const float gs = c.cgb[k] * fopen;
        Ich += (gs * (c.cerev[k] - v) * 1e-5f) * A;
        Gch += (gs * 1e-5f) * A;
    }
    float Iin = 0.0f;
    for (int k = ci.pu0; k < ci.pu1; k++) {
        const float st = m.pu_start[k], du = m.pu_dur[k];
        Iin += (st <= t && t <= st + du) ? m.pu_aw[k] : 0.0f;
    }
    // synaptic drive: inputs, then connections (eden/Eden.cpp:6057-6060)
    float Gin = 0.0f, Isyn = 0.0f, Gsyn = 0.0f;
    for (int k = ci.gr0; k < ci.gr1; k++) {
        const float g = m.gtab[n * m.n_grp + k];
        if (m.gr_kind[k] == 0) {
            Iin += g * (m.gr_erev[k] - v);
            Gin += g;
        } else {
            Isyn += g * (m.gr_erev[k] - v);
            Gsyn += g;
        }
    }
    const float I = Ich + Iin + Isyn;
    const float G = Gch + Gin + Gsyn;
    const float C = c.Cc[j];
    d = 1.0f * div_known(G, C, ci.rC) + c.IRCs[j];
    x = v + div_known(m.dt * (I + (v * G)), C, ci.rC);
}

// Backward-Euler Hines solve of the cell (eden/Eden.cpp:6114-6225) by one warp,
// from XD, which keeps the eliminated V and the reciprocal pivots, into VN;
// every node pulls its children in order, deepest first, then back-substitution
// runs root first.  Cells with few compartments per depth (chains,
// ball-and-stick) are solved by one lane in reverse breadth-first order with the
// last node's values in registers; the others depth by depth across the warp.
// Both do the same operations.
__device__ __forceinline__ void hines_cell(const Cell &c, float *VN) {
    const int lane = threadIdx.x & 31;
    float2 *XD = c.XD;
    const float2 *UL = c.UL;
    if (c.chain) {
        // the next nodes are loaded before these are stored: left to itself the
        // compiler keeps a load behind a store that might be to the same place.
        // The last block runs into the padding.
        if (lane == 0) {
            const int n = c.nc;
            float rc = pivot(XD[n - 1].y), xc = XD[n - 1].x;
            XD[n - 1].y = rc;
            float2 xd[kBlock], ul[kBlock];
#pragma unroll
            for (int k = 0; k < kBlock; k++) { xd[k] = XD[n - 2 - k]; ul[k] = UL[n - 1 - k]; }
            for (int j = n - 2; j >= 0; j -= kBlock) {
                float2 out[kBlock];
#pragma unroll
                for (int k = 0; k < kBlock; k++) {
                    const float ratio = ul[k].y * rc;
                    rc = pivot(fmaf(-ratio, ul[k].x, xd[k].y));
                    xc = fmaf(-ratio, xc, xd[k].x);
                    out[k] = make_float2(xc, rc);
                }
                if (j >= kBlock)
#pragma unroll
                    for (int k = 0; k < kBlock; k++) { xd[k] = XD[j - kBlock - k]; ul[k] = UL[j + 1 - kBlock - k]; }
#pragma unroll
                for (int k = 0; k < kBlock; k++) XD[j - k] = out[k];
            }
            float xp = XD[0].x * XD[0].y;
            VN[0] = xp;
#pragma unroll
            for (int k = 0; k < kBlock; k++) { xd[k] = XD[1 + k]; ul[k] = UL[1 + k]; }
            for (int j = 1; j < n; j += kBlock) {
                float out[kBlock];
#pragma unroll
                for (int k = 0; k < kBlock; k++) {
                    xp = fmaf(-ul[k].x, xp, xd[k].x) * xd[k].y;
                    out[k] = xp;
                }
                if (j + kBlock < n)
#pragma unroll
                    for (int k = 0; k < kBlock; k++) { xd[k] = XD[j + kBlock + k]; ul[k] = UL[j + kBlock + k]; }
#pragma unroll
                for (int k = 0; k < kBlock; k++) VN[j + k] = out[k];
            }
        }
        __syncwarp();
        return;
    }
    if (c.serial) {
        if (lane == 0) {
            float xc = 0.0f, rc = 0.0f;
            int last = -1;
            for (int j = c.nc - 1; j >= 0; j--) {
                const int kb = c.CB[j], ke = c.CE[j];
                float2 v = XD[j];
                for (int i = kb; i < ke; i++) {
                    const float2 k = i == last ? make_float2(xc, rc) : XD[i];
                    const float ratio = UL[i].y * k.y;
                    v.y = fmaf(-ratio, UL[i].x, v.y);
                    v.x = fmaf(-ratio, k.x, v.x);
                }
                rc = pivot(v.y);
                xc = v.x;
                XD[j] = make_float2(xc, rc);
                last = j;
            }
            float xp = XD[0].x * XD[0].y;
            VN[0] = xp;
            for (int j = 1; j < c.nc; j++) {
                const int p = c.P[j];
                xp = fmaf(-UL[j].x, p == j - 1 ? xp : VN[p], XD[j].x) * XD[j].y;
                VN[j] = xp;
            }
        }
        __syncwarp();
        return;
    }
    for (int l = c.nlev - 1; l >= 0; l--) {
        for (int j = c.lev[l] + lane; j < c.lev[l + 1]; j += 32) {
            float2 v = XD[j];
            for (int i = c.CB[j]; i < c.CE[j]; i++) {
                const float2 k = XD[i];
                const float ratio = UL[i].y * k.y;
                v.y = fmaf(-ratio, UL[i].x, v.y);
                v.x = fmaf(-ratio, k.x, v.x);
            }
            XD[j] = make_float2(v.x, pivot(v.y));
        }
        __syncwarp();
    }
    for (int r = c.lev[0] + lane; r < c.lev[1]; r += 32) VN[r] = XD[r].x * XD[r].y;
    __syncwarp();
    for (int l = 1; l < c.nlev; l++) {
        for (int i = c.lev[l] + lane; i < c.lev[l + 1]; i += 32) VN[i] = fmaf(-UL[i].x, VN[c.P[i]], XD[i].x) * XD[i].y;
        __syncwarp();
    }
}

// The run of a cell (block x) over steps [1, N], or, recomputing, over segment
// seg0 + block y from its checkpoint.  The first `cw` warps compute the currents
// and the first of them solves the cable; the others update the gates in the
// meantime, into the other of two buffers, and write the step's records.  A
// step is the currents and the solve one after the other: on a cable of 51
// compartments 2,700 cycles of the solve's chain (a product, a fused one and a
// reciprocal a compartment) and about 500 of the rest, where one warp a cell,
// taking its 153 gates in turns before the solve, took 16,000.
template <bool RECOMPUTE, bool NEAR>
__global__ void __launch_bounds__(32 * kFwdWarps) k_grad_forward(GradDev m, Dims dm, int cw, int64_t seg0, int keep) {
    const int cell = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Cell c = stage_cell<NEAR>(m, cell, dm);
    const int64_t seg = RECOMPUTE ? seg0 + blockIdx.y : 0;
    const int64_t first = 1 + seg * m.S, end = RECOMPUTE && first + m.S < m.N ? first + m.S : m.N;
    float *V = c.Va, *Vn = c.Vb, *q = c.qa, *qn = c.qb;  // at the step's start, and the next's
    if (RECOMPUTE) {
        for (int j = tid; j < c.nc; j += blockDim.x) V[j] = m.ck_v[seg * m.n_comp + c.c0 + j];
        for (int k = tid; k < c.ng; k += blockDim.x) q[k] = m.ck_q[seg * m.n_gate + c.g0 + k];
    } else {
        // the four initialisation passes leave V and set every gate to inf(V)
        for (int j = tid; j < c.nc; j += blockDim.x) V[j] = m.V0[c.c0 + j];
        __syncthreads();
        for (int k = tid; k < c.ng; k += blockDim.x) q[k] = gate_step(m, c, k, V[c.gmap[k] & 0xffff], 0.0f, true);
    }
    const int r0 = m.cell_r0[cell], r1 = m.cell_r0[cell + 1];
    // threads of the gates' share (all of them where there is one share)
    const int gw = (int)(blockDim.x >> 5) - cw, gt = gw > 0 ? tid - 32 * cw : tid, gn = gw > 0 ? 32 * gw : (int)blockDim.x;
    int64_t ck = 0;
    int to_ck = 0;  // steps until the next checkpoint
    __syncthreads();
    // a thread's only compartment, where it has no more, and the next step's
    // time: loaded ahead of the steps (600 steps of 256 cells of 51
    // compartments: 1.86 ms with both in the step and C divided by, 1.81 so)
    CompInputs ci{};
    if (warp < cw && tid < c.nc) ci = comp_inputs(m, c, tid);
    float t = m.tk[first];
    for (int64_t n = first; n <= end; n++) {
        if (gt >= 0) {
            if (!RECOMPUTE && to_ck == 0 && n < m.N) {
                for (int j = gt; j < c.nc; j += gn) m.ck_v[ck * m.n_comp + c.c0 + j] = V[j];
                for (int k = gt; k < c.ng; k += gn) m.ck_q[ck * m.n_gate + c.g0 + k] = q[k];
            }
            // (a segment's last state is the next one's first, which writes it)
            if (RECOMPUTE ? n < end || blockIdx.y + 1 == gridDim.y : keep) {
                const int64_t row = n - m.tr_n0;
                for (int j = gt; j < c.nc; j += gn) m.tr_v[row * m.n_comp + c.c0 + j] = V[j];
                for (int k = gt; k < c.ng; k += gn) m.tr_q[row * m.n_gate + c.g0 + k] = q[k];
            }
            if (!RECOMPUTE)
                for (int r = r0 + gt; r < r1; r += gn) m.trace[(n - 1) * m.n_rec + m.rec_col[r]] = V[m.rec_local[r]];
        }
        if (to_ck == 0) {
            ck++;
            to_ck = m.S;
        }
        to_ck--;
        if (n == end) break;
        if (warp < cw) {
            const float t_next = m.tk[n + 1];
            for (int j = tid; j < c.nc; j += 32 * cw) {
                float x, d;
                if (c.nc > 32 * cw) ci = comp_inputs(m, c, j);
                comp_pre(m, c, q, j, ci, n, t, V[j], x, d);
                c.XD[j] = make_float2(x, fmaf(d, m.dt, 1.0f));
            }
            t = t_next;
            // (the warps of the currents only: named barrier 1)
            if (cw > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * cw) : "memory");
            else __syncwarp();
            if (warp == 0) {
                hines_cell(c, Vn);
                if (RECOMPUTE || keep)
                    for (int j = lane; j < c.nc; j += 32) m.tr_d[(n - m.tr_n0) * m.n_comp + c.c0 + j] = c.XD[j].y;
            }
        }
        if (gt >= 0)
            for (int k = gt; k < c.ng; k += gn) qn[k] = gate_step(m, c, k, V[c.gmap[k] & 0xffff], q[k], false);
        __syncthreads();
        float *x = V;
        V = Vn;
        Vn = x;
        x = q;
        q = qn;
        qn = x;
    }
}

// The adjoint's coefficients of `rows` steps from co_n0 on, a thread per step and
// compartment.  dQ/dq = b and dQ/dV = cv where the gate did not clamp, 0 where
// it did; d fopen / dq_g = inst q_g^(inst-1) * prod over the other gates.
__global__ void __launch_bounds__(128) k_grad_coef(GradDev m, int64_t rows) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= rows * m.n_comp) return;
    const int64_t row = id / m.n_comp;
    const int gc = (int)(id - row * m.n_comp);
    const int64_t tr = m.co_n0 + row - m.tr_n0;
    const int cell = m.comp_cell[gc], c0 = m.cell_c0[cell], nc = m.cell_c0[cell + 1] - c0, j = gc - c0;
    const int g0 = m.cell_g0[cell], ng = m.cell_g0[cell + 1] - g0;
    float *co = m.co + row * m.co_len + m.cell_k0[cell];
    const float dt = m.dt, s = axial_scale(m, cell);
    const float rc = m.tr_d[tr * m.n_comp + gc];
    co[j] = (m.U[gc] * s) * rc;
    co[nc + j] = (m.L[gc] * s) * rc;
    co[2 * nc + j] = rc;
    co += 3 * nc;
    const float v = m.tr_v[tr * m.n_comp + gc], vn = m.tr_v[(tr + 1) * m.n_comp + gc];
    const float *q = m.tr_q + tr * m.n_gate + g0;
    const float C = m.C[gc], A = m.A[gc];
    const int h0 = m.cell_ch0[cell], hend = j + 1 < nc ? h0 + m.comp_ch0[gc + 1] : m.cell_ch0[cell + 1];
    for (int h = h0 + m.comp_ch0[gc]; h < hend; h++) {
        const EdenGpuChannelType &ct = m.types[m.ch_type[h]];
        const int q0 = m.ch_g0[h], p = m.ch_param[h];
        float qo[EDEN_MAX_GATES], pw[EDEN_MAX_GATES];
#pragma unroll
        for (int g = 0; g < EDEN_MAX_GATES; g++) {
            qo[g] = 1.0f;
            pw[g] = 1.0f;
            if (g < ct.n_gates) {
                qo[g] = q[q0 + g];
                float x = 1.0f;
                for (int r = 0; r < ct.gate_instances[g]; r++) x = x * qo[g];
                pw[g] = x;
            }
        }
        // d(loss)/d(conductance) is mu times this
        const float gb = p >= 0 ? m.params[p] : m.ch_gbase[h];
        const float fb = ((-dt * vn + dt * m.ch_erev[h]) / C) * gb * 1e-5f * A;
#pragma unroll
        for (int g = 0; g < EDEN_MAX_GATES; g++) {
            if (g >= ct.n_gates) break;
            const int inst = ct.gate_instances[g];
            float dfdq = 0.0f;
            if (inst > 0) {
                dfdq = (float)inst;
                for (int r = 1; r < inst; r++) dfdq = dfdq * qo[g];
#pragma unroll
                for (int h2 = 0; h2 < EDEN_MAX_GATES; h2++)
                    if (h2 != g) dfdq = dfdq * pw[h2];
            }
            const float al = rate_value(ct.fwd_kind[g], ct.fwd_rate[g], ct.fwd_mid[g], ct.fwd_scale[g], v);
            const float be = rate_value(ct.rev_kind[g], ct.rev_rate[g], ct.rev_mid[g], ct.rev_scale[g], v);
            const float sum = al + be;
            const float tau = 1.0f / sum;
            const float inf = al / sum;
            const float b = expf(-((dt * ct.q10[g]) / tau));
            const float qn = b * qo[g] + (1.0f - b) * inf;
            const bool clamped = !(qn > 1e-6f) || !(qn < (float)(1 - 1e-6));
            float cv = 0.0f;
            if (!clamped) {
                const float dal = rate_slope(ct.fwd_kind[g], ct.fwd_rate[g], ct.fwd_mid[g], ct.fwd_scale[g], v, al);
                const float dbe = rate_slope(ct.rev_kind[g], ct.rev_rate[g], ct.rev_mid[g], ct.rev_scale[g], v, be);
                const float db = -(dt * ct.q10[g]) * (dal + dbe) * b;
                const float dinf = (dal * be - al * dbe) / (sum * sum);
                cv = db * (qo[g] - inf) + (1.0f - b) * dinf;
            }
            co[q0 + g] = clamped ? 0.0f : b;
            co[ng + q0 + g] = cv;
            co[2 * ng + q0 + g] = fb * dfdq;
        }
    }
}

// M^T y = X for the staged cell, from the factors of M^T: y up, F = U / pivot of
// the child, down, A = L / pivot of the node, D the reciprocal pivots.  X is
// replaced by the solution.
__device__ __forceinline__ void adjoint_solve(float *X, const float *F, const float *A, const float *D, int nc, bool chain,
                                              bool serial, const int32_t *P, const int32_t *CB, const int32_t *CE,
                                              const int32_t *lev, int nlev) {
    const int lane = threadIdx.x & 31;
    if (chain) {
        // both sweeps are first-order recurrences: each lane composes its own
        // consecutive nodes' maps, a scan over the lanes composes those, and
        // the lane runs its nodes from what the scan gives (51 nodes: about 200
        // cycles a sweep, where a node after the other takes twice that, and
        // longer cables more)
        const int L = (nc + 31) / 32, ja = lane * L < nc ? lane * L : nc, jb = ja + L < nc ? ja + L : nc;
        // up: x_j = X_j - F_{j+1} x_{j+1}; the lane's map of the x below it
        float a = 1.0f, b = 0.0f;
        for (int j = jb - 1; j >= ja; j--) {
            const float f = j + 1 < nc ? -F[j + 1] : 0.0f;
            b = X[j] + f * b;
            a = f * a;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float a2 = __shfl_down_sync(0xffffffffu, a, o), b2 = __shfl_down_sync(0xffffffffu, b, o);
            if (lane + o < 32) {
                b += a * b2;
                a *= a2;
            }
        }
        float x = __shfl_down_sync(0xffffffffu, b, 1);
        if (lane == 31) x = 0.0f;
        for (int j = jb - 1; j >= ja; j--) {
            x = X[j] - (j + 1 < nc ? F[j + 1] : 0.0f) * x;
            X[j] = x * D[j];
        }
        // down: v_j = X_j D_j - A_j v_{j-1}
        a = 1.0f;
        b = 0.0f;
        for (int j = ja; j < jb; j++) {
            const float f = j > 0 ? -A[j] : 0.0f;
            b = X[j] + f * b;
            a = f * a;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float a2 = __shfl_up_sync(0xffffffffu, a, o), b2 = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                b += a * b2;
                a *= a2;
            }
        }
        x = __shfl_up_sync(0xffffffffu, b, 1);
        if (lane == 0) x = 0.0f;
        for (int j = ja; j < jb; j++) {
            x = X[j] - (j > 0 ? A[j] : 0.0f) * x;
            X[j] = x;
        }
        __syncwarp();
        return;
    }
    if (serial) {
        if (lane == 0) {
            for (int j = nc - 1; j >= 0; j--) {
                float x = X[j];
                for (int i = CB[j]; i < CE[j]; i++) x -= F[i] * X[i];
                X[j] = x;
            }
            X[0] = X[0] * D[0];
            for (int j = 1; j < nc; j++) X[j] = X[j] * D[j] - A[j] * X[P[j]];
        }
        __syncwarp();
        return;
    }
    for (int l = nlev - 1; l >= 0; l--) {
        for (int j = lev[l] + lane; j < lev[l + 1]; j += 32) {
            float x = X[j];
            for (int i = CB[j]; i < CE[j]; i++) x -= F[i] * X[i];
            X[j] = x;
        }
        __syncwarp();
    }
    for (int r = lev[0] + lane; r < lev[1]; r += 32) X[r] = X[r] * D[r];
    __syncwarp();
    for (int l = 1; l < nlev; l++) {
        for (int i = lev[l] + lane; i < lev[l + 1]; i += 32) X[i] = X[i] * D[i] - A[i] * X[P[i]];
        __syncwarp();
    }
}

__device__ __forceinline__ void copy16(float *smem_dst, const float *gmem_src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src)
                 : "memory");
}
__device__ __forceinline__ void copy4(float *smem_dst, const float *gmem_src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(gmem_src)
                 : "memory");
}

// The adjoint recurrence of a cell (a block) back over the steps [n0, n0 + rows)
// whose coefficients are there; lv and lq hold the adjoints of the state after
// them and receive those of the state before.  The first warp solves; the others
// fetch a row of coefficients, `ring` - 1 steps ahead of its use, in the
// meantime; then every thread takes its compartments and their gates.  Without
// STAGED (a cell of which not one row fits shared memory; `ring` 0) the rows are read
// where they are.
template <bool STAGED>
__global__ void __launch_bounds__(256) k_grad_adjoint(GradDev m, Dims dm, int64_t rows, int ring, int stage, int last) {
    extern __shared__ __align__(16) double smem_d[];
    const int cell = blockIdx.x, tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5;
    const int c0 = m.cell_c0[cell], nc = m.cell_c0[cell + 1] - c0, g0 = m.cell_g0[cell], ng = m.cell_g0[cell + 1] - g0;
    const int r0 = m.cell_r0[cell], nr = m.cell_r0[cell + 1] - r0;
    const int len = (3 * (nc + ng) + 3) & ~3;
    float *f = reinterpret_cast<float *>(smem_d);
    float *R = f; f += (size_t)ring * stage;  // a stage: the row, then the step's trace gradients
    float *X = f; f += dm.c;
    float *LQ = f; f += dm.g;
    int32_t *i32 = reinterpret_cast<int32_t *>(f);
    int32_t *P = i32; i32 += dm.c;
    int32_t *CB = i32; i32 += dm.c;
    int32_t *CE = i32; i32 += dm.c;
    int32_t *G0 = i32; i32 += dm.c + 1;
    int32_t *RC = i32;
    for (int j = tid; j < nc; j += nt) {
        P[j] = m.P[c0 + j]; CB[j] = m.CB[c0 + j]; CE[j] = m.CE[c0 + j];
        G0[j] = m.comp_g0[c0 + j]; RC[j] = m.comp_rc0[c0 + j] - r0;
        X[j] = m.lv[c0 + j];
    }
    if (tid == 0) { G0[nc] = ng; RC[nc] = nr; }
    for (int k = tid; k < ng; k += nt) LQ[k] = m.lq[g0 + k];
    const int32_t *lev = m.lev + m.cell_l0[cell];
    const int nlev = m.cell_l0[cell + 1] - m.cell_l0[cell] - 1;
    const bool chain = m.cell_chain[cell] != 0, serial = nc <= 6 * nlev;
    auto fetch = [&](int64_t row) {  // by the threads of all warps but the first
        if (row >= 0) {
            float *dst = R + (row % ring) * stage;
            const float *src = m.co + row * m.co_len + m.cell_k0[cell];
            for (int k = 4 * (tid - 32); k < len; k += 4 * (nt - 32)) copy16(dst + k, src + k);
            const float *tg = m.trace_grad + (m.co_n0 + row - 1) * m.n_rec;
            for (int r = tid - 32; r < nr; r += nt - 32) copy4(dst + len + r, tg + m.rec_col[r0 + r]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();
    // the trace gradient of the last state, which no step follows
    if (last)
        for (int j = tid; j < nc; j += nt)
            for (int r = RC[j]; r < RC[j + 1]; r++) X[j] += m.trace_grad[(m.N - 1) * m.n_rec + m.rec_col[r0 + r]];
    if (STAGED && warp > 0) {
        fetch(rows - 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        for (int k = 1; k < ring - 1; k++) fetch(rows - 1 - k);
    }
    for (int64_t row = rows - 1; row >= 0; row--) {
        __syncthreads();
        const float *co = STAGED ? R + (row % ring) * stage : m.co + row * m.co_len + m.cell_k0[cell];
        if (warp == 0) {
            adjoint_solve(X, co, co + nc, co + 2 * nc, nc, chain, serial, P, CB, CE, lev, nlev);
        } else if (STAGED && ring > 1) {
            // into the stage of the row before this one's in time, which is done
            // with; then the next row is there
            fetch(row - (ring - 1));
            if (ring == kRing) asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const float *gb = co + 3 * nc, *tg = co + len;
        for (int j = tid; j < nc; j += nt) {
            const float mu = X[j];
            m.mu[row * m.n_comp + c0 + j] = mu;
            float x = mu;
            for (int k = G0[j]; k < G0[j + 1]; k++) {
                const float lq = LQ[k];
                x += lq * gb[ng + k];
                LQ[k] = lq * gb[k] + mu * gb[2 * ng + k];
            }
            for (int r = RC[j]; r < RC[j + 1]; r++)
                x += STAGED ? tg[r] : m.trace_grad[(m.co_n0 + row - 1) * m.n_rec + m.rec_col[r0 + r]];
            X[j] = x;
        }
        if (STAGED && ring == 1) {  // (one row at a time)
            __syncthreads();
            if (warp > 0) {
                fetch(row - 1);
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
        }
    }
    __syncthreads();
    for (int j = tid; j < nc; j += nt) m.lv[c0 + j] = X[j];
    for (int k = tid; k < ng; k += nt) m.lq[g0 + k] = LQ[k];
}

// The parameters' terms of kSumSteps steps of a cell (block x: the cell, y: the
// steps), from mu and the trajectory, in double per thread and slot, then over
// the threads in order; and the drive groups' conductance adjoints.
__global__ void __launch_bounds__(64) k_grad_terms(GradDev m, int64_t rows) {
    extern __shared__ __align__(16) double smem_d[];
    const int cell = blockIdx.x, tid = threadIdx.x;
    const int s0 = m.cell_s0[cell], ns = m.cell_s0[cell + 1] - s0;
    const int c0 = m.cell_c0[cell], nc = m.cell_c0[cell + 1] - c0, h0 = m.cell_ch0[cell], g0 = m.cell_g0[cell];
    double *acc = smem_d + tid;
    for (int k = 0; k < ns; k++) acc[64 * k] = 0.0;
    const int64_t a = (int64_t)blockIdx.y * kSumSteps, b = a + kSumSteps < rows ? a + kSumSteps : rows;
    const float dt = m.dt, s = axial_scale(m, cell);
    const int ra = m.cell_ra_slot[cell];
    for (int j = tid; j < nc; j += 64) {
        const int gc = c0 + j;
        const float C = m.C[gc], A = m.A[gc], Us = m.U[gc] * s, Ls = m.L[gc] * s, irc = m.IRC[gc] * s;
        const int p = m.P[gc], k0 = m.comp_gr0[gc], k1 = m.comp_gr0[gc + 1];
        const int ha = h0 + m.comp_ch0[gc], hb = j + 1 < nc ? h0 + m.comp_ch0[gc + 1] : m.cell_ch0[cell + 1];
        for (int64_t row = a; row < b; row++) {
            const int64_t n = m.co_n0 + row, tr = n - m.tr_n0;
            const float mu = m.mu[row * m.n_comp + gc], vn = m.tr_v[(tr + 1) * m.n_comp + gc];
            const float dbar = -dt * mu * vn;
            if (ra >= 0) {
                double r = (double)mu * (double)(dt * irc) * vn;
                if (p >= 0)
                    r += (double)mu * (double)Us * m.tr_v[(tr + 1) * m.n_comp + c0 + p] +
                         (double)m.mu[row * m.n_comp + c0 + p] * (double)Ls * vn;
                acc[64 * ra] += r;
            }
            for (int k = k0; k < k1; k++) m.gbar[n * m.n_grp + k] = (dbar + mu * dt * m.gr_erev[k]) / C;
            for (int h = ha; h < hb; h++) {
                const int slot = m.ch_slot[h];
                if (slot < 0) continue;
                const EdenGpuChannelType &ct = m.types[m.ch_type[h]];
                const float *q = m.tr_q + tr * m.n_gate + g0 + m.ch_g0[h];
                float fopen = 1.0f;
                for (int g = 0; g < ct.n_gates; g++) {
                    float x = 1.0f;
                    for (int r = 0; r < ct.gate_instances[g]; r++) x = x * q[g];
                    fopen = fopen * x;
                }
                const float gbar = (dbar + mu * dt * m.ch_erev[h]) / C;
                acc[64 * slot] += (double)gbar * (double)(fopen * 1e-5f * A);
            }
        }
    }
    __syncthreads();
    for (int k = tid; k < ns; k += 64) {
        double tot = 0.0;
        for (int l = 0; l < 64; l++) tot += smem_d[64 * k + l];
        m.part[(int64_t)(s0 + k) * m.n_part + blockIdx.y] = tot;
    }
}

// slot_grad += the terms of `chunks` blocks of steps, the latest first; a
// resistivity's share is complete, and divided by it, once `done`.
__global__ void k_grad_sum(GradDev m, int n_slot, const int32_t *slot_cell, int chunks, int done) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_slot) return;
    double tot = m.slot_grad[k];
    for (int c = chunks - 1; c >= 0; c--) tot += m.part[(int64_t)k * m.n_part + c];
    const int cell = slot_cell[k];
    if (done && k - m.cell_s0[cell] == m.cell_ra_slot[cell]) tot /= (double)m.params[m.cell_ra_param[cell]];
    m.slot_grad[k] = tot;
}

// The unit-weight exposure of item s at step n and its state update
// (forward Euler; the event's jump instead of the decay in its step).
__device__ __forceinline__ float item_exposure(const GradSyn &st, float a, float b) {
    return st.kind == EDEN_SYN_EXPTWO ? st.gbase * (b - a) : a;
}
__device__ __forceinline__ void item_update(const GradSyn &st, float dt, bool event, float &a, float &b) {
    if (st.kind == EDEN_SYN_EXPTWO) {
        if (event) {
            a = a + st.wf_w;
            b = b + st.wf_w;
        } else {
            a = a + dt * (-a / st.tau_rise);
            b = b + dt * (-b / st.tau_decay);
        }
    } else {
        a = event ? a + st.gbase : a - dt * (a / st.tau_decay);
    }
}

// Unit-weight exposures of the steps [n0, n0 + rows) into ex, a thread per item;
// the items' states go on from the call before (n0 = 1: from rest).
__global__ void k_grad_expose(GradDev m, int64_t n0, int64_t rows) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n_item) return;
    const GradSyn st = m.syn[m.it_type[i]];
    float a = n0 == 1 ? 0.0f : m.it_a[i], b = n0 == 1 ? 0.0f : m.it_b[i];
    int64_t e = n0 == 1 ? m.it_ev0[i] : m.it_cur[i];
    const int64_t e1 = m.it_ev0[i + 1];
    int32_t next = e < e1 ? m.it_ev[e] : -1;
    for (int64_t r = 0; r < rows; r++) {
        m.ex[r * m.n_item + i] = item_exposure(st, a, b);
        const bool event = next == (int32_t)(n0 + r);
        if (event) next = ++e < e1 ? m.it_ev[e] : -1;
        item_update(st, m.dt, event, a, b);
    }
    m.it_a[i] = a;
    m.it_b[i] = b;
    m.it_cur[i] = e;
}

// gtab[n][k] = sum over the group's items of weight * unit-weight exposure for
// the steps in ex (a thread per step and group; items in group order).
__global__ void k_grad_drive(GradDev m, int64_t n0, int64_t rows) {
    const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= rows * m.n_grp) return;
    const int64_t r = id / m.n_grp;
    const int k = (int)(id - r * m.n_grp);
    float g = 0.0f;
    for (int i = m.gr_it0[k]; i < m.gr_it0[k + 1]; i++) {
        const float w = m.it_param[i] >= 0 ? m.params[m.it_param[i]] : m.it_w[i];
        g += w * m.ex[r * m.n_item + i];
    }
    m.gtab[(n0 + r) * m.n_grp + k] = g;
}

// d loss / d weight of each item: sum over the steps in ex, up to N - 1, of the
// group's conductance adjoint times the item's unit-weight exposure, in double
// (a warp per item), added to what the steps before gave.
__global__ void k_grad_weights(GradDev m, int64_t n0, int64_t rows) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= m.n_item) return;
    const int k = m.it_grp[i];
    double acc = 0.0;
    for (int64_t r = lane; r < rows && n0 + r < m.N; r += 32)
        acc += (double)m.gbar[(n0 + r) * m.n_grp + k] * (double)m.ex[r * m.n_item + i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) m.item_grad[i] = n0 == 1 ? acc : m.item_grad[i] + acc;
}

}  // namespace eden_grad

using namespace eden_grad;

struct EdenGpuGrad {
    std::string err;
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    GradDev d{};
    std::vector<void *> allocs;
    int n_params = 0, n_cells = 0, n_rec = 0;
    Dims dims{1, 1, 1, 1};
    // launch shapes: threads of a forward block and its warps of currents; steps
    // of coefficients in flight in the adjoint, and the floats of one
    int fwd_threads = 64, fwd_cw = 1, adj_threads = 64, ring = 1, stage = 4;
    size_t smem = 0, smem_adj = 0;
    bool near_gates = true;  // the forward stages the gates' map
    // rows of the buffers: whether every step's trajectory is kept, the segments
    // recomputed at a time where not, the steps of coefficients, of exposures
    bool keep = false;
    int64_t seg_group = 1, co_rows = 1, ex_rows = 1;
    int32_t *d_slot_cell = nullptr;
    std::vector<int32_t> slot_param;     // slot -> parameter
    std::vector<int32_t> cell_ra_param;  // host copy, for the forward's checks
    std::vector<int32_t> item_param;     // parameter that is each drive item's weight, or -1
    std::vector<float> h_params;
    float *d_params = nullptr, *d_trace = nullptr, *d_tgrad = nullptr;
    double *d_slot = nullptr;
    bool have_forward = false;
    double fwd_ms = 0.0, bwd_ms = 0.0;

    int fail(int code, const char *fmt, ...) {
        char buf[1024];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        err = buf;
        return code;
    }
};

#define GTRY(g, call)                                                                               \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            return (g)->fail(e_ == cudaErrorMemoryAllocation ? EDEN_GPU_E_NOMEM : EDEN_GPU_E_CUDA,  \
                             "%s failed: %s", #call, cudaGetErrorString(e_));                       \
    } while (0)

namespace {

template <typename T>
int upload(EdenGpuGrad *g, const T **dst, const std::vector<T> &src) {
    void *p = nullptr;
    const size_t bytes = std::max<size_t>(src.size(), 1) * sizeof(T);
    GTRY(g, cudaMalloc(&p, bytes));
    g->allocs.push_back(p);
    if (!src.empty()) GTRY(g, cudaMemcpy(p, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
    *dst = static_cast<const T *>(p);
    return 0;
}

template <typename T>
int alloc(EdenGpuGrad *g, T **dst, size_t n) {
    void *p = nullptr;
    GTRY(g, cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
    g->allocs.push_back(p);
    *dst = static_cast<T *>(p);
    return 0;
}

bool finite_pos(float x) { return std::isfinite(x) && x > 0.0f; }

// The bytes of the buffers whose rows can be cut: the trajectory, the adjoint's
// coefficients, the unit-weight exposures.  What a caller says (buffer_mib), else
// a 64th of the device's memory, and of what is free an eighth at most: several
// contexts, or one beside a program that holds most of the device, each take a
// part of the rest.  Fewer rows cost time only: 256 cells of 51 compartments over
// 8,001 steps take 2.1 GB of trajectory and 5.4 GB of coefficients; with 4.4 GB in
// all the first is kept whole and the second is done in three parts.
int buffer_bytes(EdenGpuGrad *g, const EdenGpuGradSpec *s, int64_t *bytes) {
    if (s->buffer_mib > 0) {
        *bytes = (int64_t)s->buffer_mib << 20;
        return 0;
    }
    size_t free_bytes = 0, total = 0;
    GTRY(g, cudaMemGetInfo(&free_bytes, &total));
    *bytes = (int64_t)std::min(total / 64, free_bytes / 8);
    return 0;
}

int validate(EdenGpuGrad *g, const EdenGpuModel *m, const EdenGpuGradSpec *s) {
    if (m->abi_version != EDEN_GPU_ABI_VERSION)
        return g->fail(EDEN_GPU_E_INVALID, "ABI version %d, library is %d", m->abi_version, EDEN_GPU_ABI_VERSION);
    if (!finite_pos(m->dt)) return g->fail(EDEN_GPU_E_INVALID, "dt must be positive");
    if (m->n_izh != 0 || m->n_pois != 0 || m->n_wave != 0 || m->n_clamp != 0 || m->n_gap != 0 || m->n_graded != 0)
        return g->fail(EDEN_GPU_E_INVALID,
                       "gradients cover independent physical cells with HH channels, pulse inputs and synaptic drive "
                       "with fixed events: the model has %d point neurons, %lld Poisson, %lld waveform and %lld clamp "
                       "inputs and %lld gap-junction and graded-synapse ends",
                       m->n_izh, (long long)m->n_pois, (long long)m->n_wave, (long long)m->n_clamp,
                       (long long)(m->n_gap + m->n_graded));
    if (m->cable_solver != EDEN_CABLE_BWD_EULER)
        return g->fail(EDEN_GPU_E_INVALID, "gradients follow the backward-Euler cable solve only");
    for (int k = 0; k < m->n_syn_types; k++) {
        const EdenGpuSynapseType &t = m->syn_types[k];
        if ((t.kind != EDEN_SYN_EXPONE && t.kind != EDEN_SYN_EXPTWO) || !std::isfinite(t.gbase) ||
            !std::isfinite(t.erev) || !finite_pos(t.tau_decay) || (t.kind == EDEN_SYN_EXPTWO && !finite_pos(t.tau_rise)))
            return g->fail(EDEN_GPU_E_INVALID, "synapse type %d: bad parameters", k);
    }
    for (int64_t k = 0; k < m->n_syn; k++) {
        const int src = m->syn_src[k];
        if (src < 0 || src >= m->n_src) return g->fail(EDEN_GPU_E_INVALID, "synapse %lld: bad source", (long long)k);
        if (m->src_target[src] >= 0)
            return g->fail(EDEN_GPU_E_INVALID,
                           "synapse %lld: its presynaptic cell %d spikes, so its events depend on the parameters; "
                           "gradients need synaptic events fixed in advance (spike sources without a membrane)",
                           (long long)k, src);
        if (m->syn_target[k] < 0 || m->syn_target[k] >= m->n_comp || m->syn_type[k] < 0 ||
            m->syn_type[k] >= m->n_syn_types || !(m->syn_delay[k] >= 0.0f) || !std::isfinite(m->syn_delay[k]) ||
            !std::isfinite(m->syn_weight[k]))
            return g->fail(EDEN_GPU_E_INVALID, "synapse %lld: bad target, type, delay or weight", (long long)k);
    }
    for (int64_t k = 0; k < m->n_timed; k++) {
        if (m->timed_target[k] < 0 || m->timed_target[k] >= m->n_comp || m->timed_type[k] < 0 ||
            m->timed_type[k] >= m->n_syn_types || !std::isfinite(m->timed_weight[k]) ||
            m->timed_off[k + 1] < m->timed_off[k])
            return g->fail(EDEN_GPU_E_INVALID, "timed input %lld: bad target, type, weight or steps", (long long)k);
    }
    for (int64_t e = 0; e < m->n_ext; e++)
        if (m->ext_src[e] < 0 || m->ext_src[e] >= m->n_src || (e > 0 && m->ext_step[e] < m->ext_step[e - 1]))
            return g->fail(EDEN_GPU_E_INVALID, "spike-source events must name a source and be sorted by step");
    if (m->n_phys <= 0 || m->n_comp <= 0) return g->fail(EDEN_GPU_E_INVALID, "no physical cells");
    for (int k = 0; k < m->n_chan_types; k++)
        for (int q = 0; q < m->chan_types[k].n_gates && q < EDEN_MAX_GATES; q++)
            if (m->chan_types[k].gate_kind[q] != EDEN_GATE_RATES)
                return g->fail(EDEN_GPU_E_INVALID,
                               "gradients cover gateHHrates gates: channel type %d gate %d is of another kind", k, q);
    if (m->phys_comp_off[0] != 0 || m->phys_comp_off[m->n_phys] != m->n_comp)
        return g->fail(EDEN_GPU_E_INVALID, "phys_comp_off must span [0, n_comp]");
    for (int c = 0; c < m->n_phys; c++) {
        const int a = m->phys_comp_off[c], b = m->phys_comp_off[c + 1];
        if (b <= a) return g->fail(EDEN_GPU_E_INVALID, "cell %d has no compartments", c);
        if (m->comp_parent[a] != -1) return g->fail(EDEN_GPU_E_INVALID, "cell %d: compartment 0 must be the root", c);
        for (int i = a + 1; i < b; i++) {
            const int p = m->comp_parent[i];
            if (p < 0 || p >= i - a)
                return g->fail(EDEN_GPU_E_INVALID, "cell %d compartment %d: parent %d must precede it", c, i - a, p);
            if (!finite_pos(m->comp_r_axial[i])) return g->fail(EDEN_GPU_E_INVALID, "compartment %d: bad axial resistance", i);
        }
    }
    for (int i = 0; i < m->n_comp; i++) {
        if (!finite_pos(m->comp_c[i])) return g->fail(EDEN_GPU_E_INVALID, "compartment %d: bad capacitance", i);
        if (!std::isfinite(m->comp_area[i]) || !std::isfinite(m->comp_inv_rc[i]) || !std::isfinite(m->comp_v0[i]))
            return g->fail(EDEN_GPU_E_INVALID, "compartment %d: non-finite constant", i);
        if (m->comp_chan_off[i + 1] < m->comp_chan_off[i]) return g->fail(EDEN_GPU_E_INVALID, "comp_chan_off not monotone");
    }
    if (m->comp_chan_off[0] != 0) return g->fail(EDEN_GPU_E_INVALID, "comp_chan_off[0] != 0");
    const int n_chan = m->comp_chan_off[m->n_comp];
    for (int ch = 0; ch < n_chan; ch++)
        if (m->chan_type[ch] < 0 || m->chan_type[ch] >= m->n_chan_types)
            return g->fail(EDEN_GPU_E_INVALID, "channel %d: bad type", ch);
    for (int k = 0; k < m->n_chan_types; k++) {
        const EdenGpuChannelType &t = m->chan_types[k];
        if (t.n_gates < 0 || t.n_gates > EDEN_MAX_GATES) return g->fail(EDEN_GPU_E_INVALID, "channel type %d: gate count", k);
        for (int q = 0; q < t.n_gates; q++) {
            if (t.gate_instances[q] < 0 || t.gate_instances[q] > 16) return g->fail(EDEN_GPU_E_INVALID, "gate instances");
            if (t.fwd_kind[q] < 0 || t.fwd_kind[q] > 2 || t.rev_kind[q] < 0 || t.rev_kind[q] > 2)
                return g->fail(EDEN_GPU_E_INVALID, "channel type %d gate %d: rate kind", k, q);
        }
    }
    for (int64_t k = 0; k < m->n_pulse; k++)
        if (m->pulse_target[k] < 0 || m->pulse_target[k] >= m->n_comp)
            return g->fail(EDEN_GPU_E_INVALID, "pulse %lld: target out of range", (long long)k);
    if (s->n_params < 0) return g->fail(EDEN_GPU_E_INVALID, "negative parameter count");
    if (s->n_steps < 1) return g->fail(EDEN_GPU_E_INVALID, "n_steps must be at least 1");
    if (s->checkpoint_every < 0) return g->fail(EDEN_GPU_E_INVALID, "checkpoint_every must not be negative");
    if (s->n_rec < 0 || (s->n_rec > 0 && !s->rec_comp)) return g->fail(EDEN_GPU_E_INVALID, "recorded compartments missing");
    for (int r = 0; r < s->n_rec; r++)
        if (s->rec_comp[r] < 0 || s->rec_comp[r] >= m->n_comp)
            return g->fail(EDEN_GPU_E_INVALID, "recorded compartment %d out of range", r);
    std::vector<char> chan_use(s->n_params, 0), ra_use(s->n_params, 0);
    if (s->chan_param)
        for (int ch = 0; ch < n_chan; ch++) {
            const int p = s->chan_param[ch];
            if (p < -1 || p >= s->n_params) return g->fail(EDEN_GPU_E_INVALID, "channel %d: parameter %d out of range", ch, p);
            if (p >= 0) chan_use[p] = 1;
        }
    if (s->cell_ra_param)
        for (int c = 0; c < m->n_phys; c++) {
            const int p = s->cell_ra_param[c];
            if (p < -1 || p >= s->n_params) return g->fail(EDEN_GPU_E_INVALID, "cell %d: parameter %d out of range", c, p);
            if (p >= 0) {
                if (!s->cell_ra || !finite_pos(s->cell_ra[c]))
                    return g->fail(EDEN_GPU_E_INVALID, "cell %d: resistivity parameter without a positive cell_ra", c);
                ra_use[p] = 1;
            }
        }
    for (int p = 0; p < s->n_params; p++)
        if (chan_use[p] && ra_use[p])
            return g->fail(EDEN_GPU_E_INVALID, "parameter %d is both a conductivity and a resistivity", p);
    auto weight_params = [&](const int32_t *par, int64_t n, const char *what) {
        if (!par) return 0;
        for (int64_t k = 0; k < n; k++) {
            const int p = par[k];
            if (p < -1 || p >= s->n_params)
                return g->fail(EDEN_GPU_E_INVALID, "%s %lld: parameter %d out of range", what, (long long)k, p);
            if (p >= 0 && (chan_use[p] || ra_use[p]))
                return g->fail(EDEN_GPU_E_INVALID, "parameter %d is both a weight and a conductivity or resistivity", p);
        }
        return 0;
    };
    int rc = weight_params(s->syn_param, m->n_syn, "synapse");
    if (rc) return rc;
    return weight_params(s->timed_param, m->n_timed, "timed input");
}

// Host layout: each cell's compartments breadth-first (children in increasing
// order, so a node's children are consecutive), channels and pulses in that
// order, per-cell parameter slots and recorded columns.
int build(EdenGpuGrad *g, const EdenGpuModel *m, const EdenGpuGradSpec *s) {
    const float dt = m->dt;
    const int nphys = m->n_phys;
    GradDev &d = g->d;
    d.n_cells = nphys;
    d.n_rec = s->n_rec;
    d.S = s->checkpoint_every > 0 ? s->checkpoint_every : 100;
    d.N = s->n_steps;
    d.n_comp = m->n_comp;
    d.dt = dt;
    std::vector<int32_t> cell_c0(nphys + 1, 0), cell_g0(nphys + 1, 0), cell_ch0(nphys + 1, 0), cell_l0(nphys + 1, 0),
        cell_s0(nphys + 1, 0), cell_r0(nphys + 1, 0), cell_ra_slot(nphys, -1), cell_ra_param(nphys, -1),
        cell_chain(nphys, 0);
    std::vector<float> cell_ra(nphys, 1.0f);
    std::vector<int32_t> lev, P(m->n_comp), CB(m->n_comp), CE(m->n_comp), comp_ch0, comp_pu0;
    std::vector<float> C(m->n_comp), A(m->n_comp), IRC(m->n_comp), U(m->n_comp, 0.0f), L(m->n_comp, 0.0f),
        V0(m->n_comp);
    std::vector<int32_t> ch_type, ch_g0, ch_param, ch_slot;
    std::vector<float> ch_gbase, ch_erev, pu_start, pu_dur, pu_aw;
    std::vector<int32_t> new_of(m->n_comp);  // model compartment -> breadth-first position
    std::vector<int32_t> comp_g0, comp_cell, gate_map, cell_k0(nphys + 1, 0), slot_cell;
    // pulses by compartment, in pulse order
    std::vector<std::vector<int64_t>> pulses_of(m->n_comp);
    for (int64_t k = 0; k < m->n_pulse; k++) pulses_of[m->pulse_target[k]].push_back(k);
    int64_t n_gate = 0;
    comp_pu0.push_back(0);
    for (int c = 0; c < nphys; c++) {
        const int a = m->phys_comp_off[c], b = m->phys_comp_off[c + 1], nc = b - a;
        std::vector<std::vector<int>> kids(nc);
        for (int i = 1; i < nc; i++) kids[m->comp_parent[a + i]].push_back(i);
        std::vector<int> order, depth_of(nc, 0);
        order.reserve(nc);
        order.push_back(0);
        std::vector<int> pos(nc, 0);
        lev.push_back(0);
        int cur_depth = 0;
        for (size_t h = 0; h < order.size(); h++) {
            const int i = order[h];
            if (depth_of[i] != cur_depth) {
                lev.push_back((int)h);
                cur_depth = depth_of[i];
            }
            pos[i] = (int)h;
            for (int k : kids[i]) {
                depth_of[k] = depth_of[i] + 1;
                order.push_back(k);
            }
        }
        lev.push_back(nc);
        cell_l0[c + 1] = (int32_t)lev.size();
        bool chain = true;  // breadth-first order of an unbranched cable from its end
        for (int h = 0; h + 1 < nc && chain; h++) chain = kids[order[h]].size() == 1 && pos[kids[order[h]][0]] == h + 1;
        cell_chain[c] = chain ? 1 : 0;
        const int gbase_cell = (int)n_gate;
        const int ch_first = (int)ch_type.size();
        std::vector<int32_t> slots;  // parameter of each local slot
        auto slot_of = [&](int p) {
            for (size_t k = 0; k < slots.size(); k++)
                if (slots[k] == p) return (int)k;
            slots.push_back(p);
            return (int)slots.size() - 1;
        };
        for (int h = 0; h < nc; h++) {
            const int i = order[h], gi = a + i, gn = a + h;
            new_of[gi] = gn;
            const int p = m->comp_parent[gi];
            P[gn] = p >= 0 ? pos[p] : -1;
            CB[gn] = kids[i].empty() ? 0 : pos[kids[i].front()];
            CE[gn] = kids[i].empty() ? 0 : pos[kids[i].front()] + (int)kids[i].size();
            C[gn] = m->comp_c[gi];
            A[gn] = m->comp_area[gi];
            IRC[gn] = m->comp_inv_rc[gi];
            V0[gn] = m->comp_v0[gi];
            if (p >= 0) {
                const float R = m->comp_r_axial[gi];
                U[gn] = -dt / (R * m->comp_c[gi]);
                L[gn] = -dt / (R * m->comp_c[a + p]);
            }
            comp_ch0.push_back((int32_t)ch_type.size() - ch_first);  // local to the cell
            comp_g0.push_back((int32_t)(n_gate - gbase_cell));
            comp_cell.push_back(c);
            for (int ch = m->comp_chan_off[gi]; ch < m->comp_chan_off[gi + 1]; ch++) {
                const int pp = s->chan_param ? s->chan_param[ch] : -1;
                ch_type.push_back(m->chan_type[ch]);
                ch_g0.push_back((int32_t)(n_gate - gbase_cell));
                ch_param.push_back(pp);
                ch_slot.push_back(pp >= 0 ? slot_of(pp) : -1);
                ch_gbase.push_back(m->chan_gbase[ch]);
                ch_erev.push_back(m->chan_erev[ch]);
                for (int q = 0; q < m->chan_types[m->chan_type[ch]].n_gates; q++)
                    gate_map.push_back((int32_t)((uint32_t)h | (uint32_t)(m->chan_type[ch] << 2 | q) << 16));
                n_gate += m->chan_types[m->chan_type[ch]].n_gates;
            }
            for (int64_t k : pulses_of[gi]) {
                pu_start.push_back(m->pulse_start[k]);
                pu_dur.push_back(m->pulse_duration[k]);
                pu_aw.push_back(m->pulse_amplitude[k] * m->pulse_weight[k]);
            }
            comp_pu0.push_back((int32_t)pu_start.size());
        }
        if (s->cell_ra_param && s->cell_ra_param[c] >= 0) {
            cell_ra_param[c] = s->cell_ra_param[c];
            cell_ra[c] = s->cell_ra[c];
            cell_ra_slot[c] = slot_of(s->cell_ra_param[c]);
        }
        if ((int)slots.size() > kMaxSlots)
            return g->fail(EDEN_GPU_E_INVALID, "cell %d uses %d parameters, at most %d", c, (int)slots.size(), kMaxSlots);
        for (int32_t p : slots) {
            g->slot_param.push_back(p);
            slot_cell.push_back(c);
        }
        // (rows of coefficients are copied 16 bytes at a time)
        cell_k0[c + 1] = cell_k0[c] + (int32_t)((3 * (nc + (n_gate - gbase_cell)) + 3) & ~(int64_t)3);
        cell_c0[c + 1] = b;
        cell_g0[c + 1] = (int32_t)n_gate;
        cell_ch0[c + 1] = (int32_t)ch_type.size();
        cell_s0[c + 1] = (int32_t)g->slot_param.size();
        g->dims.c = std::max(g->dims.c, nc);
        g->dims.g = std::max(g->dims.g, (int)(n_gate - gbase_cell));
        g->dims.ch = std::max(g->dims.ch, (int)ch_type.size() - ch_first);
        g->dims.slots = std::max(g->dims.slots, (int)slots.size());
    }
    if (n_gate > INT32_MAX) return g->fail(EDEN_GPU_E_INVALID, "too many gates");
    d.n_gate = n_gate;
    // recorded columns grouped by cell
    std::vector<int32_t> cell_of(m->n_comp);
    for (int c = 0; c < nphys; c++)
        for (int i = m->phys_comp_off[c]; i < m->phys_comp_off[c + 1]; i++) cell_of[i] = c;
    std::vector<std::vector<int32_t>> rec_by_cell(nphys);
    for (int r = 0; r < s->n_rec; r++) rec_by_cell[cell_of[s->rec_comp[r]]].push_back(r);
    std::vector<int32_t> rec_local, rec_col, comp_rc0(m->n_comp, 0);
    int max_rec = 0;
    for (int c = 0; c < nphys; c++) {
        // by compartment, then column
        std::stable_sort(rec_by_cell[c].begin(), rec_by_cell[c].end(),
                         [&](int32_t x, int32_t y) { return new_of[s->rec_comp[x]] < new_of[s->rec_comp[y]]; });
        size_t k = 0;
        for (int gc = cell_c0[c]; gc < cell_c0[c + 1]; gc++) {
            comp_rc0[gc] = (int32_t)rec_local.size();
            for (; k < rec_by_cell[c].size() && new_of[s->rec_comp[rec_by_cell[c][k]]] == gc; k++) {
                rec_local.push_back(gc - cell_c0[c]);
                rec_col.push_back(rec_by_cell[c][k]);
            }
        }
        cell_r0[c + 1] = (int32_t)rec_local.size();
        max_rec = std::max(max_rec, (int)rec_by_cell[c].size());
    }
    // step times: the reference accumulates the float dt in double from 0
    // at step 1 and runs each step at that time as a float
    std::vector<float> tk((size_t)d.N + 1, 0.0f);
    double time = 0.0;
    for (int64_t n = 1; n <= d.N; n++) {
        tk[n] = (float)time;
        time += (double)dt;
    }
    // ---- synaptic drive: each item's firing steps (timed inputs: listed;
    // connections from spike sources: the reference's delivery and single
    // pending-spike rule, eden/Eden.cpp:3646-3686, replayed on the source's
    // spikes), then groups of one compartment, kind and synapse type --
    // inputs before connections, types in increasing order -- with their
    // items in model order
    struct Item { int comp, kind, type, param; float w; std::vector<int32_t> ev; };
    std::vector<Item> items;
    {
        std::vector<std::vector<int64_t>> spikes_of(m->n_src);
        for (int64_t e = 0; e < m->n_ext; e++)
            if (m->ext_step[e] >= 1 && m->ext_step[e] < d.N) spikes_of[m->ext_src[e]].push_back(m->ext_step[e]);
        auto due_step = [&](float p) -> int64_t {  // step k in 1 .. N-1 with tk[k] <= p < tk[k] + dt
            const auto it = std::upper_bound(tk.begin() + 1, tk.begin() + d.N, p);
            const int64_t j = (int64_t)(it - tk.begin()) - 1;
            for (int64_t k = std::max<int64_t>(1, j - 1); k <= j && k < d.N; k++)
                if (tk[k] <= p && p < tk[k] + dt) return k;
            return 0;
        };
        for (int64_t k = 0; k < m->n_timed; k++) {
            Item it{new_of[m->timed_target[k]], 0, m->timed_type[k], s->timed_param ? s->timed_param[k] : -1,
                    m->timed_weight[k], {}};
            for (int64_t e = m->timed_off[k]; e < m->timed_off[k + 1]; e++)
                if (m->timed_step[e] >= 1 && m->timed_step[e] < d.N) it.ev.push_back((int32_t)m->timed_step[e]);
            items.push_back(std::move(it));
        }
        for (int64_t k = 0; k < m->n_syn; k++) {
            Item it{new_of[m->syn_target[k]], 1, m->syn_type[k], s->syn_param ? s->syn_param[k] : -1,
                    m->syn_weight[k], {}};
            const float delay = m->syn_delay[k];
            float pend = -INFINITY;
            for (int64_t step : spikes_of[m->syn_src[k]]) {
                const float t = tk[step], fresh = t + delay, tdt = t + dt;
                if (t <= fresh && fresh < tdt) it.ev.push_back((int32_t)step);
                if (pend < tdt && pend < fresh) {
                    pend = fresh;
                    const int64_t kd = due_step(pend);
                    if (kd > 0) it.ev.push_back((int32_t)kd);
                }
            }
            std::sort(it.ev.begin(), it.ev.end());
            it.ev.erase(std::unique(it.ev.begin(), it.ev.end()), it.ev.end());
            items.push_back(std::move(it));
        }
        std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) {
            if (a.comp != b.comp) return a.comp < b.comp;
            if (a.kind != b.kind) return a.kind < b.kind;
            return a.type < b.type;
        });
    }
    std::vector<int32_t> comp_gr0(m->n_comp + 1, 0), gr_kind, gr_it0, it_grp, it_type, it_param, it_ev;
    std::vector<int64_t> it_ev0{0};
    std::vector<float> gr_erev, it_w;
    for (size_t i = 0; i < items.size(); i++) {
        const Item &it = items[i];
        if (i == 0 || it.comp != items[i - 1].comp || it.kind != items[i - 1].kind || it.type != items[i - 1].type) {
            gr_kind.push_back(it.kind);
            gr_erev.push_back(m->syn_types[it.type].erev);
            gr_it0.push_back((int32_t)i);
            comp_gr0[it.comp + 1]++;
        }
        it_grp.push_back((int32_t)gr_kind.size() - 1);
        it_type.push_back(it.type);
        it_param.push_back(it.param);
        it_w.push_back(it.w);
        it_ev.insert(it_ev.end(), it.ev.begin(), it.ev.end());
        it_ev0.push_back((int64_t)it_ev.size());
    }
    gr_it0.push_back((int32_t)items.size());
    for (int i = 0; i < m->n_comp; i++) comp_gr0[i + 1] += comp_gr0[i];
    std::vector<GradSyn> syn(std::max(m->n_syn_types, 1));
    for (int k = 0; k < m->n_syn_types; k++) {
        const EdenGpuSynapseType &t = m->syn_types[k];
        syn[k] = GradSyn{t.kind, t.gbase, t.tau_decay, t.tau_rise, t.weight_prop * t.waveform_factor};
    }
    d.n_grp = (int32_t)gr_kind.size();
    d.n_item = (int64_t)items.size();
    g->item_param = it_param;
    g->cell_ra_param = cell_ra_param;
    // launch shapes and shared memory
    const Dims &dm = g->dims;
    d.n_types = m->n_chan_types;
    g->fwd_cw = std::min(4, (dm.c + 31) / 32);
    g->fwd_threads = 32 * (g->fwd_cw + std::min(kFwdWarps - g->fwd_cw, n_gate > 0 ? std::max(1, (dm.g + 31) / 32) : 0));
    g->smem = (size_t)m->n_chan_types * sizeof(EdenGpuChannelType) +
              (size_t)(9 * dm.c + 10 * kBlock + 2 * dm.g + 2 * dm.ch) * sizeof(float) +
              (size_t)(4 * dm.c + 1 + 2 * dm.ch + dm.g) * sizeof(int32_t);
    int optin = 0;
    GTRY(g, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device));
    g->stage = ((3 * (dm.c + dm.g) + 3) / 4 * 4 + max_rec + 3) / 4 * 4;
    const size_t adj = ((size_t)6 * dm.c + 2 + dm.g) * sizeof(float);
    g->adj_threads = std::min(256, std::max(64, (dm.c + 31) / 32 * 32));
    g->ring = kRing;
    while (g->ring > 1 && adj + sizeof(float) * g->ring * (size_t)g->stage > (size_t)(g->ring > 2 ? 100 * 1024 : optin)) g->ring /= 2;
    // the largest cells: coefficients, or the gates' map, read where they are
    if (adj + sizeof(float) * g->ring * (size_t)g->stage > (size_t)optin) g->ring = 0;
    g->near_gates = g->smem <= (size_t)optin;
    if (!g->near_gates) g->smem -= dm.g * sizeof(int32_t);
    g->smem_adj = adj + sizeof(float) * g->ring * (size_t)g->stage;
    if (std::max(g->smem, g->smem_adj) > (size_t)optin)
        return g->fail(EDEN_GPU_E_INVALID, "largest cell (%d compartments, %d gates) needs %zu bytes of shared memory, "
                                           "the device allows %d", dm.c, dm.g, std::max(g->smem, g->smem_adj), optin);
    // (the limit belongs to the kernels, which every context launches: the
    // device's own, so that no context lowers another's)
    for (const void *fn : {(const void *)k_grad_forward<false, true>, (const void *)k_grad_forward<true, true>,
                           (const void *)k_grad_forward<false, false>, (const void *)k_grad_forward<true, false>,
                           (const void *)k_grad_adjoint<true>, (const void *)k_grad_adjoint<false>})
        GTRY(g, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    std::vector<EdenGpuChannelType> types(m->chan_types, m->chan_types + m->n_chan_types);
    int rc;
#define UP(dst, src) \
    if ((rc = upload(g, &d.dst, src)) != 0) return rc
    UP(cell_c0, cell_c0); UP(cell_g0, cell_g0); UP(cell_ch0, cell_ch0); UP(cell_l0, cell_l0); UP(cell_s0, cell_s0); UP(cell_r0, cell_r0);
    UP(cell_ra_slot, cell_ra_slot); UP(cell_ra_param, cell_ra_param); UP(cell_chain, cell_chain); UP(cell_ra, cell_ra); UP(lev, lev);
    UP(C, C); UP(A, A); UP(IRC, IRC); UP(U, U); UP(L, L); UP(V0, V0);
    UP(P, P); UP(CB, CB); UP(CE, CE); UP(comp_ch0, comp_ch0); UP(comp_pu0, comp_pu0);
    UP(ch_type, ch_type); UP(ch_g0, ch_g0); UP(ch_param, ch_param); UP(ch_slot, ch_slot);
    UP(ch_gbase, ch_gbase); UP(ch_erev, ch_erev); UP(types, types);
    UP(pu_start, pu_start); UP(pu_dur, pu_dur); UP(pu_aw, pu_aw);
    UP(rec_local, rec_local); UP(rec_col, rec_col); UP(tk, tk);
    UP(comp_gr0, comp_gr0); UP(gr_kind, gr_kind); UP(gr_it0, gr_it0); UP(it_grp, it_grp); UP(it_type, it_type);
    UP(it_param, it_param); UP(it_ev, it_ev); UP(it_ev0, it_ev0); UP(gr_erev, gr_erev); UP(it_w, it_w);
    UP(syn, syn); UP(cell_k0, cell_k0); UP(comp_cell, comp_cell); UP(gate_map, gate_map); UP(comp_g0, comp_g0);
    UP(comp_rc0, comp_rc0);
#undef UP
    if (d.n_grp > 0) {
        const size_t rows = (size_t)(d.N + 1) * d.n_grp;
        if ((rc = alloc(g, &d.gtab, rows)) != 0) return rc;
        if ((rc = alloc(g, &d.gbar, rows)) != 0) return rc;
        if ((rc = alloc(g, &d.it_a, (size_t)d.n_item)) != 0) return rc;
        if ((rc = alloc(g, &d.it_b, (size_t)d.n_item)) != 0) return rc;
        if ((rc = alloc(g, &d.it_cur, (size_t)d.n_item)) != 0) return rc;
        if ((rc = alloc(g, &d.item_grad, (size_t)d.n_item)) != 0) return rc;
        GTRY(g, cudaMemset(d.gbar, 0, rows * sizeof(float)));
    }
    const int64_t n_ck = d.N >= 2 ? (d.N - 2) / d.S + 1 : 1;
    if ((rc = alloc(g, &g->d_params, (size_t)std::max(s->n_params, 1))) != 0) return rc;
    d.params = g->d_params;
    if ((rc = alloc(g, &d.ck_v, (size_t)n_ck * m->n_comp)) != 0) return rc;
    if ((rc = alloc(g, &d.ck_q, (size_t)n_ck * n_gate)) != 0) return rc;
    if ((rc = alloc(g, &d.lv, (size_t)m->n_comp)) != 0) return rc;
    if ((rc = alloc(g, &d.lq, (size_t)n_gate)) != 0) return rc;
    {
        const int32_t *p = nullptr;
        if ((rc = upload(g, &p, slot_cell)) != 0) return rc;
        g->d_slot_cell = const_cast<int32_t *>(p);
    }
    if ((rc = alloc(g, &g->d_trace, (size_t)d.N * std::max(s->n_rec, 1))) != 0) return rc;
    d.trace = g->d_trace;
    if ((rc = alloc(g, &g->d_tgrad, (size_t)d.N * std::max(s->n_rec, 1))) != 0) return rc;
    d.trace_grad = g->d_tgrad;
    if ((rc = alloc(g, &g->d_slot, g->slot_param.size())) != 0) return rc;
    d.slot_grad = g->d_slot;
    // then what can be cut, from what is left: half for the trajectory, of the
    // whole run where it fits, else of as many segments; most of the rest for
    // the coefficients; a 16th for the exposures
    int64_t budget = 0;
    if ((rc = buffer_bytes(g, s, &budget)) != 0) return rc;
    const int64_t tr_row = 4 * (2 * (int64_t)m->n_comp + n_gate), tr_bytes = budget / 2;
    g->keep = d.N * tr_row <= tr_bytes;
    g->seg_group = g->keep ? n_ck : std::max<int64_t>(1, std::min<int64_t>({n_ck, 65535, tr_bytes / tr_row / d.S}));
    const int64_t tr_rows = g->keep ? d.N : std::min<int64_t>(d.N, g->seg_group * d.S + 1);
    if ((rc = alloc(g, &d.tr_v, (size_t)tr_rows * m->n_comp)) != 0) return rc;
    if ((rc = alloc(g, &d.tr_q, (size_t)tr_rows * n_gate)) != 0) return rc;
    if ((rc = alloc(g, &d.tr_d, (size_t)tr_rows * m->n_comp)) != 0) return rc;
    d.co_len = cell_k0[nphys];
    g->co_rows = std::min<int64_t>({tr_rows, 1 << 20,
                                    std::max<int64_t>(kSumSteps, budget / 16 * 7 / (4 * ((int64_t)d.co_len + m->n_comp)))});
    if ((rc = alloc(g, &d.co, (size_t)g->co_rows * d.co_len)) != 0) return rc;
    if ((rc = alloc(g, &d.mu, (size_t)g->co_rows * m->n_comp)) != 0) return rc;
    d.n_part = (int32_t)((g->co_rows + kSumSteps - 1) / kSumSteps);
    if ((rc = alloc(g, &d.part, g->slot_param.size() * (size_t)d.n_part)) != 0) return rc;
    if (d.n_grp > 0) {
        g->ex_rows = std::min<int64_t>(d.N, std::max<int64_t>(kSumSteps, budget / 16 / (4 * d.n_item)));
        if ((rc = alloc(g, &d.ex, (size_t)g->ex_rows * d.n_item)) != 0) return rc;
    }
    g->n_params = s->n_params;
    g->n_cells = nphys;
    g->n_rec = s->n_rec;
    return 0;
}

}  // namespace

extern "C" int edenGpuGradCreate(const EdenGpuModel *model, const EdenGpuGradSpec *spec, EdenGpuGrad **out) {
    if (!out) return EDEN_GPU_E_INVALID;
    EdenGpuGrad *g = new EdenGpuGrad();
    *out = g;
    if (!model || !spec) return g->fail(EDEN_GPU_E_INVALID, "null model or spec");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return g->fail(EDEN_GPU_E_NODEVICE, "no CUDA device visible");
    }
    g->device = spec->device;
    if (g->device < 0 || g->device >= ndev) return g->fail(EDEN_GPU_E_INVALID, "device %d not present", g->device);
    GTRY(g, cudaSetDevice(g->device));
    int rc = validate(g, model, spec);
    if (rc) return rc;
    GTRY(g, cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    GTRY(g, cudaEventCreate(&g->e0));
    GTRY(g, cudaEventCreate(&g->e1));
    rc = build(g, model, spec);
    if (rc) return rc;
    GTRY(g, cudaDeviceSynchronize());
    return 0;
}

extern "C" int edenGpuGradForward(EdenGpuGrad *g, const float *params, float *trace) {
    if (!g) return EDEN_GPU_E_INVALID;
    if (!g->stream) return g->fail(EDEN_GPU_E_INVALID, "gradient context was not created");
    if (g->n_params > 0 && !params) return g->fail(EDEN_GPU_E_INVALID, "params missing");
    GTRY(g, cudaSetDevice(g->device));
    g->h_params.assign(std::max(g->n_params, 1), 0.0f);
    if (g->n_params > 0)
        GTRY(g, cudaMemcpy(g->h_params.data(), params, sizeof(float) * g->n_params, cudaMemcpyDefault));
    for (int c = 0; c < g->n_cells; c++) {
        const int p = g->cell_ra_param[c];
        if (p >= 0 && !finite_pos(g->h_params[p]))
            return g->fail(EDEN_GPU_E_INVALID, "parameter %d (a resistivity) must be positive, is %g", p, g->h_params[p]);
    }
    for (int p = 0; p < g->n_params; p++)
        if (!std::isfinite(g->h_params[p])) return g->fail(EDEN_GPU_E_INVALID, "parameter %d is not finite", p);
    GTRY(g, cudaMemcpyAsync(g->d_params, g->h_params.data(), sizeof(float) * g->h_params.size(), cudaMemcpyHostToDevice,
                            g->stream));
    GTRY(g, cudaEventRecord(g->e0, g->stream));
    if (g->d.n_grp > 0)
        for (int64_t n0 = 1; n0 <= g->d.N; n0 += g->ex_rows) {
            const int64_t rows = std::min<int64_t>(g->ex_rows, g->d.N + 1 - n0);
            k_grad_expose<<<(unsigned)((g->d.n_item + 127) / 128), 128, 0, g->stream>>>(g->d, n0, rows);
            k_grad_drive<<<(unsigned)((rows * g->d.n_grp + 127) / 128), 128, 0, g->stream>>>(g->d, n0, rows);
        }
    g->d.tr_n0 = 1;
    (g->near_gates ? k_grad_forward<false, true> : k_grad_forward<false, false>)<<<g->n_cells, g->fwd_threads, g->smem, g->stream>>>(
        g->d, g->dims, g->fwd_cw, 0, g->keep ? 1 : 0);
    GTRY(g, cudaGetLastError());
    GTRY(g, cudaEventRecord(g->e1, g->stream));
    if (trace && g->n_rec > 0)
        GTRY(g, cudaMemcpyAsync(trace, g->d_trace, sizeof(float) * (size_t)g->d.N * g->n_rec, cudaMemcpyDefault,
                                g->stream));
    GTRY(g, cudaStreamSynchronize(g->stream));
    float ms = 0.0f;
    GTRY(g, cudaEventElapsedTime(&ms, g->e0, g->e1));
    g->fwd_ms = ms;
    g->have_forward = true;
    return 0;
}

extern "C" int edenGpuGradBackward(EdenGpuGrad *g, const float *trace_grad, float *param_grad) {
    if (!g) return EDEN_GPU_E_INVALID;
    if (!g->have_forward) return g->fail(EDEN_GPU_E_INVALID, "edenGpuGradBackward needs an edenGpuGradForward first");
    if (!param_grad && g->n_params > 0) return g->fail(EDEN_GPU_E_INVALID, "param_grad missing");
    if (!trace_grad && g->n_rec > 0) return g->fail(EDEN_GPU_E_INVALID, "trace_grad missing");
    GTRY(g, cudaSetDevice(g->device));
    if (g->n_rec > 0)
        GTRY(g, cudaMemcpyAsync(g->d_tgrad, trace_grad, sizeof(float) * (size_t)g->d.N * g->n_rec, cudaMemcpyDefault,
                                g->stream));
    GTRY(g, cudaEventRecord(g->e0, g->stream));
    GradDev &d = g->d;
    const int n_slot = (int)g->slot_param.size();
    GTRY(g, cudaMemsetAsync(d.lv, 0, sizeof(float) * d.n_comp, g->stream));
    GTRY(g, cudaMemsetAsync(d.lq, 0, sizeof(float) * std::max<int64_t>(d.n_gate, 1), g->stream));
    GTRY(g, cudaMemsetAsync(g->d_slot, 0, sizeof(double) * std::max(n_slot, 1), g->stream));
    // groups of segments, the last first; in each, blocks of steps, the last first
    bool last = true;
    for (int64_t hi = d.N >= 2 ? (d.N - 2) / d.S + 1 : 0; hi > 0;) {
        const int64_t lo = std::max<int64_t>(0, hi - g->seg_group);
        const int64_t n0 = 1 + lo * d.S, n1 = std::min<int64_t>(1 + hi * d.S, d.N);
        d.tr_n0 = g->keep ? 1 : n0;
        if (!g->keep)
            (g->near_gates ? k_grad_forward<true, true> : k_grad_forward<true, false>)
                <<<dim3(g->n_cells, (unsigned)(hi - lo)), g->fwd_threads, g->smem, g->stream>>>(d, g->dims, g->fwd_cw, lo, 1);
        for (int64_t b = n1; b > n0;) {
            const int64_t a = std::max<int64_t>(n0, b - g->co_rows), rows = b - a;
            const int chunks = (int)((rows + kSumSteps - 1) / kSumSteps);
            d.co_n0 = a;
            k_grad_coef<<<(unsigned)((rows * d.n_comp + 127) / 128), 128, 0, g->stream>>>(d, rows);
            (g->ring > 0 ? k_grad_adjoint<true> : k_grad_adjoint<false>)
                <<<g->n_cells, g->adj_threads, g->smem_adj, g->stream>>>(d, g->dims, rows, g->ring, g->stage, last ? 1 : 0);
            k_grad_terms<<<dim3(g->n_cells, chunks), 64, (size_t)64 * g->dims.slots * sizeof(double), g->stream>>>(d, rows);
            if (n_slot > 0)
                k_grad_sum<<<(n_slot + 127) / 128, 128, 0, g->stream>>>(d, n_slot, g->d_slot_cell, chunks, a == 1 ? 1 : 0);
            last = false;
            b = a;
        }
        hi = lo;
    }
    if (d.n_item > 0)
        for (int64_t n0 = 1; n0 <= d.N; n0 += g->ex_rows) {
            const int64_t rows = std::min<int64_t>(g->ex_rows, d.N + 1 - n0);
            // (the forward's exposures are still there where one block holds them all)
            if (g->ex_rows < d.N)
                k_grad_expose<<<(unsigned)((d.n_item + 127) / 128), 128, 0, g->stream>>>(d, n0, rows);
            k_grad_weights<<<(unsigned)((d.n_item * 32 + 127) / 128), 128, 0, g->stream>>>(d, n0, rows);
        }
    GTRY(g, cudaGetLastError());
    GTRY(g, cudaEventRecord(g->e1, g->stream));
    std::vector<double> slots(g->slot_param.size()), items((size_t)g->d.n_item);
    if (!slots.empty())
        GTRY(g, cudaMemcpyAsync(slots.data(), g->d_slot, sizeof(double) * slots.size(), cudaMemcpyDeviceToHost, g->stream));
    if (!items.empty())
        GTRY(g, cudaMemcpyAsync(items.data(), g->d.item_grad, sizeof(double) * items.size(), cudaMemcpyDeviceToHost,
                                g->stream));
    GTRY(g, cudaStreamSynchronize(g->stream));
    float ms = 0.0f;
    GTRY(g, cudaEventElapsedTime(&ms, g->e0, g->e1));
    g->bwd_ms = ms;
    // per parameter, the cells' terms in cell order
    std::vector<double> acc(std::max(g->n_params, 1), 0.0);
    for (size_t k = 0; k < slots.size(); k++) acc[g->slot_param[k]] += slots[k];
    for (size_t k = 0; k < items.size(); k++)  // the weights' terms in item order
        if (g->item_param[k] >= 0) acc[g->item_param[k]] += items[k];
    std::vector<float> out(std::max(g->n_params, 1));
    for (int p = 0; p < g->n_params; p++) out[p] = (float)acc[p];
    if (g->n_params > 0) GTRY(g, cudaMemcpy(param_grad, out.data(), sizeof(float) * g->n_params, cudaMemcpyDefault));
    return 0;
}

extern "C" int edenGpuGradTiming(EdenGpuGrad *g, double *forward_ms, double *backward_ms) {
    if (!g) return EDEN_GPU_E_INVALID;
    if (forward_ms) *forward_ms = g->fwd_ms;
    if (backward_ms) *backward_ms = g->bwd_ms;
    return 0;
}

extern "C" const char *edenGpuGradLastError(EdenGpuGrad *g) { return g ? g->err.c_str() : "null gradient context"; }

extern "C" void edenGpuGradDestroy(EdenGpuGrad *g) {
    if (!g) return;
    if (g->stream) {
        cudaSetDevice(g->device);
        cudaStreamSynchronize(g->stream);
    }
    for (void *p : g->allocs) cudaFree(p);
    if (g->e0) cudaEventDestroy(g->e0);
    if (g->e1) cudaEventDestroy(g->e1);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
}
