// The kernels of libeden_gpu.  This header is compiled twice: ahead of time
// into the library, and at context creation by NVRTC together with code
// generated for the model's mechanisms (EDEN_RTC, see eden_codegen.cu), the
// GPU counterpart of the per-cell-type C the reference generates and
// compiles with gcc (eden/Eden.cpp:7017-7180).
#pragma once
#include "eden_kernels.cuh"

namespace eden {

constexpr int kThreads = 256;
constexpr int kInputThreads = 128;  // k_inputs_t: four warps, each with two event tiles
constexpr int kCellThreads = 768;   // k_cells_t: at most, a warp per unit; the registers of 24 warps an SM
constexpr int kHinesThreads = 128;  // k_hines_t: four warps, each staging one forest

}  // namespace eden

// ---------------------------------------------------------------------------
// kernels; each reads its WindowArgs from a device table so that a captured
// graph can be replayed over many windows
//
// edenGpuRun launches a window's kernels so that each may start while the one
// before it drains: `kernel_order` waits until everything before has finished
// and is visible, and only then lets the next kernel start, so that one kernel
// at most is ahead of the running one.  Before it a kernel reads nothing but
// its arguments, the window tables and the model's constants, which no kernel of
// a window writes.  (Launched without that allowance, it does not wait.)
// ---------------------------------------------------------------------------
namespace eden {

__device__ __forceinline__ void kernel_order() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Phase 1 of both paths: input blocks over the window (the per-step path runs
// it with K = 1), a warp per group of consecutive chunks.  A group grows past
// one chunk only when there are more chunks than resident warps: a small
// model's chunks all run at once, a large model's items with full warps.
// The event tiles are only as long as the model's windows (dynamic shared
// memory), so that the registers, 32 warps an SM, bound the occupancy.
__global__ void __launch_bounds__(kInputThreads, 8) k_inputs_t(DevModel m, const WindowArgs *tab,
                                                             const WindowTimes *ttab, const int *base, int idx) {
    extern __shared__ __align__(16) float sm[];
    __shared__ HotItem lists[kInputThreads / 32][kHotItems];
    __shared__ float tk[64];  // the window's step times, then the previous window's
    const int wi = *base + idx;
    const WindowArgs w = tab[wi];
    kernel_order();
    if (threadIdx.x < 64) tk[threadIdx.x] = threadIdx.x < 32 ? ttab[wi].tk[threadIdx.x] : ttab[wi].tprev[threadIdx.x - 32];
    __syncthreads();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    float *tileA = sm + (threadIdx.x >> 5) * 64 * m.acc_stride, *tileB = tileA + 32 * m.acc_stride;
    HotItem *list = lists[threadIdx.x >> 5];
    const int group = min(kInputGroup, (m.n_chunk + nwarps - 1) / nwarps);
    for (int64_t c = (int64_t)warp * group; c < m.n_chunk; c += (int64_t)nwarps * group)
        input_group(m, (int)c, min(group, m.n_chunk - (int)c), w, tileA, tileB, list, tk);
}

// Per-step path, phase 2: one thread per target.
__global__ void __launch_bounds__(256) k_targets_t(DevModel m, const WindowArgs *tab, const WindowTimes *ttab,
                                                   const int *base, int idx) {
    const WindowArgs w = tab[*base + idx];
    const float tnow = ttab[*base + idx].tk[0];
    // the constants of the thread's first target into L1 before the wait
    {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i < m.n_target) {
            auto fetch = [](const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); };
            const int b0 = m.t_blk0[i], b1 = m.t_blk0[i + 1], h0 = m.c_chan0[i], h1 = m.c_chan0[i + 1];
            fetch(&m.t_izh[i]); fetch(&m.t_trace0[i]);
            fetch(&m.c_area[i]); fetch(&m.c_cm[i]); fetch(&m.c_inv_rc[i]);
            if (b1 > b0) { fetch(&m.bk_kind[b0]); fetch(&m.bk_erev[b0]); fetch(&m.bk_c0[b0]); }
            if (h1 > h0) {
                fetch(&m.ch_type[h0]); fetch(&m.ch_gate0[h0]); fetch(&m.ch_gbase[h0]); fetch(&m.ch_erev[h0]);
            }
        }
    }
    kernel_order();
    const bool init = w.step0 <= 0;
    const float *vin = m.v[w.par];
    float *vout = m.v[w.par ^ 1];
    const int n = m.n_target;
    const int nround = (n + 31) & ~31;  // whole warps stay converged for the spike ballot
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nround; i += gridDim.x * blockDim.x) {
        if (i < n) {
            float v = vin[i], Iin, Gin, Isyn, Gsyn;
            block_currents(m.Gp, m.gp_stride, m.t_blk0[i], m.t_blk0[i + 1], m.bk_kind, m.bk_erev, m.bk_c0, v, Iin, Gin,
                           Isyn, Gsyn, m.bk_block);
            if (EDEN_KIND_GAP) Isyn += gap_current(m, i, v, vin, init);
            const float Iax = (m.fwd_euler && !init && m.t_izh[i] < 0) ? axial_current(m, i, v, vin) : 0.0f;
            target_step(m, i, init, w.step0, tnow, v, Iin, Gin, Isyn, Gsyn, &vout[i], &m.diag[i], w.wpar, Iax);
        }
    }
}

// Per-step path, phase 3: one warp per forest, staged in the warp's slice of
// shared memory when the forest has at most `cap` compartments.
__global__ void __launch_bounds__(kHinesThreads) k_hines_t(DevModel m, const WindowArgs *tab, const int *base, int idx, int cap) {
    extern __shared__ float sm[];
    const WindowArgs w = tab[*base + idx];
    const bool init = w.step0 <= 0;
    const float *vin = m.v[w.par];
    float *x = m.v[w.par ^ 1];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    // per-warp slice: D, X, U, L, V, child ends, parents, depth boundaries (cap each)
    float *sD = sm + (size_t)wib * 8 * cap, *sX = sD + cap, *sU = sX + cap, *sL = sU + cap, *sV = sL + cap;
    int32_t *sCE = (int32_t *)(sV + cap), *sP = sCE + cap, *sLV = sP + cap;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // What no kernel writes -- a forest's off-diagonals, its tree, its spike
    // sources -- is loaded before the wait, beside the kernel of the targets.
    // Bound by a step's chain of depths; a test of every compartment for a
    // source took five rounds of loads after it.  (1,000 trees, a step of all four
    // kernels: 38.0 us, 35.2 so and with the targets' constants fetched early.)
    bool waited = false;
    for (int f = warp; f < m.n_forest; f += nwarps) {
        const int c0 = m.fo_t0[f], n = m.fo_t1[f] - c0, nlev = m.fo_nlev[f];
        const int32_t *lv = m.lvl + m.fo_l0[f];
        const bool staged = !m.fwd_euler && !m.fo_f64[f] && n <= cap && nlev < cap;
        if (staged) {
            for (int i = lane; i < n; i += 32) {
                sU[i] = m.c_u[c0 + i]; sL[i] = m.c_l[c0 + i];
                sCE[i] = m.c_cend[c0 + i] - c0; sP[i] = m.c_parent[c0 + i] - c0;
            }
            for (int i = lane; i <= nlev; i += 32) sLV[i] = lv[i] - c0;
        }
        const ForestSource src = forest_source(m, m.fo_s0[f] + lane, m.fo_s0[f + 1]);
        if (!waited) kernel_order();
        waited = true;
        if (m.fwd_euler) {
            // V_next is final already: only the threshold test
        } else if (m.fo_f64[f]) {
            hines_forest_f64(m, init, m.diag, x, m.c_u, m.c_l, m.c_cend, m.c_parent, lv, nlev, m.dscr,
                             m.dscr + m.n_target);
        } else if (staged) {
            for (int i = lane; i < n; i += 32) {
                sD[i] = m.diag[c0 + i]; sX[i] = x[c0 + i]; sV[i] = vin[c0 + i];
            }
            __syncwarp();
            hines_forest(m, init, sD, sX, sU, sL, sCE, sP, sLV, nlev);
            __syncwarp();
            for (int i = lane; i < n; i += 32) x[c0 + i] = sX[i];
            forest_spikes(m, f, src, w.step0, w.t0, sX, sV, c0, w.wpar);
            __syncwarp();
            continue;
        } else {
            hines_forest(m, init, m.diag, x, m.c_u, m.c_l, m.c_cend, m.c_parent, lv, nlev);
        }
        __syncwarp();
        forest_spikes(m, f, src, w.step0, w.t0, x, vin, 0, w.wpar);
    }
    // Warps without a forest wait as well: a grid that ended without it would let
    // the delivery, which waits for this grid only, start while the targets' kernel
    // still runs.  (Of a network without any forest it is not launched.)
    if (!waited) kernel_order();
}

// Fan the spikes of window `w` out to their synapses' trigger masks
// (bit = logging step - window start = the step at which the reference reads
// the trigger, eden/Eden.cpp:3964-3992) and append them to the spike log.
__global__ void __launch_bounds__(256) k_deliver_t(DevModel m, const WindowArgs *tab, const int *base, int idx) {
    const WindowArgs w = tab[*base + idx];
    kernel_order();
    const int wp = w.wpar;
    const int n = m.wspk_count[wp];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // the other parity's list was consumed by the previous window's delivery
    // and is refilled only by the next window: clear it for that window
    if (blockIdx.x == 0 && threadIdx.x == 0) m.wspk_count[wp ^ 1] = 0;
    // then the window's spikes of sources with no target (spike lists and
    // generators, computed in advance)
    const int n_all = n + (w.ext1 - w.ext0);
    for (int e = warp; e < n_all; e += nwarps) {
        const bool own = e < n;
        int src = own ? m.wspk_src[wp][e] : m.ext_src[w.ext0 + e - n];
        int log_step = own ? m.wspk_step[wp][e] : m.ext_step[w.ext0 + e - n];
        uint32_t bit = 1u << (uint32_t)(log_step - w.step0);
        int64_t f0 = m.fan0[src], f1 = m.fan0[src + 1];
        for (int64_t f = f0 + lane; f < f1; f += 32) atomicOr(&m.sy_mask[m.fan_syn[f]], bit);
    }
    // the log, 32 spikes a warp and from the last warp on: its count is one
    // address for all, where additions of one spike each queued (5,400 spikes of
    // 100 synapses: 37 us, 17 so)
    for (int64_t e0 = 32 * (int64_t)(nwarps - 1 - warp); e0 < n_all; e0 += 32 * (int64_t)nwarps) {
        const int e = (int)e0 + lane, count = min(32, n_all - (int)e0);
        unsigned long long slot = 0;
        if (lane == 0) slot = atomicAdd(m.log_count, (unsigned long long)count);
        slot = __shfl_sync(0xffffffffu, slot, 0) + lane;
        if (lane < count) {
            if ((int64_t)slot < m.log_cap) {
                const bool own = e < n;
                m.log_src[slot] = own ? m.wspk_src[wp][e] : m.ext_src[w.ext0 + e - n];
                m.log_step[slot] = own ? m.wspk_step[wp][e] : m.ext_step[w.ext0 + e - n];
                m.log_time[slot] = own ? m.wspk_time[wp][e] : no_time();
            } else {
                atomicOr(m.status, ST_LOG_OVERFLOW);
            }
        }
    }
}

// Windowed path: every warp advances one unit (a forest of physical cells or
// a batch of izhikevich neurons) K steps on its own, synchronising only within
// the warp.  Within a window no cell reads another cell's state: the only
// coupling is through synaptic triggers, and every connection delay is
// >= K * dt, so a spike emitted inside the window cannot fire a synapse before
// the window ends.  Its trigger bits are delivered after the window
// (k_deliver_t) and replayed in order at the start of the next one
// (replay_mask), which reproduces the step-by-step pending-spike decisions
// exactly.  Synaptic conductances do not depend on V, so k_inputs_t has
// already produced them for all K steps.  Everything else a step reads is
// staged in the warp's shared-memory slice for the whole window.

// The series of a unit's blocks, into shared memory, where some have several
// chunks: those are summed over them here, a thread four steps.  In the steps it
// would be a lane a block, one load after the other.  (One compartment of 128,000
// inputs, a window of 29 steps: 742 us by steps, 129 so; 20 compartments with
// 51,200 together: 102 and 87.)
__device__ __noinline__ void stage_sums(float *GS, const float *Gp, const int32_t *c0, int nblk, int gps, int th, int nth) {
    const int quads = gps >> 2;
    for (int i = th; i < nblk * quads; i += nth) {
        const int b = i / quads, c = c0[b], nc = c0[b + 1] - c;
        const float *p = &Gp[(size_t)c * gps + 4 * (i - b * quads)];
        if (nc == 1) stage_rec(&GS[4 * i], p);
        else *reinterpret_cast<float4 *>(&GS[4 * i]) = sum_chunks(p, gps, nc);
    }
}
// The same of a point neuron's blocks [b0, b1), into their first chunk's series,
// by the lane that reads it.  (100 neurons of 10,000 synapses, a window of 10 steps:
// 218 us by steps, 80 so; 300 of 300: 28 and 28.)
__device__ __noinline__ void sum_blocks(float *Gk, const int4 *BK, int b0, int b1, int gps, int K) {
    for (int b = b0; b < b1; b++) {
        const int4 r = BK[b];
        if (r.y == 1) continue;
#pragma unroll 2
        for (int k = 0; k < K; k += 4) {
            float *p = &Gk[r.x + k];
            *reinterpret_cast<float4 *>(p) = sum_chunks(p, gps, r.y);
        }
    }
}

// A forest unit over the window.  At the window start the unit stages its
// nodes', twigs' and non-flat compartments' records, its gates, its input
// blocks, and the conductance series of its input chunks for all K steps
// (written by k_inputs_t), so that a step reads shared memory only.  Per step: trajectory samples of the step's starting V; the
// non-flat compartments' currents (inputs, channels with the gate values before
// this step's update), diagonal and pre-update; gate updates from the starting
// V, into the other of the gates' two buffers; the cable solve; threshold
// crossings.  A lane with at most one non-flat compartment, or one gate, keeps
// its record in registers for the whole window.
//
// The gates and the currents of a step both read its starting state only, so a
// unit with gates is run by two warps: one (`gates`) updates the gates, and
// tests the thresholds a step behind, beside the other's currents and solve,
// with a barrier of the two a step.  With gate_warp unset one warp does all of it
// in turn.
//
// With the unit in shared memory the kernel moves 15 times less than a step
// over HBM would, and is bound by the length of a step's dependent chain and,
// with many units, by the instructions issued: hence few instructions a pass,
// divisions by constants done as div_known, and units sized in edenGpuCreate.
// (A kernel compiled for a model without gate warps keeps the threshold test in
// the loop that takes V over; with them, one body for both roles: compiled
// apart, the solve of 50 trees took 112 us a window instead of 100.)
//
// WIDE: for models with many inputs.  Blocks of several chunks are summed as they
// are staged (stage_sums), and a unit too large for a block's shared memory (un_far)
// reads its blocks' records where they are; a step finds them in L1.  (Without it
// a block has one chunk.  One kernel for both: 2,000 trees, the built-in kernels,
// 8.08 us a step, 7.19 apart; with the body in a function of its own the same 8.08.)
template <bool WIDE>
__device__ __forceinline__ void forest_window(const DevModel &m, const WindowArgs &w, int u, float *S, bool gates,
                                              int barrier, bool first) {
    const int lane = threadIdx.x & 31;
    const int t0 = m.un_t0[u], fi = m.un_f[u], ub0 = m.t_blk0[t0], nblk = m.t_blk0[m.un_t1[u]] - ub0;
    const int n0 = m.fo_n0[fi], n = m.fo_n0[fi + 1] - n0, w0 = m.fo_w0[fi], nw = m.fo_w0[fi + 1] - w0;
    const int ngt = m.un_ngt[u], gt0 = m.un_gt0[u];
    const bool pair = EDEN_GATE_WARPS && m.gate_warp && ngt > 0;
    if (gates && !pair) return;
    // the unit's threads, and a barrier of them
    const int th = gates ? lane + 32 : lane, nth = pair ? 64 : 32;
    auto unit_sync = [&]() {
        if (pair) asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
        else __syncwarp();
    };
    const int r0 = m.un_r0[u], r1 = m.un_r1[u];
    const int nf0 = m.un_nf0[u], nf = m.un_nf1[u] - nf0;
    const int ps0 = m.fo_p0[fi], np = m.fo_p0[fi + 1] - ps0;
    const int uc0 = m.bk_c0[ub0], nck = m.bk_c0[ub0 + nblk] - uc0;
    const int uch0 = m.un_ch0[u], nch = m.un_ch1[u] - uch0;
    float2 *XR = reinterpret_cast<float2 *>(S);
    float *TX = S + twig_words(n + 1), *TV = TX + 32 * nw;
    float4 *CN = reinterpret_cast<float4 *>(TV + 32 * nw), *TR = CN + n + 1;
    float4 *NF = TR + 32 * nw;
    const bool far = WIDE && m.un_far[u] != 0;
    int4 *BKs = reinterpret_cast<int4 *>(NF + kSlotRecs * nf);
    const int4 *BK = far ? m.bk_rec + ub0 : BKs;
    const int gps = m.gp_stride;
    float *GS = reinterpret_cast<float *>(BKs + (far ? 0 : nblk));
    float2 *TS = reinterpret_cast<float2 *>(GS + gps * nblk);
    uint32_t *TA = reinterpret_cast<uint32_t *>(TS + nf);
    float *VO = (float *)(TA + 32 * nw);  // three buffers of nf: step k starts from buffer k % 3
    float *CHG = VO + 3 * nf, *CHE = CHG + nch;
    int32_t *CHQ = (int32_t *)(CHE + nch), *CHI = CHQ + nch;
    int32_t *GI = CHI + nch;
    float *GT = (float *)(GI + ngt);  // two buffers of ngt
    int32_t *PS = (int32_t *)(GT + 2 * ngt);
    // a double-precision forest's eliminated values, pivots and factors
    const bool f64 = m.fo_f64[fi] != 0;
    double *XD = reinterpret_cast<double *>((reinterpret_cast<unsigned long long>(PS + np) + 7ull) & ~7ull);
    double *PVD = XD + n, *RTD = PVD + n;
    // the steps of a window are all initialisation passes or none is
    const bool init = w.step0 <= 0;
    // ---- stage the unit: its records first, which are there before the window's
    // inputs, then what earlier kernels wrote
    for (int i = th; i < n; i += nth) {
        stage_rec(&CN[i], &m.c_rec[n0 + i]);
        stage_word(&XR[i].y, &m.nd_rt[n0 + i]);
    }
    if (th == 0) {
        XR[n] = make_float2(0.0f, 0.0f);
        CN[n] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    for (int i = th; i < 32 * nw; i += nth) {
        stage_rec(&TR[i], &m.tw_rec[32 * w0 + i]);
        stage_word(&TA[i], &m.tw_adr[32 * w0 + i]);
    }
    for (int i = th; i < kSlotRecs * nf; i += nth) stage_rec(&NF[i], &m.nf_rec[(size_t)kSlotRecs * nf0 + i]);
    if (!far)
        for (int i = th; i < nblk; i += nth) stage_rec(&BKs[i], &m.bk_rec[ub0 + i]);
    for (int j = th; j < nf; j += nth) {
        stage_word(&TS[j].x, &m.nf_ts[nf0 + j].x); stage_word(&TS[j].y, &m.nf_ts[nf0 + j].y);
    }
    for (int c = th; c < nch; c += nth) {
        stage_word(&CHG[c], &m.nfc_g[uch0 + c]); stage_word(&CHE[c], &m.nfc_e[uch0 + c]);
        stage_word(&CHQ[c], &m.nfc_q[uch0 + c]); stage_word(&CHI[c], &m.nfc_i[uch0 + c]);
    }
    for (int i = th; i < ngt; i += nth) stage_word(&GI[i], &m.gt_idx[gt0 + i]);
    for (int i = th; i < np; i += nth) stage_word(&PS[i], &m.ps[ps0 + i]);
    if (first) kernel_order();
    const float *vsrc = m.v[w.par];
    for (int i = th; i < n; i += nth) {
        const int t = m.nd_t[n0 + i];
        stage_word(&XR[i].x, &vsrc[t0 + (t >= 0 ? t : -1 - t)]);
    }
    for (int i = th; i < 32 * nw; i += nth) {
        const int t = m.tw_t[32 * w0 + i];
        stage_word(&TV[i], &vsrc[t0 + (t >= 0 ? t : 0)]);
    }
    for (int i = th; i < ngt; i += nth) stage_word(&GT[i], &m.gate[gt0 + i]);
    if (!WIDE || nck == nblk)
        for (int i = 4 * th; i < gps * nck; i += 4 * nth) stage_rec(&GS[i], &m.Gp[(size_t)uc0 * gps + i]);
    else
        stage_sums(GS, m.Gp, m.bk_c0 + ub0, nblk, gps, th, nth);
    stage_wait();
    unit_sync();
    for (int j = th; j < nf; j += nth) VO[j] = XR[__float_as_int(NF[kSlotRecs * j].x) & kPassStart].x;
    for (int i = th; i < 32 * nw; i += nth) TX[i] = TV[i] + TR[i].x;  // the first step's pre-update
    unit_sync();
    const float dt = m.dt;
    float *Gq = GT, *Gn = GT + ngt;  // gate values at the step's start, and at the next's
    float4 ga, gb, gc;               // the lane's only gate, where it has no more
    int gs = 0;
    // gate updates from step k's starting V and gate values (an instantaneous
    // gate takes the potential after the step: one warp, after the solve)
    auto update_gates = [&](int k, const float *Vq) {
#pragma unroll 1
        for (int q = lane; q < ngt; q += 32) {
            if (k == 0 || ngt > 32) {
                gs = GI[q];
                const float4 *r = m.gate_tab + kGateRecs * (gs >> 10);
                ga = r[0]; gb = r[1]; gc = r[2];
                gs &= kPassStart;
            }
            Gn[q] = gate_next_p(ga, gb, gc, m.gate_ext, init, dt, Vq[gs],
                                EDEN_KIND_GATEFORMS && !pair ? XR[__float_as_int(NF[kSlotRecs * gs].x) & kPassStart].x : 0.0f,
                                Gq[q]);
        }
    };
    // the lanes' threshold crossings in step k (eden/Eden.cpp:6247-6252)
    auto threshold = [&](int k, bool slot, const float2 &ts, float vo, float vn) {
        const bool spk = slot && vo < ts.x && ts.x < vn;
        if (__any_sync(0xffffffffu, spk)) {
            // (this step's time, accumulated in double as the host does)
            double t = w.t0;
            if (!init)
                for (int i = 0; i < k; i++) t += (double)dt;
            push_spike(m, spk, spk ? __float_as_int(ts.y) : -1, (int32_t)(w.step0 + k + 1), w.wpar,
                       spk ? crossing_time(t, dt, vo, vn, ts.x) : 0.0);
        }
    };
    auto thresholds = [&](int k, const float *Vl, const float *Vq) {
#pragma unroll 1
        for (int j0 = 0; j0 < nf; j0 += 32) {
            const int j = j0 + lane;
            threshold(k, j < nf, j < nf ? TS[j] : make_float2(0.0f, 0.0f), j < nf ? Vl[j] : 0.0f, j < nf ? Vq[j] : 0.0f);
        }
    };
    if (EDEN_GATE_WARPS && gates) {
        const float *Vl = nullptr, *Vq = VO;  // the potentials the last step and this one start from
#pragma unroll 1
        for (int k = 0; k < w.K; k++) {
            update_gates(k, Vq);
            if (k > 0) thresholds(k - 1, Vl, Vq);
            unit_sync();
            float *g = Gq;
            Gq = Gn;
            Gn = g;
            Vl = Vq;
            Vq = Vq == VO + 2 * nf ? VO : Vq + nf;
        }
        thresholds(w.K - 1, Vl, Vq);
        for (int i = lane; i < ngt; i += 32) m.gate[gt0 + i] = Gq[i];
        return;
    }
    int p1 = 0;  // the first pass below the roots
    while (p1 < np && (PS[p1] & kPassRoot)) p1++;
    __syncwarp();
    int row = 0;  // the first step's row of the trajectory buffer
    if (r1 > r0) row = (int)((w.step0 + m.trace_cap - 1) % m.trace_cap);
    float4 sa, sb;  // the lane's only slot, where it has no more
    float2 ts;
    float *Vq = VO;
#pragma unroll 1
    for (int k = 0; k < w.K; k++) {
        if (r1 > r0) {
            // trajectory samples of this step's starting state
            if (!init) {
#pragma unroll 1
                for (int q = r0 + lane; q < r1; q += 32) {
                    const int32_t tq = m.gr_t[q];
                    m.trace_buf[(size_t)row * m.n_trace + m.gr_col[q]] =
                        tq < 0 ? Gq[-1 - tq] : (tq & 1) ? TV[tq >> 1] : XR[tq >> 1].x;
                }
                row = row + 1 == (int)m.trace_cap ? 0 : row + 1;
            }
            __syncwarp();
        }
        const float *Gk = GS + k;
#pragma unroll 1
        for (int j = lane; j < nf; j += 32) {
            // channels + voltage pre-update (eden/Eden.cpp:5013-6107)
            if (k == 0 || nf > 32) { sa = NF[kSlotRecs * j]; sb = NF[kSlotRecs * j + 1]; }
            const int slot = __float_as_int(sa.x), ti = slot & kPassStart;
            const int brange = __float_as_int(sb.y), crange = __float_as_int(sb.z);
            const int ch0 = crange & 0xffff;
            const float v = Vq[j];
            float Iin, Gin, Isyn, Gsyn;
            block_currents_rec(Gk, BK, brange & 0xffff, (int)((uint32_t)brange >> 16), v, Iin, Gin, Isyn, Gsyn);
            // (a model with gap junctions runs one-step windows: vsrc holds
            // every target's potential at this step's start)
            if (EDEN_KIND_GAP) Isyn += gap_current(m, t0 + m.nd_t[n0 + ti], v, vsrc, init);
            const float A = sa.y;
            float Ich = 0.f, Gch = 0.f;
#ifdef EDEN_RTC_CHANNELS
            // the routine generated for this compartment's channel set
            if (!rtc_channels(__float_as_int(sb.w), Gq + CHQ[ch0], CHG, CHE, ch0, v, A, Ich, Gch))
#endif
#pragma unroll 1
            for (int c = ch0; c < ch0 + (int)((uint32_t)crange >> 16); c++) {
                const int gi_pack = CHI[c];
                const float *q = Gq + CHQ[c];
                float fopen = 1.0f;
                for (int gi = 0; gi < (gi_pack & 7); gi++) {
                    const float qo = q[gi];
                    const int inst = (gi_pack >> (3 + 5 * gi)) & 31;
                    for (int rr = 0; rr < inst; rr++) fopen = fopen * qo;
                }
                const float g = CHG[c] * fopen;
                Ich += (g * (CHE[c] - v) * 1e-5f) * A;
                Gch += (g * 1e-5f) * A;
            }
            const float I = Ich + Iin + Isyn;
            const float G = Gch + Gin + Gsyn;
            const float C = sa.z, rC = sa.w;
            float d = 1.0f * div_known(G, C, rC) + sb.x;
            float x = init ? v : v + div_known(dt * (I + (v * G)), C, rC);
            if (!f64) {
                d = 1.0f + d * dt;
                if ((slot & kSlotDone) && !init) x = x * pivot(d);
            }
            CN[ti].z = d;
            XR[ti].x = x;
        }
        if (!EDEN_KIND_GATEFORMS && !pair) update_gates(k, Vq);
        __syncwarp();
        if (!init) {
            // (a double-precision forest has no twigs: its nodes are its compartments)
            if (f64) hines_window_f64(dt, XR, CN, m.c_l + t0, PS, np, n, XD, PVD, RTD);
            else hines_window(dt, S, XR, CN, PS, np, p1, n, TX, TV, TR, TA, nw);
        }
        if (EDEN_KIND_GATEFORMS && !pair) {
            update_gates(k, Vq);
            __syncwarp();
        }
        // V for the next step, and the thresholds if there is no other warp for them
        if (EDEN_GATE_WARPS) {
            float *Vn = Vq == VO + 2 * nf ? VO : Vq + nf;
#pragma unroll 1
            for (int j = lane; j < nf; j += 32) {
                if (nf > 32) sa.x = NF[kSlotRecs * j].x;
                Vn[j] = XR[__float_as_int(sa.x) & kPassStart].x;
            }
            unit_sync();
            if (!pair) thresholds(k, Vq, Vn);
            Vq = Vn;
        } else {
#pragma unroll 1
            for (int j0 = 0; j0 < nf; j0 += 32) {
                const int j = j0 + lane;
                float vo = 0.0f, vn = 0.0f;
                if (j < nf) {
                    if (nf > 32) sa.x = NF[kSlotRecs * j].x;
                    if (k == 0 || nf > 32) ts = TS[j];
                    vo = Vq[j];
                    vn = XR[__float_as_int(sa.x) & kPassStart].x;
                    Vq[j] = vn;
                }
                threshold(k, j < nf, ts, vo, vn);
            }
            __syncwarp();
        }
        float *g = Gq;
        Gq = Gn;
        Gn = g;
    }
    // ---- write the unit back into the buffer that holds the window's final state
    float *vdst = m.v[w.par ^ (w.K & 1)];
    for (int i = lane; i < n; i += 32) {
        const int t = m.nd_t[n0 + i];
        if (t >= 0) vdst[t0 + t] = XR[i].x;
    }
    for (int i = lane; i < 32 * nw; i += 32) {
        const int t = m.tw_t[32 * w0 + i];
        if (t >= 0) vdst[t0 + t] = TV[i];
    }
    if (!pair)
        for (int i = lane; i < ngt; i += 32) m.gate[gt0 + i] = Gq[i];
}

// A batch of up to 32 point neurons over the window (izhikevich2007Cell,
// iaf*Cell, adExIaFCell; point_update), one lane each.
// Beside forests it is called, not inlined: in one body with them it took
// registers from their loops (5,000 cells of 100 compartments with neurons, a
// window: 108 us, 100 so); alone it is inlined (100,000 neurons: 29 us, 34 called).
#if EDEN_KIND_FOREST
#define EDEN_IZH_CALL __noinline__
#else
#define EDEN_IZH_CALL __forceinline__
#endif
template <bool WIDE>
__device__ EDEN_IZH_CALL void izh_window(const DevModel &m, const WindowArgs &w, const float *tk, int u, float *S,
                                           bool first) {
    const int lane = threadIdx.x & 31;
    const int t0 = m.un_t0[u], n = m.un_t1[u] - t0;
    const int r0 = m.un_r0[u], r1 = m.un_r1[u];
    // slice: V (two buffers), the parameters (stride n), then u, s and the kind
    float *P = S + 2 * n;
    float *SU = P + EDEN_POINT_PARAMS * n, *SS = SU + n;
    int32_t *KIND = (int32_t *)(SS + n);
    const int izh0 = m.t_izh[t0];
    for (int i = lane; i < n; i += 32) {
        const int iz = izh0 + i;
        for (int f = 0; f < EDEN_POINT_PARAMS; f++) stage_word(&P[f * n + i], &m.iz_p[(size_t)f * m.n_izh + iz]);
        stage_word(&KIND[i], &m.iz_kind[iz]);
    }
    if (first) kernel_order();
    for (int i = lane; i < n; i += 32) {
        const int iz = izh0 + i;
        stage_word(&S[w.par * n + i], &m.v[w.par][t0 + i]);
        stage_word(&SU[i], &m.iz_u[iz]);
        stage_word(&SS[i], &m.iz_s[iz]);
    }
    stage_wait();
    __syncwarp();
    int par = w.par;
    const float dt = m.dt;
    // the lane's neuron: its input blocks, the unit's chunks, its spike source, and
    // the steps of the window it spikes in
    const int ub0 = m.t_blk0[t0];
    const int b0 = lane < n ? m.t_blk0[t0 + lane] - ub0 : 0, b1 = lane < n ? m.t_blk0[t0 + lane + 1] - ub0 : 0;
    const int4 *BK = m.bk_rec + ub0;
    float *Gk = m.Gp + (size_t)m.bk_c0[ub0] * m.gp_stride;
    if (WIDE) sum_blocks(Gk, BK, b0, b1, m.gp_stride, w.K);
    const int src = lane < n ? m.t_src[t0 + lane] : -1;
    uint32_t spikes = 0;
    for (int k = 0; k < w.K; k++) {
        const int64_t step = w.step0 + k;
        const bool init = step <= 0;
        const float *vin = S + par * n;
        float *vout = S + (par ^ 1) * n;
        const int i = lane;
        if (i < n) {
            const float v = vin[i];
            float Iin, Gin, Isyn, Gsyn;
            block_currents_rec(Gk + k, BK, b0, b1, v, Iin, Gin, Isyn, Gsyn);
            float uu = SU[i], ss = SS[i], vn;
            if (point_update(KIND[i], P + i, n, init, tk[k], dt, v, Isyn + Iin, uu, ss, vn)) spikes |= 1u << k;
            vout[i] = vn;
            SU[i] = uu;
            SS[i] = ss;
        }
        if (!init && r1 > r0) {
            const int64_t row = (step - 1) % m.trace_cap;
            for (int q = r0 + lane; q < r1; q += 32) m.trace_buf[row * m.n_trace + m.gr_col[q]] = vin[m.gr_t[q]];
        }
        __syncwarp();
        par ^= 1;
    }
    // the window's spikes take their places in the list together: its count is
    // one address for all warps, and a step would wait for its own addition
    // (100,000 neurons, 10 steps: 41 us with one a step, 29 so and with the
    // input blocks' records read whole)
    if (src < 0) spikes = 0;
    int at = __popc(spikes);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, at, d);
        if (lane >= d) at += u;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31);
    if (total > 0) {
        int first_at = 0;
        if (lane == 0) first_at = atomicAdd(&m.wspk_count[w.wpar], total);
        at += __shfl_sync(0xffffffffu, first_at, 0) - __popc(spikes);
        for (uint32_t r = spikes; r; r &= r - 1, at++) {
            m.wspk_src[w.wpar][at] = src;
            m.wspk_step[w.wpar][at] = (int32_t)(w.step0 + __ffs(r));
            m.wspk_time[w.wpar][at] = no_time();
        }
    }
    for (int i = lane; i < n; i += 32) {
        m.v[par][t0 + i] = S[par * n + i];
        m.iz_u[izh0 + i] = SU[i];
        m.iz_s[izh0 + i] = SS[i];
    }
}

// This launch runs CTAs [cta_begin, cta_end), each a few units, one per warp of
// the first half of the block, where units' gates have warps of their own (the
// other half's, unit by unit, so that each half spreads over the SM's four
// schedulers), else one per warp.
// A block runs several CTAs in turn when there are more CTAs than blocks;
// their units are laid out differently in shared memory, so every warp of
// the block finishes its unit before any starts on the next CTA.
// WIDE: for models with many inputs (forest_window); compiled for a model, as it is.
#ifdef EDEN_RTC
constexpr bool WIDE = EDEN_WIDE_INPUTS != 0;
#else
template <bool WIDE>
#endif
__global__ void __launch_bounds__(kCellThreads, 1) k_cells_t(const __grid_constant__ DevModel m, const WindowArgs *tab,
                                                          const WindowTimes *ttab, const int *base, int idx,
                                                          int cta_begin, int cta_end) {
    extern __shared__ __align__(16) float sm[];
    const WindowArgs w = tab[*base + idx];
    const float *tk = ttab[*base + idx].tk;
    const int units = EDEN_GATE_WARPS && m.gate_warp ? blockDim.x >> 6 : blockDim.x >> 5;
    const int warp = threadIdx.x >> 5;
    const bool gates = warp >= units;
    const int slot = gates ? warp - units : warp;
    for (int cta = cta_begin + blockIdx.x; cta < cta_end; cta += gridDim.x) {
        const bool first = cta == cta_begin + (int)blockIdx.x;
        const int u = m.cta_u0[cta] + slot;
        if (u < m.cta_u0[cta + 1]) {
            if (m.un_f[u] >= 0) {
                if (EDEN_KIND_FOREST) forest_window<WIDE>(m, w, u, sm + m.un_off[u], gates, 1 + slot, first);
            } else if (EDEN_KIND_IZH && !gates) izh_window<WIDE>(m, w, tk, u, sm + m.un_off[u], first);
        }
        if (cta + (int)gridDim.x < cta_end) __syncthreads();
    }
}

__global__ void k_bump(int *base, int by) { *base += by; }

}  // namespace eden
