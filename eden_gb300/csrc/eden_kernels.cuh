// Device functions of libeden_gpu: one step of EDEN's loop, split into the
// phases of the reference's generated per-cell kernel, over structure-of-arrays
// device tables.  The kernels that drive them are in eden_window.cuh:
//   * the per-step path launches k_inputs -> k_targets -> k_hines -> k_deliver
//     once per step (the reference runs one OpenMP pass per step);
//   * the windowed path launches k_inputs -> k_cells -> k_deliver once per window:
//     k_cells advances each unit K steps with its state in shared memory,
//     because within K <= min synaptic delay / dt steps no cell can affect
//     another.
//
// Internal layout (built on the host in eden_gpu.cu):
//   units     a forest of physical cells, or up to 32 point neurons: one warp, or
//             one and another for its gates;
//   forests   a forest's compartments are numbered breadth-first over all its
//             cells at once, so each tree depth is one contiguous range and
//             every node's children are contiguous, in increasing original
//             index; a forest is solved by one warp;
//   targets   every membrane potential: forest compartments, then the
//             point neurons;
//   inputs    connection synapses, Poisson inputs and pulses sorted by target;
//             a target's are cut into blocks of a kind and chunks of a block.
#pragma once
#ifndef __CUDACC_RTC__
#include <cstdint>
#endif

#include "eden_math.cuh"

namespace eden {

struct ChanTypeDev {
    int n_gates;
    int inst[EDEN_MAX_GATES];
    int fk[EDEN_MAX_GATES];
    float fr[EDEN_MAX_GATES], fm[EDEN_MAX_GATES], fs[EDEN_MAX_GATES];
    int rk[EDEN_MAX_GATES];
    float rr[EDEN_MAX_GATES], rm[EDEN_MAX_GATES], rs[EDEN_MAX_GATES];
    float q10[EDEN_MAX_GATES];
    int gk[EDEN_MAX_GATES];  // EDEN_GATE_*, then the timeCourse and steadyState forms
    int tk[EDEN_MAX_GATES];
    float tr[EDEN_MAX_GATES], tm[EDEN_MAX_GATES], ts[EDEN_MAX_GATES];
    int ik[EDEN_MAX_GATES];
    float ir[EDEN_MAX_GATES], im[EDEN_MAX_GATES], is[EDEN_MAX_GATES];
};
struct SynTypeDev {
    int kind;
    float gbase, erev, tau_decay, tau_rise, wf_w;  // wf_w = weight_prop * waveform_factor
    float r_decay, r_rise;                          // correctly rounded 1 / tau
    float f_decay, f_rise;                          // 1 - dt / tau, one step's decay factor
    float c_alpha;                                  // alpha kinds: e dt / tau, g' = f g + c A
    // blockingPlasticSynapse: plasticity (plastic != 0) with release
    // probability p and one step's factors 1 - dt/tau_rec, 1 - dt/tau_fac
    // (f_fac 1: U stays p)
    int plastic;
    float rel_p, f_rec, f_fac;
};

// x / tau, correctly rounded, from r = RN(1/tau): q = RN(x*r) is within an
// ulp of the quotient, the residual x - tau*q is exact in one FMA, and
// RN(q + r*residual) is the correctly rounded quotient (Markstein's
// theorem, the basis of software division on FMA machines).  The residual
// is exact only away from the underflow range, so an operand below 2^-100
// is scaled by 2^64 first (exact) and the quotient scaled back (exact unless
// the quotient itself is subnormal, where it may differ from the correctly
// rounded one by one subnormal ulp, 2^-149).  Branch-free: synapse states
// that have decayed to tiny values or zero are common, and a divergent
// branch to a hardware division there cost more than the division saves.
__device__ __forceinline__ float div_by_tau(float x, float tau, float r) {
    const bool tiny = fabsf(x) < 0x1p-100f;
    const float xs = tiny ? x * 0x1p64f : x;
    const float q = xs * r;
    const float e = fmaf(-q, tau, xs);
    const float qs = fmaf(e, r, q);
    return tiny ? qs * 0x1p-64f : qs;
}


enum : int { ST_OK = 0, ST_LOG_OVERFLOW = 1 };
enum : int { BK_PULSE = 0, BK_POIS = 1, BK_SYN = 2, BK_TIMED = 3 };
// block-level only: a voltage clamp's sum of weight / R, applied as -V g
// (its chunks run as pulse-block type kClampB)
enum : int { BK_CLAMPV = 4 };
// a synapse block of a current-based kind (alphaCurrentSynapse) carries this
// flag beside its kind: its exposure is a current, with no conductance
enum : int { BK_KIND_MASK = 7, BK_CURRENT = 8, BK_BLOCK = 16 };
// pulse-block types: 0 pulses, then the waveform shapes, then the two halves of a clamp
enum : int { kPulseSine = 1 + EDEN_WAVE_SINE, kPulseRamp = 1 + EDEN_WAVE_RAMP, kClampA = 3, kClampB = 4 };
constexpr int kMaxWindow = 31;  // trigger bits 1..K of a 32-bit mask
constexpr int kChunkItems = 128; // input items per chunk (one warp, up to four per lane)
constexpr int kPowLen = 33;      // powers 0..32 of a synapse decay factor
constexpr int kWaveWords = 8;    // waveform input record: delay, duration, 3 shape parameters, weight, 2 spare
constexpr int kClampWords = 8;   // clamp record: delay, duration, 3 phase targets, R, weight, spare

struct DevModel {
    int32_t n_target, n_src, n_forest;
    // channel and synapse type tables (per context, so that contexts of
    // different models can run side by side)
    const ChanTypeDev *chan_types;
    const SynTypeDev *syn_types;
    float dt;
    // targets
    float *v[2];
    float *diag;
    const float *c_cm, *c_inv_rc, *c_area, *c_u, *c_l;  // U = -dt/(R C_i), L = -dt/(R C_parent)
    const int32_t *c_cend, *c_parent;  // end of each node's child range; parent (internal, -1 at roots)
    const int32_t *t_izh;                            // izhikevich index or -1
    // forward-Euler cable update (fwd_euler != 0): each node's axial
    // resistance to its parent and the start of its child range
    int32_t fwd_euler;
    const float *c_rax;
    const int32_t *c_kb;
    // windowed-path constants of each physical compartment.  A "flat"
    // compartment has one gateless channel, no inputs, is no spike source and
    // has only flat compartments below it; everything else is "non-flat".
    // c_rec, one 16-byte record:
    //   x  flat: the pre-update increment dt*(G*E)/C (V' = V + x, the
    //      reference's V + dt*(I + V*G)/C with I = G*(E - V)); non-flat:
    //      its L (its elimination factor is L / pivot, rebuilt each step)
    //   y  U
    //   z  flat: reciprocal of its Hines pivot, which is the same every
    //      step because nothing below it changes (in a double-precision
    //      forest its constant diagonal term G/C + sum 1/(R C)); non-flat:
    //      written each step
    //   w  children | first child << 10 | parent (a root: 0) << 20
    //      | non-flat << 30 | a twig's topmost << 31, as nodes of the
    //      compartment's forest
    // A forest's compartments are its nodes -- the non-flat ones and the flat
    // ones over a large subtree, solved depth by depth -- and its twigs: flat
    // subtrees, each walked by one lane (hines_window).  A twig's topmost
    // compartment is a node too, a leaf of them.  Nodes [fo_n0[f], fo_n0[f + 1]):
    // c_rec; nd_t, the compartment (local to its unit), or -1 - it for a twig's
    // topmost; nd_rt, flat: L / pivot, the elimination factor into the parent.
    // Twigs: rows [fo_w0[f], fo_w0[f + 1]) of 32 places, a lane's compartments
    // children first; per place tw_rec (the pre-update increment, U, reciprocal
    // pivot, elimination factor), tw_adr (the word its elimination goes to
    // | kTwigTop | the word of its parent's V << 16, in the unit's slice of
    // shared memory) and tw_t, the compartment (-1: empty).
    const float4 *c_rec, *tw_rec;
    const float *nd_rt;
    const int32_t *fo_n0, *nd_t, *fo_w0, *tw_t;
    const uint32_t *tw_adr;
    // forests: physical compartments [fo_t0, fo_t1), depth boundaries lvl[fo_l0 .. fo_l0 + fo_nlev]
    const int32_t *fo_t0, *fo_t1, *fo_l0, *fo_nlev, *lvl;
    // the windowed path's warp passes over forest f, ps[fo_p0[f] .. fo_p0[f + 1]),
    // roots first: up to 32 consecutive compartments of one depth (kPass*)
    const int32_t *fo_p0, *ps;
    // channels
    const int32_t *c_chan0, *ch_type, *ch_gate0;
    const float *ch_gbase, *ch_erev;
    float *gate;
    // point neurons: kind, parameters field-major ([EDEN_POINT_PARAMS][n_izh]),
    // two state variables besides V (izhikevich u, adEx w; last spike time)
    int32_t n_izh;
    const int32_t *iz_kind;
    const float *iz_p;
    float *iz_u, *iz_s;
    // input blocks: each target's pulses, then Poisson inputs and connection
    // synapses in runs of one synapse type; a block's value for a step of the window
    // is its conductance (of pulses and currents, the current)
    const int32_t *t_blk0;            // [n_target + 1]
    const int32_t *bk_kind;           // BK_PULSE, BK_POIS, BK_SYN, BK_TIMED
    const float *bk_erev;
    // blocks are cut into chunks of at most kChunkItems items, one warp each; step k's
    // partial sum of chunk c is Gp[c * gp_stride + k] and a block's value is the
    // sum of its chunks' partials in chunk order
    int32_t n_chunk;
    const int32_t *bk_c0;             // [blocks + 1] chunk range of each block
    const int32_t *ck_info;           // kind | synapse type << 2 | items << 8
    const int64_t *ck_i0;             // first item of each chunk
    float *Gp;                        // [n_chunk * gp_stride]
    int32_t gp_stride;                // steps of the longest window, a multiple of four (1: per-step path)
    int32_t acc_stride;               // of the input kernel's event tiles: odd, at least those steps
    const float *syn_pow;             // per synapse type: f_rise^j, then f_decay^j, j < kPowLen
    int32_t pois_exact;               // dt is a whole number of us: Poisson clocks advance exactly
    float *ck_a, *ck_b;               // aggregate synapse state of each chunk (weighted sums)
    const float *pu_start, *pu_dur, *pu_amp, *pu_w;
    const float *gate_ext;            // per channel type and gate, kGateExtWords (gate_next_p)
    const float *wv_p;                // sine / ramp generators, kWaveWords per item
    const float *cl_p;                // voltage clamps, kClampWords per item
    // Poisson inputs
    float *po_ts, *po_isi, *po_a, *po_b;  // po_a/po_b: own synapse state just after its last event
    int32_t *po_last;                      // step of that event
    const float *po_rate, *po_w;
    const int32_t *po_seed, *po_inst;
    const int32_t *po_rng;                 // random-call id of the input's first draw
    // timedSynapticInput items: own synapse state (as Poisson items), weight,
    // type, the steps each fires in (tm_step[tm_off[i] .. tm_off[i+1]]) and
    // the next one due
    float *tm_a, *tm_b;
    int32_t *tm_last;
    const float *tm_w;
    const int64_t *tm_off, *tm_step;
    int64_t *tm_cur;
    // connection synapses
    float *sy_a, *sy_b, *sy_pend;     // sy_a/sy_b: state just after the synapse's last event
    float *sy_R, *sy_U;               // blockingPlasticSynapse: plasticity state after the last event
    const float2 *bk_block;           // per input block: the voltage block's ratio and scaling voltage
    int32_t *sy_last;                 // step of that event
    uint32_t *sy_mask;
    const float *sy_w, *sy_delay;
    // the targets of forest f that spike sources watch, fo_s[fo_s0[f] .. fo_s0[f + 1])
    const int32_t *fo_s0, *fo_s;
    // spike sources and fan-out (source -> synapses, connection order)
    const int32_t *t_src;
    const float *src_thr;
    const int64_t *fan0;
    const int32_t *fan_syn;
    // spikes of the sources with no target, in step order: source, logging step
    const int32_t *ext_src, *ext_step;
    // window spike lists (double-buffered by window parity) and the spike log;
    // *_time: the threshold-crossing time (us) interpolated in double
    // between the step's starting and final potential (NaN where there is
    // none: point neurons and sources with no membrane)
    int32_t *wspk_src[2];
    int32_t *wspk_step[2];
    double *wspk_time[2];
    int32_t *wspk_count;  // [2]
    int32_t *log_src;
    int64_t *log_step;
    double *log_time;
    unsigned long long *log_count;
    int64_t log_cap;
    // trajectory recording: CSR target -> recorded columns
    const int32_t *t_trace0, *trace_col;
    const int32_t *trace_gate;  // per listed column: the gate slot it records, or -1 for V
    int32_t n_trace;
    float *trace_buf;
    int64_t trace_cap;
    // units of the windowed kernel, one warp each: targets [un_t0, un_t1),
    // forest un_f (-1: a batch of izhikevich neurons), shared-memory slice at
    // word un_off of its CTA, gates [un_gt0, un_gt0 + un_ngt) and recorded
    // targets gr_*[un_r0 .. un_r1) (target indices local to the unit); CTA c
    // runs units [cta_u0[c], cta_u0[c+1])
    const int32_t *un_t0, *un_t1, *un_f, *un_off, *un_gt0, *un_ngt, *un_r0, *un_r1;
    const int32_t *cta_u0;
    // per unit: trace columns [un_r0, un_r1): gr_t is the node << 1 or the twig
    // place << 1 | 1 (of a point neuron the unit-local target), or -1 - the
    // unit-local gate slot of a gate's state; gr_col the column
    const int32_t *gr_t, *gr_col;
    // non-flat compartments ("slots") of forest units, [un_nf0[u], un_nf1[u]):
    // nf_rec, two 16-byte records a slot (forest_window: node | kSlot*, area,
    // C, 1/C; sum 1/(R C), block range, channel range, channel set), and nf_ts,
    // its spike threshold (NaN: no spike source) and source
    const int32_t *un_nf0, *un_nf1;
    const uint8_t *un_far;  // the unit's slice has no room for its blocks' records
    const float4 *nf_rec;
    const float2 *nf_ts;
    // channels of the slots, [un_ch0[u], un_ch1[u]): conductivity, reversal
    // potential, first gate (index in the unit's gates) and gate count
    // | instances << (3 + 5 * gate)
    const int32_t *un_ch0, *un_ch1;
    const float *nfc_g, *nfc_e;
    const int32_t *nfc_q, *nfc_i;
    // per gate, its slot | row of gate_tab << 10; gate_tab: the parameters of a
    // gate of a channel type, three 16-byte records (gate_next_p)
    const int32_t *gt_idx;
    const float4 *gate_tab;
    int32_t gate_warp;  // a unit's gates have a warp of their own (no gate takes V after the solve)
    // per input block: where its series begins in the unit's (forests: a series
    // of gp_stride a block, staged; point neurons: a block's first chunk's in Gp),
    // chunks, kind and reversal potential
    const int4 *bk_rec;
    int32_t *status;
    // forests whose cells may lose diagonal dominance: their elimination runs
    // in double precision (hines_window_f64, hines_forest_f64); dscr is
    // the per-step path's double scratch (two per target)
    const uint8_t *fo_f64;
    double *dscr;
    // gap-junction ends of each target [t_gap0[t], t_gap0[t+1]): the peer
    // (internal target), conductance (uS) and weight
    const int32_t *t_gap0, *gap_peer;
    const float *gap_g, *gap_w;
    // gradedSynapse ends of each target [t_gr0[t], t_gr0[t+1]): the peer,
    // EDEN_GRADED_PARAMS parameters, weight and state s
    const int32_t *t_gr0, *gr_peer;
    const float *gr_par, *gr_w;
    float *gr_s;
};

// The gap-junction current into target t at potential v, its peers read
// from the step's starting potentials vnow: each end contributes
// (g (V_peer - v)) w, as the reference sums a synapse's exposure times its
// weight (eden/Eden.cpp:3407-3422, 3708-3710); no conductance term.
__device__ __forceinline__ float gap_current(const DevModel &m, int t, float v, const float *vnow, bool init) {
    float i = 0.0f;
    for (int k = m.t_gap0[t]; k < m.t_gap0[t + 1]; k++) i += (m.gap_g[k] * (vnow[m.gap_peer[k]] - v)) * m.gap_w[k];
    // gradedSynapse ends (LEMS_CoreComponents.inc.xml:38-80, as the
    // reference's LEMS code steps it: the derived values and the current
    // from the step's starting state, s by forward Euler, the OnCondition
    // overriding; s = 0 in the initialisation steps).  Each end's state is
    // read and written by its own target's thread, once per step.
    for (int k = m.t_gr0[t]; k < m.t_gr0[t + 1]; k++) {
        const float *p = m.gr_par + (size_t)EDEN_GRADED_PARAMS * k;  // conductance, delta, k, Vth, erev
        const float s = m.gr_s[k];
        const float inf = 1.0f / (1.0f + expf((p[3] - vnow[m.gr_peer[k]]) / p[1]));
        const float tau = (1.0f - inf) / p[2];
        i += ((p[0] * s) * (p[4] - v)) * m.gr_w[k];
        float sn = 0.0f;
        if (!init) {
            sn = s + m.dt * ((1.0f - inf) > 1e-4f ? (inf - s) / tau : 0.0f);
            if ((1.0f - inf) < 1e-4f) sn = inf;
        }
        m.gr_s[k] = sn;
    }
    return i;
}

constexpr uint32_t kCepMask = 0x3ffu;
constexpr int kCepBeginShift = 10;
constexpr int kCepParentShift = 20;
constexpr uint32_t kCepNonFlat = 1u << 30;
constexpr uint32_t kCepTwig = 1u << 31;  // a twig's topmost compartment
constexpr uint32_t kTwigTop = 1u << 15;
// a slot's node, with
constexpr int32_t kSlotDone = 1 << 16;  // a cell of one compartment, in no pass: solved with its currents
// a warp pass over a forest: first compartment | compartments << 10 | most
// children of one of them << 16 | flags
constexpr int32_t kPassStart = 0x3ff;
constexpr int kPassCountShift = 10;
constexpr int kPassKidsShift = 16;
constexpr int32_t kPassFirst = 1 << 26;    // the first pass of its depth
constexpr int32_t kPassLast = 1 << 27;     // the last pass of its depth
constexpr int32_t kPassRoot = 1 << 28;     // depth 0
constexpr int32_t kPassNonFlat = 1 << 29;  // holds a non-flat compartment
constexpr int kPassPad = 32;               // lanes past a pass's end read, and do not use, up to this many records
constexpr int kGateRecs = 3;      // 16-byte records of a gate (gate_next_p)
constexpr int kSlotRecs = 2;      // 16-byte records of a non-flat compartment
constexpr int kGateExtWords = 9;  // a non-rates gate's kind and timeCourse / steadyState forms

// Shared-memory words of a unit's slice in the windowed kernel (a multiple of
// four, so that every slice starts 16-byte aligned).  A forest of n nodes (and
// one of zeros after them) and nw twig rows, what addresses refer to first:
// pairs, V and elimination factor per node; two words per twig place, pre-updated V and V; then the 16-byte
// records: one per node, one per twig place, two per non-flat compartment, one
// per input block, and the window's conductance series of each (gps words, its
// chunks summed); then pairs: threshold and source per non-flat
// compartment; then words: a twig place's addresses, V at the start of the step,
// the next and the last per non-flat compartment, four per channel of these, three per gate (its index
// word, its value in alternate steps), and the passes.  A batch of izhikevich
// neurons: V twice and 19 parameter / state words per neuron.
__host__ __device__ inline int twig_words(int n) { return (2 * n + 3) & ~3; }  // where the twigs' words start
__host__ __device__ inline int forest_words(int n, int nw, int nf, int nfch, int ngt, int np, int nblk, int gps,
                                            bool f64 = false, bool far = false) {
    // a double-precision forest adds its eliminated values, pivots and
    // factors in double (6 words per compartment, 8-byte aligned)
    const int w = twig_words(n + 1) + 64 * nw + 4 * (n + 1 + 32 * nw + kSlotRecs * nf + (far ? 0 : nblk)) + gps * nblk +
                  2 * nf + 32 * nw + 3 * nf + 4 * nfch + 3 * ngt + np + (f64 ? 6 * n + 2 : 0);
    return (w + 3) & ~3;
}
__host__ __device__ inline int izh_words(int n) { return ((2 + EDEN_POINT_PARAMS + 3) * n + 3) & ~3; }

// Per-window arguments: the window covers steps [step0, step0 + K); steps
// <= 0 are initialisation passes.  The previous window began at step
// step0 - Kprev; its triggers are the mask bits 1..Kprev-1 (replayed before
// step0) and bit Kprev (the trigger of step0 itself).
struct WindowArgs {
    double t0;     // simulation time of step0 (us), accumulated in double on the host
    int64_t step0;
    int32_t K, Kprev;
    int32_t par;   // which V buffer holds the state at step0
    int32_t wpar;  // window parity: which spike list this window fills
    int32_t ext0, ext1;  // the spikes of sources with no target logged in steps step0+1 .. step0+K
};

// Single-precision times (us) of the window's steps and of the previous
// window's, accumulated on the host in double from 0 as the reference
// accumulates its time (eden/Eden.cpp:11486, 11931).
struct WindowTimes {
    float tk[32];
    float tprev[32];
};

// ---------------------------------------------------------------------------
// spike compaction: warp ballot, one atomic per warp
// ---------------------------------------------------------------------------
// NaN: a spike with no interpolated crossing time
__device__ __forceinline__ double no_time() { return __longlong_as_double(0x7ff8000000000000ll); }

// Staging copies: one 4-byte word from global to shared memory without a
// register round trip (cp.async), so that all of a lane's staging loads are
// in flight together; stage_wait() waits for the lane's copies, and a
// __syncwarp() after it publishes them to the warp.
__device__ __forceinline__ void stage_word(void *smem_dst, const void *gmem_src) {
    unsigned s;
    asm("{\n .reg .u64 a;\n cvta.to.shared.u64 a, %1;\n cvt.u32.u64 %0, a;\n}" : "=r"(s) : "l"(smem_dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void stage_rec(void *smem_dst, const void *gmem_src) {  // 16 bytes, both sides aligned
    unsigned s;
    asm("{\n .reg .u64 a;\n cvta.to.shared.u64 a, %1;\n cvt.u32.u64 %0, a;\n}" : "=r"(s) : "l"(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void push_spike(const DevModel &m, bool spiked, int32_t src, int32_t log_step,
                                           int wpar, double tcross) {
    unsigned active = __activemask();
    unsigned ballot = __ballot_sync(active, spiked);
    if (ballot == 0) return;
    int lane = threadIdx.x & 31;
    int leader = __ffs(ballot) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&m.wspk_count[wpar], __popc(ballot));
    base = __shfl_sync(active, base, leader);
    if (spiked) {
        int rank = __popc(ballot & ((1u << lane) - 1));
        m.wspk_src[wpar][base + rank] = src;
        m.wspk_step[wpar][base + rank] = log_step;
        m.wspk_time[wpar][base + rank] = tcross;
    }
}

// The time (us) at which V crossed thr during a step that starts at time t
// (double) with potential v0 and ends with v1 (v0 < thr < v1), by linear
// interpolation in double.  A diagnostic beside the logged step: the
// reference quantises spike times to the step (eden/Eden.cpp:6247-6252).
__device__ __forceinline__ double crossing_time(double t, float dt, float v0, float v1, float thr) {
    return t + (double)dt * (((double)thr - (double)v0) / ((double)v1 - (double)v0));
}

// ---------------------------------------------------------------------------
// synapses and inputs
// ---------------------------------------------------------------------------
// Pending-spike rule for a trigger read at time t (eden/Eden.cpp:3646-3686):
// fire now if t <= t+delay < t+dt; keep it as the single pending spike only if
// the old one is already due (pend < t+dt) and earlier than the new one.
__device__ __forceinline__ bool trigger_arrival(float t, float dt, float delay, float &pend) {
    float fresh = t + delay;
    bool now = (t <= fresh && fresh < t + dt);
    if (pend < t + dt && pend < fresh) pend = fresh;
    return now;
}

// Replay triggers of the previous window (bits 1..Kprev-1) and return the
// trigger of the window's first step (bit Kprev).  Exact because every delay
// is at least Kprev * dt, so none of these spikes can fall due before step0.
__device__ __forceinline__ bool replay_mask(uint32_t mask, const WindowArgs &w, const float *tprev, float dt,
                                            float delay, float &pend) {
    for (uint32_t r = mask & ((1u << w.Kprev) - 1) & ~1u; r; r &= r - 1)
        trigger_arrival(tprev[__ffs(r) - 1], dt, delay, pend);
    return (mask >> w.Kprev) & 1u;
}

// ---------------------------------------------------------------------------
// input chunks: event-driven synapses with an aggregate state per chunk
// ---------------------------------------------------------------------------
// expOne and expTwo synapses are linear between events, so the weighted sum
// of a chunk's synapse states obeys the same update as one synapse (expOne
// G' = G - dt*G/tau, eden/Eden.cpp:3424-3466; expTwo A' = A - dt*A/tau_rise,
// B' = B - dt*B/tau_decay, LEMS_CoreComponents.inc.xml:145-180) and the
// chunk's conductance is its exposure (G, or gbase*(B - A)).  A synapse only
// costs work when it fires.  On that step the reference replaces the
// synapse's decay by the jump (G += gbase; A, B += weight_prop*wf), so the
// aggregate gets back the decay it applied to that synapse plus the jump,
// both times its weight.  For that the synapse keeps its own state as of its
// last event and the step of that event.

// A synapse's own state at the start of step s from its value just after its
// event at step `last`: the reference's per-step a - dt*(a/tau), in closed
// form a * f^n with f = 1 - dt/tau (used only for the decay its event replaces).
__device__ __forceinline__ float decayed(float a, float f, const float *fpow, int n) {
    if (n <= 0) return a;
    return a * (n < kPowLen ? fpow[n] : powf(f, (float)n));
}

// The contribution (dA, dB) of one synapse's event at step s to its chunk's
// aggregate, and the synapse's own state after it.  Roundings are written out:
// they do not depend on what the code around is contracted to.
template <int KIND, bool SYN = false>
__device__ __forceinline__ void input_event(const SynTypeDev &st, const float *pw, float dt, float w, int64_t s,
                                            float &a, float &b, int32_t &last, float &dA, float &dB, float js = 1.0f) {
    const int n = (int)(s - (int64_t)last) - 1;
    if (KIND == EDEN_SYN_EXPTWO) {
        // (js: a blockingPlasticSynapse's plasticity factor for this event, 1 for other connections)
        const float jump = SYN ? st.wf_w * js : st.wf_w;
        const float ai = decayed(a, st.f_rise, pw, n), bi = decayed(b, st.f_decay, pw + kPowLen, n);
        const float da = div_by_tau(ai, st.tau_rise, st.r_rise), db = div_by_tau(bi, st.tau_decay, st.r_decay);
        dA = __fmul_rn(w, SYN ? fmaf(st.wf_w, js, __fmul_rn(dt, da)) : fmaf(dt, da, jump));
        dB = __fmul_rn(w, SYN ? fmaf(st.wf_w, js, __fmul_rn(dt, db)) : fmaf(dt, db, jump));
        a = ai + jump;
        b = bi + jump;
    } else {
        const float gi = decayed(a, st.f_decay, pw + kPowLen, n);
        dA = __fmul_rn(w, fmaf(dt, div_by_tau(gi, st.tau_decay, st.r_decay), st.gbase));
        dB = 0.0f;
        a = gi + st.gbase;
    }
    last = (int32_t)s;
}

// An item's events in the window: the first in registers, the others (an item
// has more than one only where it fires again within the window) in its rows
// of the tiles.
struct ItemEvents {
    int n, j;
    float dA, dB;
};

// Adds an event at window step j, each in a step of its own.
template <int KIND>
__device__ __forceinline__ void put_event(float *rowA, float *rowB, ItemEvents &ev, int K, int j, float dA, float dB) {
    if (ev.n == 0) {
        ev.n = 1;
        ev.j = j;
        ev.dA = dA;
        ev.dB = dB;
        return;
    }
    if (ev.n == 1) {
        ev.n = 2;
        for (int q = 0; q < K; q++) {
            rowA[q] = 0.0f;
            if (KIND == EDEN_SYN_EXPTWO) rowB[q] = 0.0f;
        }
    }
    rowA[j] = __fadd_rn(rowA[j], dA);
    if (KIND == EDEN_SYN_EXPTWO) rowB[j] = __fadd_rn(rowB[j], dB);
}

// Poisson input `it` over the K steps of a window (poissonFiringSynapse,
// LEMS_CoreComponents.inc.xml:623-672): initialisation draws the first
// interval at each init step; afterwards the input fires its own synapse on
// the step its time since the last spike exceeds the interval (then restarts
// that time at 0 and draws the next interval), else adds dt to it.  When dt
// is a whole number of us and the times stay below 2^24 us, every such sum
// is exact, so the firing step is found directly instead of step by step.
__device__ __forceinline__ float pois_draw(const DevModel &m, int64_t it, int64_t step, int invocation) {
    return (-(1.0f / m.po_rate[it])) *
           logf(1.0f - randof(1.0f, (int64_t)m.po_seed[it], m.po_inst[it], step, m.po_rng[it] + invocation));
}

template <int KIND>
__device__ __forceinline__ void pois_fire(const DevModel &m, int64_t it, const SynTypeDev &st, const float *pw, int64_t s,
                                          int j, int K, float *rowA, float *rowB, ItemEvents &ev) {
    float a = m.po_a[it], b = KIND == EDEN_SYN_EXPTWO ? m.po_b[it] : 0.0f;
    int32_t last = m.po_last[it];
    float dA, dB;
    input_event<KIND>(st, pw, m.dt, m.po_w[it], s, a, b, last, dA, dB);
    m.po_a[it] = a;
    if (KIND == EDEN_SYN_EXPTWO) m.po_b[it] = b;
    m.po_last[it] = last;
    put_event<KIND>(rowA, rowB, ev, K, j, dA, dB);
}

template <int KIND>
__device__ __forceinline__ void pois_window(const DevModel &m, int64_t it, const WindowArgs &w, const SynTypeDev &st,
                                            const float *pw, float ts, float isi, float *rowA, float *rowB, ItemEvents &ev) {
    const float dt = m.dt;
    if (w.step0 <= 0) {
        for (int j = 0; j < w.K; j++) {
            ts = 0.0f;
            isi = pois_draw(m, it, w.step0 + j, 0);
        }
    } else if (m.pois_exact && isi < 0x1p23f) {
        // (one that cannot fire in the window has been dealt with: input_group)
        int j = 0;
        while (true) {
            // first step from j on whose time since the last spike exceeds isi
            int jn = 0;
            if (!(ts > isi)) {
                jn = (int)floorf((isi - ts) / dt) + 1;
                while (jn > 1 && ts + (float)(jn - 1) * dt > isi) jn--;
                while (!(ts + (float)jn * dt > isi)) jn++;
            }
            if (j + jn >= w.K) {
                ts = ts + (float)(w.K - j) * dt;
                break;
            }
            j += jn;
            isi = pois_draw(m, it, w.step0 + j, 1);
            pois_fire<KIND>(m, it, st, pw, w.step0 + j, j, w.K, rowA, rowB, ev);
            ts = 0.0f;
            j += 1;
            if (j >= w.K) break;
        }
    } else {
        for (int j = 0; j < w.K; j++) {
            if (ts > isi) {
                ts = 0.0f;
                isi = pois_draw(m, it, w.step0 + j, 1);
                pois_fire<KIND>(m, it, st, pw, w.step0 + j, j, w.K, rowA, rowB, ev);
            } else {
                ts = ts + dt * 1.0f;
            }
        }
    }
    m.po_ts[it] = ts;
    m.po_isi[it] = isi;
}

// Connection synapse `it` over the window: replay the previous window's
// triggers (replay_mask), then fire the single pending spike on the step
// whose interval holds it (eden/Eden.cpp:3646-3686).  That step is in this
// window for at most one pending spike: a trigger replaces the pending
// spike only once it is due, and a spike read at the first step lands at
// least K steps later.  The first step's trigger fires at once only for a
// delay below dt.
template <int KIND>
__device__ __forceinline__ void syn_window(const DevModel &m, int64_t it, const WindowArgs &w, const SynTypeDev &st,
                                           const float *pw, const float *tk, float pend, uint32_t mask, float *rowA, float *rowB,
                                           ItemEvents &ev) {
    // (input_group leaves out initialisation: no spikes reach a synapse in it)
    const float dt = m.dt;
    const float pend0 = pend;
    // a spike that is due, and so its state, is known before the replay: the
    // loads overlap
    const bool due = pend >= tk[0] && pend < tk[w.K - 1] + dt;
    float a = 0.0f, b = 0.0f, wt = 0.0f;
    int32_t last = 0;
    if (due) {
        a = m.sy_a[it];
        if (KIND == EDEN_SYN_EXPTWO) b = m.sy_b[it];
        last = m.sy_last[it];
        wt = m.sy_w[it];
    }
    bool trig = false;
    float delay = 0.0f;
    if (mask) {
        m.sy_mask[it] = 0;
        delay = m.sy_delay[it];
        trig = replay_mask(mask, w, tk + 32, dt, delay, pend);
    }
    // the first step j with pend < tk[j] + dt (these ends never fall), if its
    // start is not past pend
    int jf = -1;
    if (pend >= tk[0] && pend < tk[w.K - 1] + dt) {
        int j = 0, e = w.K - 1;
        while (j < e) {
            const int h = (j + e) >> 1;
            if (pend < tk[h] + dt) e = h;
            else j = h + 1;
        }
        if (tk[j] <= pend) jf = j;
    }
    bool now = false;
    if (trig) now = trigger_arrival(tk[0], dt, delay, pend);
    if (pend != pend0) m.sy_pend[it] = pend;
    if (jf < 0 && !now) return;
    if (!due) {
        a = m.sy_a[it];
        if (KIND == EDEN_SYN_EXPTWO) b = m.sy_b[it];
        last = m.sy_last[it];
        wt = m.sy_w[it];
    }
    float dA, dB;
    // a blockingPlasticSynapse's Tsodyks-Markram state (LEMS_CoreComponents.inc.xml:
    // 263-312): forward Euler from the last event, 1 - R and U - p shrinking
    // by their factor each step; the event's jump scaled by R U before the
    // event, which then sets R = R (1 - U), U = U + p (1 - U)
    const bool plastic = KIND == EDEN_SYN_EXPTWO && st.plastic;
    float R = plastic ? m.sy_R[it] : 1.0f, U = plastic ? m.sy_U[it] : 1.0f;
    auto factor = [&](int64_t s) {
        if (!plastic) return 1.0f;
        const float n = (float)(s - (int64_t)last - 1);
        R = 1.0f - (1.0f - R) * powf(st.f_rec, n);
        U = st.rel_p + (U - st.rel_p) * powf(st.f_fac, n);
        const float f = R * U;
        R = R * (1.0f - U);
        U = U + st.rel_p * (1.0f - U);
        if (st.f_fac == 1.0f) U = st.rel_p;
        return f;
    };
    if (now && jf != 0) {
        const float js = factor(w.step0);
        input_event<KIND, true>(st, pw, dt, wt, w.step0, a, b, last, dA, dB, js);
        put_event<KIND>(rowA, rowB, ev, w.K, 0, dA, dB);
    }
    if (jf >= 0) {
        const float js = factor(w.step0 + jf);
        input_event<KIND, true>(st, pw, dt, wt, w.step0 + jf, a, b, last, dA, dB, js);
        put_event<KIND>(rowA, rowB, ev, w.K, jf, dA, dB);
    }
    m.sy_a[it] = a;
    if (KIND == EDEN_SYN_EXPTWO) m.sy_b[it] = b;
    if (plastic) { m.sy_R[it] = R; m.sy_U[it] = U; }
    m.sy_last[it] = last;
}

// Input and target kinds the kernels handle: all of them in the library's
// own build; a build generated for one model (eden_codegen.cuh) defines only
// the model's, and the compiler drops the code of the others.
#ifndef EDEN_KIND_PULSE
#define EDEN_KIND_PULSE 1
#define EDEN_KIND_GATEFORMS 1
#define EDEN_KIND_CLAMP 1
#define EDEN_KIND_SINE 1
#define EDEN_KIND_RAMP 1
#define EDEN_KIND_POIS 1
#define EDEN_KIND_TIMED 1
#define EDEN_KIND_SYN 1
#define EDEN_KIND_EXPONE 1
#define EDEN_KIND_EXPTWO 1
#define EDEN_KIND_FOREST 1
#define EDEN_KIND_IZH 1
#define EDEN_KIND_GAP 1
#define EDEN_KIND_ALPHA 1
#define EDEN_KIND_CURRENT 1
#endif
#ifndef EDEN_GATE_WARPS
#define EDEN_GATE_WARPS 1  // units' gates may have a warp of their own (DevModel::gate_warp)
#endif
#ifndef EDEN_WIDE_INPUTS
#define EDEN_WIDE_INPUTS 0  // a model with many inputs (k_cells_t)
#endif

// A timedSynapticInput item over the window: its synapse fires in each
// listed step (eden/Eden.cpp:3759-3790, 3859-3871: the first step whose
// t + dt exceeds a listed time, the same step), which lowering has computed.
template <int KIND>
__device__ __forceinline__ void timed_window(const DevModel &m, int64_t it, const WindowArgs &w, const SynTypeDev &st,
                                             const float *pw, float *rowA, float *rowB, ItemEvents &ev) {
    int64_t c = m.tm_cur[it];
    const int64_t c1 = m.tm_off[it + 1];
    const int64_t end = w.step0 + w.K;
    if (c >= c1 || m.tm_step[c] >= end) return;
    float a = m.tm_a[it], b = KIND == EDEN_SYN_EXPTWO ? m.tm_b[it] : 0.0f;
    int32_t last = m.tm_last[it];
    for (; c < c1 && m.tm_step[c] < end; c++) {
        const int64_t s = m.tm_step[c];
        if (s < w.step0) continue;
        float dA, dB;
        input_event<KIND>(st, pw, m.dt, m.tm_w[it], s, a, b, last, dA, dB);
        put_event<KIND>(rowA, rowB, ev, w.K, (int)(s - w.step0), dA, dB);
    }
    m.tm_a[it] = a;
    if (KIND == EDEN_SYN_EXPTWO) m.tm_b[it] = b;
    m.tm_last[it] = last;
    m.tm_cur[it] = c;
}

// Per-warp accumulation tiles: row `lane` (stride acc_stride, odd so that
// both a row write and a column read are free of bank conflicts) holds the
// lane's terms for each step of the window.

// An alpha chunk's aggregate over the window (alphaSynapse: conductance g
// and rise state A; alphaCurrentSynapse: current I and J).  Per step the
// reference integrates A' = -A / tau and g' = (e A - g) / tau by forward
// Euler (LEMS_CoreComponents.inc.xml:85-142), so over the chunk's weighted
// sums A_{j+1} = f A_j + E_j and g_{j+1} = f g_j + c A_j, f = 1 - dt / tau,
// c = e dt / tau, E_j the events of step j (each a synapse's skipped decay
// plus its jump, as input_event gives them for the expOne-like rise state).
// In closed form g_j = f^j g_0 + c j f^(j-1) A_0 + c T_j with S_j the
// events' part of A_j (a scan over the lanes, as for the other kinds) and
// T_j = sum_{k<j} f^(j-1-k) S_k a second scan over S.  Lane j keeps the
// exposure g_j of step j for Gp.
__device__ __forceinline__ float alpha_chunk_window(const float *pd, const SynTypeDev &st, const WindowArgs &w,
                                                    bool events, float ea, float &A, float &B) {
    const int lane = threadIdx.x & 31;
    const float cc = st.c_alpha;
    const float jf = (float)lane;
    // the parts from the window's starting state
    float gj = lane < w.K ? B * pd[lane] + (lane > 0 ? cc * (jf * pd[lane - 1]) * A : 0.0f) : 0.0f;
    float Ak = A * pd[w.K], Bk = B * pd[w.K] + cc * ((float)w.K * pd[w.K - 1]) * A;
    if (events) {  // (ea of lane j: the chunk's events of step j)
        // S: inclusive scan of the events with factor f, then exclusive
        float va = lane < w.K ? ea : 0.0f;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, va, d);
            if (lane >= d) va = fmaf(pd[d], u, va);
        }
        float sj = __shfl_up_sync(0xffffffffu, va, 1);
        if (lane == 0) sj = 0.0f;
        // T: the same scan over S
        float vt = lane < w.K ? sj : 0.0f;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, vt, d);
            if (lane >= d) vt = fmaf(pd[d], u, vt);
        }
        float tj = __shfl_up_sync(0xffffffffu, vt, 1);
        if (lane == 0) tj = 0.0f;
        if (lane < w.K) gj += cc * tj;
        Ak += __shfl_sync(0xffffffffu, va, w.K - 1);
        Bk += cc * __shfl_sync(0xffffffffu, vt, w.K - 1);
    }
    if (w.step0 > 0) { A = Ak; B = Bk; }
    return gj;
}

// An item that may have an event in the window: its state, its chunk's place
// in the warp's group, and its place in the chunk (at = chunk * kChunkItems + item).
struct HotItem {
    float s0, s1;
    int at;
};
constexpr int kInputGroup = 16;                // chunks of a group, at most
constexpr int kHotItems = kChunkItems + 32;    // items listed before they are worked off, at most

// A chunk of pulses, clamps or generators (at most kChunkItems items of one
// input block) over the K steps of a window: lane l adds the current of items
// l, l + 32, ... to row l of the tile, and lane j sums column j in row order
// into the chunk's series in Gp.
__device__ __forceinline__ void pulse_chunk(const DevModel &m, int c, int32_t info, int64_t ck_i0, const WindowArgs &w,
                                            float *tileA, const float *tk) {
    const int lane = threadIdx.x & 31;
    const int kind = info & 3;
    const int n = info >> 8;
    const int stride = m.acc_stride;
    float *rowA = tileA + lane * stride;
    if (EDEN_KIND_CLAMP && kind == BK_PULSE && ((info >> 2) & 63) >= kClampA) {
        // voltage clamps (LEMS_CoreComponents.inc.xml:555-620): the target
        // of the phase each step's time is in (the last OnCondition that
        // holds assigns); half A sums weight * target / R, half B weight / R,
        // and the cell kernel takes A - V B at the step's starting V
        const bool half_a = ((info >> 2) & 63) == kClampA;
        for (int r = 0; lane + 32 * r < n; r++) {
            const float *p = m.cl_p + (size_t)(ck_i0 + lane + 32 * r) * kClampWords;
            const float del = p[0], dur = p[1], vb = p[2], vd = p[3], va = p[4], res = p[5], wt = p[6];
            for (int j = 0; j < w.K; j++) {
                const float tf = tk[j];
                const float tv = (tf > dur + del) ? va : (tf < del) ? vb : vd;
                const bool on = w.step0 + j > 0 && tv == tv;
                const float term = on ? __fmul_rn(half_a ? tv / res : 1.0f / res, wt) : 0.0f;
                rowA[j] = r > 0 ? rowA[j] + term : term;
            }
        }
        __syncwarp();
        if (lane < w.K) {
            const int rows = n < 32 ? n : 32;
            float tot = 0.0f;
            for (int r = 0; r < rows; r++) tot += tileA[r * stride + lane];
            m.Gp[(size_t)c * m.gp_stride + lane] = tot;
        }
        __syncwarp();
        return;
    }
    if ((EDEN_KIND_SINE || EDEN_KIND_RAMP) && kind == BK_PULSE && ((info >> 2) & 63) != 0) {
        // sineGenerator / rampGenerator (LEMS_CoreComponents.inc.xml:430-458,
        // 489-521): the value the OnConditions assign at the step's time,
        // which the reference's LEMS code exposes in the same step; OnStart's
        // in the initialisation passes
        const bool sine = ((info >> 2) & 63) == kPulseSine;
        for (int r = 0; lane + 32 * r < n; r++) {
            const float *p = m.wv_p + (size_t)(ck_i0 + lane + 32 * r) * kWaveWords;
            const float del = p[0], dur = p[1], a = p[2], b = p[3], cc = p[4], wt = p[5];
            for (int j = 0; j < w.K; j++) {
                const float tf = tk[j];
                const bool init = w.step0 + j <= 0;
                const bool off = tf < del || !(tf < dur + del);
                float i;
                if (sine) i = (init || off) ? 0.0f : (1.0f * a) * sinf(cc + ((2.0f * 3.14159265f) * (tf - del)) / b);
                else i = init ? cc : off ? 1.0f * cc : 1.0f * (a + ((b - a) * (tf - del)) / dur);
                const float term = __fmul_rn(i, wt);
                rowA[j] = r > 0 ? rowA[j] + term : term;
            }
        }
        __syncwarp();
        if (lane < w.K) {
            const int rows = n < 32 ? n : 32;
            float tot = 0.0f;
            for (int r = 0; r < rows; r++) tot += tileA[r * stride + lane];
            m.Gp[(size_t)c * m.gp_stride + lane] = tot;
        }
        __syncwarp();
        return;
    }
    if (EDEN_KIND_PULSE && kind == BK_PULSE && 2 * n <= w.K) {
        // a few pulses: lane j evaluates step j of each.  About 10 n
        // instructions, where the rows below take 6 K + 2 n: the line is where
        // these meet, on the safe side.  (30,011 cells of one pulse, 31 steps:
        // 22 us by rows, 11 by steps.)
        float tot = 0.0f;
        const float tf = tk[lane];
        for (int q = 0; q < n; q++) {
            const int64_t it = ck_i0 + q;
            const float st = m.pu_start[it], du = m.pu_dur[it], aw = __fmul_rn(m.pu_amp[it], m.pu_w[it]);
            tot = __fadd_rn(tot, (st <= tf && tf <= st + du) ? aw : 0.0f);
        }
        if (lane < w.K) m.Gp[(size_t)c * m.gp_stride + lane] = tot;
        return;
    }
    if (EDEN_KIND_PULSE && kind == BK_PULSE) {
        for (int r = 0; lane + 32 * r < n; r++) {
            const int64_t it = ck_i0 + lane + 32 * r;
            const float st = m.pu_start[it], du = m.pu_dur[it], aw = m.pu_amp[it] * m.pu_w[it];
            for (int j = 0; j < w.K; j++) {
                const float tf = tk[j];
                const float term = (st <= tf && tf <= st + du) ? aw : 0.0f;
                rowA[j] = r > 0 ? rowA[j] + term : term;
            }
        }
        __syncwarp();
        if (lane < w.K) {
            const int rows = n < 32 ? n : 32;
            float tot = 0.0f;
            for (int r = 0; r < rows; r++) tot += tileA[r * stride + lane];
            m.Gp[(size_t)c * m.gp_stride + lane] = tot;
        }
        __syncwarp();
        return;
    }
}

// The events of a listed item in the window.
__device__ __forceinline__ void item_window(const DevModel &m, int32_t info, int64_t it, const WindowArgs &w, const HotItem &h,
                                            const float *tk, float *rowA, float *rowB, ItemEvents &ev) {
    const int kind = info & 3, type = (info >> 2) & 63;
    const SynTypeDev &st = m.syn_types[type];
    const float *pw = m.syn_pow + (size_t)type * 2 * kPowLen;
    const bool two = EDEN_KIND_EXPTWO && (!EDEN_KIND_EXPONE || st.kind == EDEN_SYN_EXPTWO ||
                                          st.kind == EDEN_SYN_BLOCKING_PLASTIC);
    // only the input kinds the kernels are compiled for (all, or the model's)
    if (kind == BK_TIMED) {
        if (EDEN_KIND_TIMED) {
            if (two) { if (EDEN_KIND_EXPTWO) timed_window<EDEN_SYN_EXPTWO>(m, it, w, st, pw, rowA, rowB, ev); }
            else if (EDEN_KIND_EXPONE) timed_window<EDEN_SYN_EXPONE>(m, it, w, st, pw, rowA, rowB, ev);
        }
    } else if (kind == BK_POIS) {
        if (EDEN_KIND_POIS) {
            if (two) { if (EDEN_KIND_EXPTWO) pois_window<EDEN_SYN_EXPTWO>(m, it, w, st, pw, h.s0, h.s1, rowA, rowB, ev); }
            else if (EDEN_KIND_EXPONE) pois_window<EDEN_SYN_EXPONE>(m, it, w, st, pw, h.s0, h.s1, rowA, rowB, ev);
        }
    } else if (EDEN_KIND_SYN) {
        const uint32_t mask = __float_as_uint(h.s1);
        if (two) { if (EDEN_KIND_EXPTWO) syn_window<EDEN_SYN_EXPTWO>(m, it, w, st, pw, tk, h.s0, mask, rowA, rowB, ev); }
        else if (EDEN_KIND_EXPONE) syn_window<EDEN_SYN_EXPONE>(m, it, w, st, pw, tk, h.s0, mask, rowA, rowB, ev);
    }
}

// A synapse chunk's aggregate through the window from its state (A, B) and,
// in lane j, its events ea, eb of step j.  Returns, for lane j, the exposure of
// step j: the conductance before the step's update, as the reference exposes
// it.  With one step's decay factor f, X_j = f^j X_0 + sum_{i<j} f^(j-1-i) e_i,
// the sums by a scan over the lanes; without events in closed form, A f^j,
// from the factors' powers (syn_pow).
__device__ __forceinline__ float chunk_series(const DevModel &m, int type, const WindowArgs &w, bool events, float ea,
                                              float eb, float &A, float &B) {
    const int lane = threadIdx.x & 31;
    const SynTypeDev &st = m.syn_types[type];
    const float *pr = m.syn_pow + (size_t)type * 2 * kPowLen, *pd = pr + kPowLen;
    if (EDEN_KIND_ALPHA && (st.kind == EDEN_SYN_ALPHA || st.kind == EDEN_SYN_ALPHA_CURRENT))
        return alpha_chunk_window(pd, st, w, events, ea, A, B);
    const bool two = EDEN_KIND_EXPTWO && (!EDEN_KIND_EXPONE || st.kind == EDEN_SYN_EXPTWO ||
                                          st.kind == EDEN_SYN_BLOCKING_PLASTIC);
    float gj = 0.0f;
    if (!events) {
        if (lane < w.K) gj = two ? st.gbase * (B * pd[lane] - A * pr[lane]) : A * pd[lane];
        if (w.step0 > 0) {
            A = A * (two ? pr[w.K] : pd[w.K]);
            B = two ? B * pd[w.K] : B;
        }
        return gj;
    }
    const float *pa = two ? pr : pd;
    float va = lane < w.K ? ea : 0.0f, vb = lane < w.K ? eb : 0.0f;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float ua = __shfl_up_sync(0xffffffffu, va, d);
        if (lane >= d) va = fmaf(pa[d], ua, va);
        if (two) {
            const float ub = __shfl_up_sync(0xffffffffu, vb, d);
            if (lane >= d) vb = fmaf(pd[d], ub, vb);
        }
    }
    // lane j: sums of the events before step j
    float sa = __shfl_up_sync(0xffffffffu, va, 1), sb = __shfl_up_sync(0xffffffffu, vb, 1);
    if (lane == 0) { sa = 0.0f; sb = 0.0f; }
    if (lane < w.K) {
        const float Aj = A * pa[lane] + sa, Bj = B * pd[lane] + sb;
        gj = two ? st.gbase * (Bj - Aj) : Aj;
    }
    const float ta = __shfl_sync(0xffffffffu, va, w.K - 1), tb = __shfl_sync(0xffffffffu, vb, w.K - 1);
    A = A * pa[w.K] + ta;
    B = two ? B * pd[w.K] + tb : B;
    return gj;
}

// A group of nc <= kInputGroup consecutive chunks, c0 on, over the K steps of a
// window, by one warp.  Few of a chunk's synapses and Poisson inputs have an
// event in a window, and the code of one that has is long; run chunk by chunk
// it was the whole of the kernel's time with most of its lanes idle.  So the
// warp looks at every item's state first and lists those that may have an
// event, over all chunks of the group; then each lane works off one of the
// list (100,000 neurons of 100 synapses, windows of 10 steps: 484 us by items
// of a lane one after another, 186 with a list per chunk, 123 per group of 16;
// instruction issue bounds it, 62 % of its peak, memory at 27 %); then the chunks are finished in order, lane j summing the events of
// step j -- over the items that share a lane of the chunk (l, l + 32, ...),
// then over these lanes in order -- and taking the aggregate through the window.
__device__ __forceinline__ void input_group(const DevModel &m, int c0, int nc, const WindowArgs &w, float *tileA,
                                            float *tileB, HotItem *list, const float *tk) {
    const int lane = threadIdx.x & 31;
    const int stride = m.acc_stride;
    float *rowA = tileA + lane * stride, *rowB = tileB + lane * stride;
    // lane i: chunk i of the group
    int32_t info_l = 0;
    int64_t i0_l = 0;
    float A_l = 0.0f, B_l = 0.0f;
    if (lane < nc) {
        info_l = m.ck_info[c0 + lane];
        i0_l = m.ck_i0[c0 + lane];
        A_l = m.ck_a[c0 + lane];
        B_l = m.ck_b[c0 + lane];
    }
    const float t_end = tk[w.K - 1] + m.dt;
    int count = 0, done = 0;  // listed items; chunks finished
#pragma unroll 1
    for (int i = 0;; i++) {
        const int32_t info = __shfl_sync(0xffffffffu, info_l, i);
        const int64_t ck_i0 = __shfl_sync(0xffffffffu, i0_l, i);
        const int kind = info & 3, n = info >> 8;
        if (i < nc && kind == BK_PULSE) {
            pulse_chunk(m, c0 + i, info, ck_i0, w, tileA, tk);
            continue;
        }
        if (i == nc || count + n > kHotItems) {
            // work off the list, and finish the chunks before i
            __syncwarp();
            int b = -32, last = -1;  // the list's batch, and the chunk of its last item
            unsigned rows = 0, more = 0;
            ItemEvents ev{0, 0, 0.0f, 0.0f};
            int at = -1;
#pragma unroll 1
            for (int q = done; q < i; q++) {
                const int32_t info_q = __shfl_sync(0xffffffffu, info_l, q);
                if ((info_q & 3) == BK_PULSE) continue;
                float ea = 0.0f, eb = 0.0f;  // lane j: the chunk's events of step j
                float sa = 0.0f, sb = 0.0f;  // of the items of one lane of the chunk
                int of = -1;
                bool events = false;
#pragma unroll 1
                while (true) {
                    const unsigned mine = rows & __ballot_sync(0xffffffffu, (at >> 7) == q);
                    events |= mine != 0;
                    for (unsigned r = mine; r; r &= r - 1) {
                        const int e = __ffs(r) - 1;
                        const int l = __shfl_sync(0xffffffffu, at, e) & 31, j = __shfl_sync(0xffffffffu, ev.j, e);
                        float dA = __shfl_sync(0xffffffffu, ev.dA, e);
                        float dB = EDEN_KIND_EXPTWO ? __shfl_sync(0xffffffffu, ev.dB, e) : 0.0f;
                        if (lane != j) {
                            dA = dB = 0.0f;
                            if (((more >> e) & 1u) && lane < w.K) {
                                dA = tileA[e * stride + lane];
                                if (EDEN_KIND_EXPTWO) dB = tileB[e * stride + lane];
                            }
                        }
                        if (l != of) {
                            ea += sa;
                            eb += sb;
                            sa = sb = 0.0f;
                            of = l;
                        }
                        sa = __fadd_rn(sa, dA);
                        if (EDEN_KIND_EXPTWO) sb = __fadd_rn(sb, dB);
                    }
                    if (b + 32 >= count || last > q) break;
                    // the next batch: this one's items are all of chunks up to q
                    __syncwarp();
                    b += 32;
                    ev = ItemEvents{0, 0, 0.0f, 0.0f};
                    HotItem h{0.0f, 0.0f, -1};
                    if (b + lane < count) h = list[b + lane];
                    at = h.at;
                    const int32_t info_e = __shfl_sync(0xffffffffu, info_l, (at >> 7) & 31);
                    const int64_t it = __shfl_sync(0xffffffffu, i0_l, (at >> 7) & 31) + (at & (kChunkItems - 1));
                    if (at >= 0) item_window(m, info_e, it, w, h, tk, rowA, rowB, ev);
                    rows = __ballot_sync(0xffffffffu, ev.n > 0);
                    more = __ballot_sync(0xffffffffu, ev.n > 1);
                    last = __shfl_sync(0xffffffffu, at, min(31, count - 1 - b)) >> 7;
                    __syncwarp();
                }
                ea += sa;
                eb += sb;
                float A = __shfl_sync(0xffffffffu, A_l, q), B = __shfl_sync(0xffffffffu, B_l, q);
                const float gj = chunk_series(m, (info_q >> 2) & 63, w, events, ea, eb, A, B);
                if (lane == q) { A_l = A; B_l = B; }
                if (lane < w.K) m.Gp[(size_t)(c0 + q) * m.gp_stride + lane] = gj;
            }
            __syncwarp();
            if (i == nc) break;
            done = i;
            count = 0;
        }
        // list the chunk's items that may have an event, lane by lane and a
        // lane's in order
        float s0v[kChunkItems / 32], s1v[kChunkItems / 32];
        unsigned hot[kChunkItems / 32];
#pragma unroll
        for (int r = 0; r < kChunkItems / 32; r++) {
            s0v[r] = 0.0f; s1v[r] = 0.0f;
            if (lane + 32 * r < n) {
                const int64_t it = ck_i0 + lane + 32 * r;
                if (kind == BK_POIS) { s0v[r] = m.po_ts[it]; s1v[r] = m.po_isi[it]; }
                else if (kind == BK_SYN) { s0v[r] = m.sy_pend[it]; s1v[r] = __uint_as_float(m.sy_mask[it]); }
            }
        }
        int at = count;
#pragma unroll
        for (int r = 0; r < kChunkItems / 32; r++) {
            hot[r] = 0;
            if (32 * r >= n) continue;
            bool h = false;
            if (lane + 32 * r < n) {
                const int64_t it = ck_i0 + lane + 32 * r;
                if (kind == BK_TIMED) {
                    const int64_t cur = m.tm_cur[it];
                    h = EDEN_KIND_TIMED && cur < m.tm_off[it + 1] && m.tm_step[cur] < w.step0 + w.K;
                } else if (kind == BK_POIS) {
                    // (exact sums: no firing in the window when even its last step's
                    // time since the spike stays within the interval)
                    h = !(w.step0 > 0 && m.pois_exact && s1v[r] < 0x1p23f && s0v[r] + (float)(w.K - 1) * m.dt <= s1v[r]);
                    if (!h) m.po_ts[it] = s0v[r] + (float)w.K * m.dt;
                } else {
                    // (no spikes reach a synapse during initialisation)
                    h = w.step0 > 0 && (__float_as_uint(s1v[r]) != 0 || (s0v[r] >= tk[0] && s0v[r] < t_end));
                }
            }
            hot[r] = __ballot_sync(0xffffffffu, h);
            count += __popc(hot[r]);
            at += __popc(hot[r] & ((1u << lane) - 1));
        }
#pragma unroll
        for (int r = 0; r < kChunkItems / 32; r++)
            if ((hot[r] >> lane) & 1u) list[at++] = HotItem{s0v[r], s1v[r], i * kChunkItems + lane + 32 * r};
    }
    if (lane < nc && (info_l & 3) != BK_PULSE) {
        m.ck_a[c0 + lane] = A_l;
        m.ck_b[c0 + lane] = B_l;
    }
    __syncwarp();
}

// Currents into target t at step j of the window from its input blocks:
// pulses add current; conductance blocks add g*(erev - v) and g, inputs
// first, then synapses, as eden/Eden.cpp:6057-6060 orders them.  BK_K and
// BK_E are the blocks' kinds and reversal potentials, BC0 their chunk ranges;
// Gpk is Gp at the step.
__device__ __forceinline__ void block_currents(const float *Gpk, int stride, int b0, int b1, const int32_t *BK_K,
                                               const float *BK_E, const int32_t *BC0, float v, float &Iin, float &Gin,
                                               float &Isyn, float &Gsyn,
                                               const float2 *BK_B = nullptr) {
    Iin = 0.0f; Gin = 0.0f; Isyn = 0.0f; Gsyn = 0.0f;
    for (int bk = b0; bk < b1; bk++) {
        float g = 0.0f;
        for (int c = BC0[bk]; c < BC0[bk + 1]; c++) g += Gpk[(size_t)c * stride];
        // a blockingPlasticSynapse's voltage block (voltageConcDepBlockMechanism,
        // LEMS_CoreComponents.inc.xml:231-245) scales its conductance, so both
        // the current and the conductance term (per-step kernels only)
        if (BK_B && (BK_K[bk] & BK_BLOCK)) g = (1.0f / (1.0f + BK_B[bk].x * expf(-1.0f * (v / BK_B[bk].y)))) * g;
        const int kind = BK_K[bk] & BK_KIND_MASK;
        const bool current = EDEN_KIND_CURRENT && (BK_K[bk] & BK_CURRENT);
        if (kind == BK_PULSE) {
            Iin += g;
        } else if (EDEN_KIND_CLAMP && kind == BK_CLAMPV) {
            Iin -= v * g;
        } else if (kind == BK_POIS || kind == BK_TIMED) {
            if (current) {
                Iin += g;
            } else {
                Iin += g * (BK_E[bk] - v);
                Gin += g;
            }
        } else if (current) {
            Isyn += g;
        } else {
            Isyn += g * (BK_E[bk] - v);
            Gsyn += g;
        }
    }
}

// Four steps' values of a block of nc chunks, summed in their order: p, the first
// chunk's, the others gps words apart.  Loads go ahead of the chain of additions.
__device__ __forceinline__ float4 sum_chunks(const float *p, int gps, int nc) {
    auto at = [&](int c) { return *reinterpret_cast<const float4 *>(p + (size_t)c * gps); };
    auto add = [](float4 &g, const float4 &x) { g.x += x.x; g.y += x.y; g.z += x.z; g.w += x.w; };
    float4 g = at(0);
    int c = 1;
#pragma unroll 1
    for (; c + 8 <= nc; c += 8) {
        float4 x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = at(c + j);
#pragma unroll
        for (int j = 0; j < 8; j++) add(g, x[j]);
    }
#pragma unroll 1
    for (; c < nc; c++) add(g, at(c));
    return g;
}

// block_currents from the unit's block records (where the block's series begins
// in the unit's, kind, reversal potential); Gk: the unit's series at the step
__device__ __forceinline__ void block_currents_rec(const float *Gk, const int4 *BK, int b0, int b1, float v, float &Iin,
                                                   float &Gin, float &Isyn, float &Gsyn) {
    Iin = 0.0f; Gin = 0.0f; Isyn = 0.0f; Gsyn = 0.0f;
#pragma unroll 1
    for (int bk = b0; bk < b1; bk++) {
        const int4 r = BK[bk];
        const float g = Gk[r.x];
        const int kind = r.z & BK_KIND_MASK;
        if (EDEN_KIND_CLAMP && kind == BK_CLAMPV) {
            Iin -= v * g;
            continue;
        }
        // a current is its value times 1, and adds no conductance; the sum a block
        // is not part of stays as it is, whatever the potential: no branches
        const bool current = kind == BK_PULSE || (EDEN_KIND_CURRENT && (r.z & BK_CURRENT)), syn = kind == BK_SYN;
        const float sum = fmaf(g, current ? 1.0f : __int_as_float(r.w) - v, syn ? Isyn : Iin);
        Iin = syn ? Iin : sum;
        Isyn = syn ? sum : Isyn;
        Gin += current || syn ? 0.0f : g;
        Gsyn += current || !syn ? 0.0f : g;
    }
}

__device__ __forceinline__ float gate_next(const ChanTypeDev &ct, int gi, bool init, float dt, float v, float qo) {
    if (EDEN_KIND_GATEFORMS && ct.gk[gi] != EDEN_GATE_RATES)
        return gate_general(ct.gk[gi], ct.fk[gi], ct.fr[gi], ct.fm[gi], ct.fs[gi], ct.rk[gi], ct.rr[gi], ct.rm[gi],
                            ct.rs[gi], ct.tk[gi], ct.tr[gi], ct.tm[gi], ct.ts[gi], ct.ik[gi], ct.ir[gi], ct.im[gi],
                            ct.is[gi], ct.q10[gi], init, dt, v, qo);
    const float alpha = rate_value(ct.fk[gi], ct.fr[gi], ct.fm[gi], ct.fs[gi], v);
    const float beta = rate_value(ct.rk[gi], ct.rr[gi], ct.rm[gi], ct.rs[gi], v);
    return gate_relax(alpha, beta, ct.q10[gi], init, dt, qo);
}

// The same from the three parameter records of the windowed kernel's table:
//   a  forward form | reverse form << 4 | row << 8, forward rate, midpoint, scale
//   b  0, reverse rate, midpoint, scale
//   c  q10 factor, known_reciprocal of the forward and of the reverse scale, 0
// A gate of another kind than gateHHrates carries 1 + its row of `ext` (kind,
// timeCourse form and its three values, steadyState form and its three values)
// in the first word above the forms.
// An instantaneous gate keeps the steady state at the compartment's
// potential after the step (`vnew`), which is what the next step's currents
// read as its value.
// The value is gate_next's, operation by operation, with three of its seven
// divisions known in advance (by the scales, and by alpha + beta once
// 1 / (alpha + beta) is there) and, of the two that the rate forms may take,
// only those that some lane's forms do.
__device__ __forceinline__ float gate_next_p(const float4 &a, const float4 &b, const float4 &c, const float *ext,
                                             bool init, float dt, float v, float vnew, float qo) {
    const int w0 = __float_as_int(a.x);
    if (EDEN_KIND_GATEFORMS && (w0 >> 8) != 0) {
        const float *X = ext + (size_t)((w0 >> 8) - 1) * kGateExtWords;
        const int gk = __float_as_int(X[0]);
        return gate_general(gk, w0 & 15, a.y, a.z, a.w, (w0 >> 4) & 15, b.y, b.z, b.w, __float_as_int(X[1]), X[2], X[3],
                            X[4], __float_as_int(X[5]), X[6], X[7], X[8], c.x, init, dt,
                            gk == EDEN_GATE_INSTANTANEOUS ? vnew : v, qo);
    }
    const int fk = w0 & 15, rk = (w0 >> 4) & 15;
    const bool fq = fk != EDEN_RATE_EXP, rq = rk != EDEN_RATE_EXP;
    const bool fs = fk == EDEN_RATE_SIGMOID, rs = rk == EDEN_RATE_SIGMOID;
    const float xf = div_known(v - a.z, a.w, c.y), xr = div_known(v - b.z, b.w, c.z);
    const float ef = expf(fq ? -xf : xf), er = expf(rq ? -xr : xr);
    const float fn = fs ? a.y : xf, fd = fs ? 1.0f + ef : 1.0f - ef;
    const float rn = rs ? b.y : xr, rd = rs ? 1.0f + er : 1.0f - er;
    // one quotient covers a gate with one exponential form
    const float q1 = (fq ? fn : rn) / (fq ? fd : rd);
    const float q2 = fq && rq ? rn / rd : q1;
    const float alpha = !fq ? a.y * ef : fs ? q1 : a.y * ((v == a.z) ? 1.0f : q1);
    const float beta = !rq ? b.y * er : rs ? q2 : b.y * ((v == b.z) ? 1.0f : q2);
    const float sum = alpha + beta;
    const float tau = 1.0f / sum;
    const float inf = div_known(alpha, sum, (sum >= 0x1p-60f && sum < 0x1p60f) ? tau : 0.0f);
    return gate_relax_ti(tau, inf, c.x, init, dt, qo);
}

// ---------------------------------------------------------------------------
// point neurons
// ---------------------------------------------------------------------------
// One step of a point neuron from its now state (V v, states u and s) with
// external current iext (synaptic then input currents), following the LEMS
// semantics the reference generates code from (eden/Eden.cpp:2832-2994):
// every state is integrated by forward Euler from the now state, then, where
// an OnCondition holds on the now state, its assignments (from now values)
// override; the initialisation passes apply OnStart.  Parameters are read as
// p[f * ps].  Returns whether the neuron spiked.
__device__ __forceinline__ bool point_update(int kind, const float *p, int ps, bool init, float t, float dt,
                                             float v, float iext, float &u, float &s, float &vn) {
#define PP(f) p[(f) * ps]
    bool spike = false;
    switch (kind) {
    case EDEN_POINT_IAF_TAU:
    case EDEN_POINT_IAF_TAU_REF: {
        // iafTauCell / iafTauRefCell: v' = (leakReversal - v) / tau, no synaptic input
        const bool ref = kind == EDEN_POINT_IAF_TAU_REF;
        if (init) {
            vn = PP(0);
            if (ref) s = t - PP(4);
            break;
        }
        const bool active = !ref || t > s + PP(4);
        const float rate = active ? (PP(0) - v) / PP(1) : 0.0f;
        vn = v + dt * rate;
        if (v > PP(2) && active) {
            if (ref) s = t;
            vn = PP(3);
            spike = true;
        }
        break;
    }
    case EDEN_POINT_IAF:
    case EDEN_POINT_IAF_REF: {
        // iafCell / iafRefCell: iMemb = leakConductance (leakReversal - v) + iSyn, v' = iMemb / C
        const bool ref = kind == EDEN_POINT_IAF_REF;
        if (init) {
            vn = PP(2);
            if (ref) s = t - PP(5);
            break;
        }
        const float imemb = PP(1) * (PP(2) - v) + iext;
        const bool active = !ref || t > s + PP(5);
        const float rate = active ? imemb / PP(0) : 0.0f;
        vn = v + dt * rate;
        if (v > PP(3) && active) {
            if (ref) s = t;
            vn = PP(4);
            spike = true;
        }
        break;
    }
    case EDEN_POINT_FN: {
        // fitzHughNagumoCell: V' = ((V - V^3 / 3) - W + I) / s, W' = 0.08 (V + 0.7 - 0.8 W) / s
        const float SEC = 1.0e6f;
        if (init) {
            vn = v;
            break;
        }
        const float w = u;
        vn = v + dt * ((((v - powf(v, 3.0f) / 3.0f) - w) + PP(0)) / SEC);
        u = w + dt * ((0.08f * ((v + 0.7f) - 0.8f * w)) / SEC);
        break;
    }
    case EDEN_POINT_IZH_DL: {
        // izhikevichCell: v' = (0.04 v^2 / mV + 5 v + (140 - U + I) mV) / ms,
        // U' = a (b v / mV - U) / ms; above thresh v = c mV, U += d
        const float MV = 1.0f, MS = 1000.0f;
        if (init) {
            vn = PP(0);
            u = (PP(0) * PP(3)) / MV;
            break;
        }
        const float uu = u;
        const float dv = ((0.04f * ((v * v) / MV) + 5.0f * v) + ((140.0f - uu) + iext) * MV) / MS;
        const float du = (PP(2) * ((PP(3) * v) / MV - uu)) / MS;
        vn = v + dt * dv;
        u = uu + dt * du;
        if (v > PP(1)) {
            vn = PP(4) * MV;
            u = uu + PP(5);
            spike = true;
        }
        break;
    }
    case EDEN_POINT_ADEX: {
        // adExIaFCell: iMemb = -gL (v - EL) + gL delT exp((v - VT) / delT) - w + iSyn,
        // v' = iMemb / C outside the refractory period, w' = (a (v - EL) - w) / tauw
        if (init) {
            vn = PP(2);
            u = 0.0f;
            s = t - PP(8);
            break;
        }
        const float w = u;
        const float imemb = (-1.0f * PP(1)) * (v - PP(2)) + (PP(1) * PP(6)) * expf((v - PP(3)) / PP(6)) - w + iext;
        const bool active = t > s + PP(8);
        const float rate = active ? imemb / PP(0) : 0.0f;
        vn = v + dt * rate;
        u = w + dt * ((PP(9) * (v - PP(2)) - w) / PP(7));
        if (v > PP(4) && active) {
            s = t;
            vn = PP(5);
            u = w + PP(10);
            spike = true;
        }
        break;
    }
    default: {
        // izhikevich2007Cell (LEMS_CoreComponents.inc.xml:1140-1187)
        const float uu = u, vr = PP(3);
        const float imemb = ((PP(2) * (v - vr)) * 1e-3f) * (v - PP(4)) + iext - uu;
        if (init) {
            vn = PP(1);
            u = 0.0f;
        } else {
            vn = v + dt * (imemb / PP(0));
            const float du = (PP(6) * ((PP(7) * (v - vr)) - uu)) * 1e-3f;
            u = uu + dt * du * 1e3f;
            if (v > PP(5)) {
                vn = PP(8);
                u = uu + PP(9);
                spike = true;
            }
        }
    }
    }
#undef PP
    return spike;
}

// ---------------------------------------------------------------------------
// targets
// ---------------------------------------------------------------------------
// One target for one step: the trajectory sample, then either the channels +
// voltage pre-update of a compartment (eden/Eden.cpp:5013-6107), writing the
// pre-updated V to *x and the Hines diagonal to *d, or the izhikevich2007
// update (LEMS_CoreComponents.inc.xml:1140-1185), writing v' to *x.
// Axial current into compartment t for the forward-Euler cable update
// (eden/Eden.cpp:4969-4990): (V_adj - V) / R summed over the neighbours in
// ascending compartment order -- the parent, then the children, which the
// breadth-first numbering keeps in that order -- from the potentials at the
// start of the step; R is the axial resistance of the edge's child end.
__device__ __forceinline__ float axial_current(const DevModel &m, int t, float v, const float *vin) {
    float I = 0.0f;
    const int p = m.c_parent[t];
    if (p >= 0) I += (vin[p] - v) / m.c_rax[t];
    for (int k = m.c_kb[t]; k < m.c_cend[t]; k++) I += (vin[k] - v) / m.c_rax[k];
    return I;
}

__device__ __forceinline__ void target_step(const DevModel &m, int t, bool init, int64_t step, float tnow, float v,
                                            float Iin, float Gin, float Isyn, float Gsyn, float *x, float *d, int wpar,
                                            float Iax = 0.0f) {
    if (!init) {
        for (int k = m.t_trace0[t]; k < m.t_trace0[t + 1]; k++) {
            int64_t row = (step - 1) % m.trace_cap;
            const int gq = m.trace_gate[k];
            m.trace_buf[row * m.n_trace + m.trace_col[k]] = gq < 0 ? v : m.gate[gq];
        }
    }
    int iz = m.t_izh[t];
    if (iz < 0) {
        float A = m.c_area[t];
        float Ich = 0.0f, Gch = 0.0f;
        for (int ch = m.c_chan0[t]; ch < m.c_chan0[t + 1]; ch++) {
            const ChanTypeDev &ct = m.chan_types[m.ch_type[ch]];
            float fopen = 1.0f;
            float *q = m.gate + m.ch_gate0[ch];
            for (int g = 0; g < ct.n_gates; g++) {
                const float qo = q[g];
                const float qn = gate_next(ct, g, init, m.dt, v, qo);
                q[g] = qn;
                // an instantaneous gate's value is its steady state at this V
                const float qf = (EDEN_KIND_GATEFORMS && ct.gk[g] == EDEN_GATE_INSTANTANEOUS) ? qn : qo;
                for (int r = 0; r < ct.inst[g]; r++) fopen = fopen * qf;
            }
            float gs = m.ch_gbase[ch] * fopen;
            Ich += (gs * (m.ch_erev[ch] - v) * 1e-5f) * A;
            Gch += (gs * 1e-5f) * A;
        }
        float I = Ich + Iin + Isyn;
        float G = Gch + Gin + Gsyn;
        float C = m.c_cm[t];
        *d = 1.0f * (G / C) + m.c_inv_rc[t];
        // backward Euler: the pre-updated V the Hines solve starts from;
        // forward Euler: V_next (eden/Eden.cpp:6092-6094)
        *x = init ? v : m.fwd_euler ? v + (m.dt * (I + Iax)) / C : v + (m.dt * (I + (v * G))) / C;
    } else {
        float u = m.iz_u[iz], sv = m.iz_s[iz], vn;
        const bool spike = point_update(m.iz_kind[iz], m.iz_p + iz, m.n_izh, init, tnow, m.dt, v, Isyn + Iin, u, sv, vn);
        *x = vn;
        m.iz_u[iz] = u;
        m.iz_s[iz] = sv;
        int src = m.t_src[t];
        push_spike(m, spike && src >= 0, src, (int32_t)(step + 1), wpar, no_time());
    }
}

// ---------------------------------------------------------------------------
// cable solve
// ---------------------------------------------------------------------------
// A lane's spike source of a forest: its target, its threshold.
struct ForestSource {
    int t = -1, src = -1;
    float thr = 0.0f;
};
__device__ __forceinline__ ForestSource forest_source(const DevModel &m, int q, int end) {
    ForestSource s;
    if (q < end) {
        s.t = m.fo_s[q];
        s.src = m.t_src[s.t];
        s.thr = m.src_thr[s.src];
    }
    return s;
}

// The threshold test V < thr < V_next of forest f's spike sources (eden/Eden.cpp:
// 6247-6252), s the lane's first; `base`: the target at index 0 of Vin and X.
__device__ __forceinline__ void forest_spikes(const DevModel &m, int f, ForestSource s, int64_t step, double tstep,
                                              const float *X, const float *Vin, int base, int wpar) {
    const int lane = threadIdx.x & 31, end = m.fo_s0[f + 1];
    for (int q = m.fo_s0[f]; q < end; q += 32) {
        if (q > m.fo_s0[f]) s = forest_source(m, q + lane, end);
        bool spk = false;
        double tc = 0.0;
        if (s.src >= 0) {
            const float v = Vin[s.t - base], vn = X[s.t - base];
            spk = v < s.thr && s.thr < vn;
            if (spk) tc = crossing_time(tstep, m.dt, v, vn, s.thr);
        }
        push_spike(m, spk, s.src, (int32_t)(step + 1), wpar, tc);
    }
}

// Backward-Euler Hines solve of one forest by one warp (eden/Eden.cpp:6114-6225).
// Arrays may live in shared or global memory and share one index space:
// D (diagonal, in), X (the pre-updated V, solved in place), U, L
// (off-diagonals), CE (end of each node's child range), P (parent), and LV
// (the forest's depth boundaries, nlev + 1 entries).  Depths are
// processed deepest first; each node pulls its children's elimination terms
// in increasing child order, the same sequence of operations as the
// reference's depth-first post-order, and keeps the reciprocal of its final
// pivot.  Back-substitution then runs root-first.
__device__ __forceinline__ void hines_forest(const DevModel &m, bool init, float *D, float *X, const float *U,
                                             const float *L, const int32_t *CE, const int32_t *P, const int32_t *LV,
                                             int nlev) {
    const int lane = threadIdx.x & 31;
    const int c0 = LV[0], c1 = LV[nlev];
    if (!init && c1 > c0) {
        const float dt = m.dt;
        for (int c = c0 + lane; c < c1; c += 32) D[c] = 1.0f + D[c] * dt;
        __syncwarp();
        for (int lev = nlev - 1; lev >= 0; lev--) {
            const int j0 = LV[lev], j1 = LV[lev + 1];
            for (int j = j0 + lane; j < j1; j += 32) {
                const int kb = (j == j0) ? j1 : CE[j - 1];
                const int ke = CE[j];
                float dj = D[j];
                if (ke > kb) {
                    float xj = X[j];
                    for (int i = kb; i < ke; i++) {
                        const float ratio = L[i] * D[i];  // D[i] holds the child's reciprocal pivot
                        dj -= ratio * U[i];
                        xj -= ratio * X[i];
                    }
                    X[j] = xj;
                }
                D[j] = pivot(dj);
            }
            __syncwarp();
        }
        for (int r = LV[0] + lane; r < LV[1]; r += 32) X[r] = X[r] * D[r];
        __syncwarp();
        for (int lev = 1; lev < nlev; lev++) {
            for (int i = LV[lev] + lane; i < LV[lev + 1]; i += 32) X[i] = (X[i] - U[i] * X[P[i]]) * D[i];
            __syncwarp();
        }
    }
}

// The same solve in double precision for a forest whose rows may lose
// diagonal dominance (the per-step path; D and X are global, XD and DD the
// forest's double scratch): the pre-updated V and diagonal terms stay the
// single-precision values the step computed, the elimination and the
// back-substitution carry doubles, and X receives V_next rounded once.
__device__ __forceinline__ void hines_forest_f64(const DevModel &m, bool init, const float *D, float *X, const float *U,
                                                 const float *L, const int32_t *CE, const int32_t *P, const int32_t *LV,
                                                 int nlev, double *XD, double *DD) {
    const int lane = threadIdx.x & 31;
    const int c0 = LV[0], c1 = LV[nlev];
    if (!init && c1 > c0) {
        const double dt = m.dt;
        for (int c = c0 + lane; c < c1; c += 32) {
            DD[c] = 1.0 + (double)D[c] * dt;
            XD[c] = X[c];
        }
        __syncwarp();
        for (int lev = nlev - 1; lev >= 0; lev--) {
            const int j0 = LV[lev], j1 = LV[lev + 1];
            for (int j = j0 + lane; j < j1; j += 32) {
                const int kb = (j == j0) ? j1 : CE[j - 1];
                const int ke = CE[j];
                double dj = DD[j], xj = XD[j];
                for (int i = kb; i < ke; i++) {
                    const double ratio = (double)L[i] * DD[i];  // DD[i]: the child's reciprocal pivot
                    dj -= ratio * (double)U[i];
                    xj -= ratio * XD[i];
                }
                XD[j] = xj;
                DD[j] = 1.0 / dj;
            }
            __syncwarp();
        }
        for (int r = LV[0] + lane; r < LV[1]; r += 32) XD[r] = XD[r] * DD[r];
        __syncwarp();
        for (int lev = 1; lev < nlev; lev++) {
            for (int i = LV[lev] + lane; i < LV[lev + 1]; i += 32) XD[i] = (XD[i] - (double)U[i] * XD[P[i]]) * DD[i];
            __syncwarp();
        }
        for (int c = c0 + lane; c < c1; c += 32) X[c] = (float)XD[c];
        __syncwarp();
    }
}

// Backward-Euler Hines solve of one forest by one warp for the windowed path,
// on the unit's shared-memory slice S (eden/Eden.cpp:6114-6225).  Flat
// compartments keep the reciprocal pivot and the elimination factor L / pivot
// computed once, because their diagonals never change.  Every compartment takes
// its children in increasing order, as the reference's post-order visits them.
//
// Twigs first: each lane walks its own flat subtrees up, every compartment into
// its parent's word, the topmost into its node's; their pre-update (V + the
// increment) was written with their V (TX; TV holds V).  Then the nodes, depth
// by depth (XR: V and the elimination factor; CN: the record): from the last
// pass (PS) to the roots, which it finishes, a flat node's pre-update (V +=
// CN.x) folded in, a non-flat node's pivot rebuilt from 1 + dt (G/C + sum
// 1/(RC)) (CN.z on entry, XR.x its pre-updated V) and its factor from its L;
// then from pass `p1`, the first below the roots, the back-substitution; then
// the twigs down again.
//
// A unit's step is a chain, and what it costs is the instructions a warp spends
// along it.  A depth costs 26 + 16 of them and 5 more for each child of its
// largest family, for as few compartments as there are; a twig row costs 22 for
// up to 32.  So subtrees up to a size chosen per forest become twigs
// (build_and_upload weighs the two), and depths remain only above them.  In a
// pass every lane takes as many children as the pass's largest family (an absent
// one is node n, all zeros), so the loop over them does not diverge, and lanes
// past its end load what they do not use.  A lane's places are 32 words apart: no bank
// conflicts, and no synchronisation within a twig.
// (Products are fused explicitly, as the compiler fuses them in a plain loop.)
__device__ __forceinline__ void hines_window(float dt, float *S, float2 *XR, float4 *CN, const int32_t *PS, int np,
                                             int p1, int n, float *TX, float *TV, const float4 *TR, const uint32_t *TA,
                                             int nw) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i = lane; i < 32 * nw; i += 32) {
        const uint32_t a = TA[i];
        const float x = TX[i];
        float *to = S + (a & (kTwigTop - 1));
        const float y = fmaf(-TR[i].w, x, *to);
        *to = (a & kTwigTop) ? x : y;
    }
    if (nw > 0) __syncwarp();
#pragma unroll 1
    for (int p = np - 1; p >= 0; p--) {
        const int32_t d = PS[p];
        const int j = (d & kPassStart) + lane, kids = (d >> kPassKidsShift) & 0x3ff;
        const bool on = lane < ((d >> kPassCountShift) & 63);
        const float4 c = CN[j];
        float x = XR[j].x;
        const uint32_t cep = __float_as_uint(c.w);
        int kb = (int)((cep >> kCepBeginShift) & kCepMask);
        const int ke = on ? kb + (int)(cep & kCepMask) : 0;
        // (a twig's topmost compartment among them has done its part)
        if (d & kPassNonFlat) {
            const bool nonflat = (cep & kCepNonFlat) != 0;
            float dj = c.z;
            x += (cep & (kCepNonFlat | kCepTwig)) ? 0.0f : c.x;
#pragma unroll 1
            for (int i = 0; i < kids; i++, kb++) {
                const int q = kb < ke ? kb : n;
                const float2 k = XR[q];
                dj = fmaf(-k.y, CN[q].y, dj);
                x = fmaf(-k.y, k.x, x);
            }
            const float inv = nonflat ? pivot(dj) : c.z;
            if (d & kPassRoot) x = x * inv;
            if (on && nonflat) { CN[j].z = inv; XR[j].y = c.x * inv; }
        } else {
            x += (cep & kCepTwig) ? 0.0f : c.x;
#pragma unroll 1
            for (int i = 0; i < kids; i += 2, kb += 2) {
                const float2 k = XR[kb < ke ? kb : n], l = XR[kb + 1 < ke ? kb + 1 : n];
                x = fmaf(-k.y, k.x, x);
                x = fmaf(-l.y, l.x, x);
            }
        }
        if (on) XR[j].x = x;
        if (d & kPassFirst) __syncwarp();
    }
#pragma unroll 1
    for (int p = p1; p < np; p++) {
        const int32_t d = PS[p];
        const int j = (d & kPassStart) + lane;
        const bool on = lane < ((d >> kPassCountShift) & 63);
        const float4 c = CN[j];
        const float x = XR[j].x;
        const int q = on ? (int)((__float_as_uint(c.w) >> kCepParentShift) & kCepMask) : 0;
        const float v = fmaf(-c.y, XR[q].x, x) * c.z;
        if (on) XR[j].x = v;
        if (d & kPassLast) __syncwarp();
    }
#pragma unroll 1
    for (int i = 32 * (nw - 1) + lane; i >= 0; i -= 32) {
        const float4 c = TR[i];
        const float v = fmaf(-c.y, S[TA[i] >> 16], TX[i]) * c.z;
        TV[i] = v;
        TX[i] = __fadd_rn(v, c.x);
    }
}

// hines_window in double precision, for a forest whose rows may lose
// diagonal dominance: every compartment's pivot is rebuilt each step from
// its diagonal term (CN.z: G/C + sum 1/(RC), constant for the flat ones), and
// the elimination and back-substitution carry doubles in
// XD / PVD / RTD; XR.x receives V_next rounded once.  A flat compartment's
// pre-update is its CN.x, and every compartment's L comes from Lg (global,
// indexed like the forest).  The operations are hines_window's, in its order.
__device__ __forceinline__ void hines_window_f64(float dt, float2 *XR, const float4 *CN, const float *Lg,
                                                 const int32_t *PS, int np, int n, double *XD, double *PVD,
                                                 double *RTD) {
    const int lane = threadIdx.x & 31;
    const double dtd = dt;
    for (int p = np - 1; p >= 0; p--) {
        const int32_t d = PS[p];
        const int j = (d & kPassStart) + lane;
        if (lane < ((d >> kPassCountShift) & 63)) {
            const float4 c = CN[j];
            const uint32_t cep = __float_as_uint(c.w);
            const int kb = (int)((cep >> kCepBeginShift) & kCepMask), ke = kb + (int)(cep & kCepMask);
            const float kc = (cep & kCepNonFlat) ? 0.0f : c.x;
            double xj = (double)XR[j].x + (double)kc;
            double dj = 1.0 + (double)c.z * dtd;
            for (int i = kb; i < ke; i++) {
                const double r = RTD[i];
                dj -= r * (double)CN[i].y;
                xj -= r * XD[i];
            }
            const double inv = 1.0 / dj;
            PVD[j] = inv;
            RTD[j] = (double)Lg[j] * inv;
            XD[j] = (d & kPassRoot) ? xj * inv : xj;
        }
        if (d & kPassFirst) __syncwarp();
    }
    for (int p = 0; p < np; p++) {
        const int32_t d = PS[p];
        const int i = (d & kPassStart) + lane;
        if (!(d & kPassRoot) && lane < ((d >> kPassCountShift) & 63)) {
            const float4 c = CN[i];
            const int q = (int)((__float_as_uint(c.w) >> kCepParentShift) & kCepMask);
            XD[i] = (XD[i] - (double)c.y * XD[q]) * PVD[i];
        }
        if (d & kPassLast) __syncwarp();
    }
    for (int i = lane; i < n; i += 32) XR[i].x = (float)XD[i];
    __syncwarp();
}

}  // namespace eden
