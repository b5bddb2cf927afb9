// Transport kernels.  One consumer kernel per event queue (the reference's
// ten stacks, CUDA_EGS.h:362-367), fed by a source kernel that turns
// phase-space records into primaries on the device.
//
// Persistent form: the photon and electron consumers keep every lane busy by
// refilling idle lanes from the queue with one warp-aggregated atomic per
// refill (persistent threads with regeneration), and a one-thread planner
// kernel decides the next wave and sets the CUDA-graph loop condition, so a
// whole run is a single graph launch with no host round trip.
// Plain form: the reference's structure -- each thread pops its own particle
// with a global atomic, and the host synchronises and reads the queue counters
// back after every launch (CUDA_EGS.cu:226-365, 498-799).
#pragma once
#include "dev_run.cuh"
#include "../../include/gegs.h"     // gegs_probe_state

// Step budgets in the tail of a run (fewer than batch / GX_TAIL_DIV particles
// in flight and no history left to inject) are GX_TAIL_SHIFT doublings larger.
// On the CT 5-field plan (40M-history runs, 24M in flight) this takes 180
// waves down to about 105 and the run 1.8 % faster; shifts of 3 to 6 and
// thresholds from batch/16 to batch/4096 measured the same within 0.2 %.
#ifndef GX_TAIL_SHIFT
#define GX_TAIL_SHIFT 2u
#endif
#ifndef GX_TAIL_DIV
#define GX_TAIL_DIV 256u
#endif

// Steps one particle may take inside one launch of the plain form before it is
// dropped and GX_ERR_STEP_BUDGET is raised: against a particle that stops making
// progress. (In waves such a particle goes from budget to budget until the run's
// waves are used up, and the drain kernel hands it to the waves.)
#define GX_STEP_BUDGET 4000000u

// The last of the `blocks` that took part in draining a queue resets it.
__device__ __forceinline__ void consumer_done(const DevCtx &C, uint32_t blocks, int q, int q2 = -1, uint32_t *finished = nullptr)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        uint32_t prev = atomicAdd(&C.q.done[q], 1u);
        if (prev == blocks - 1) {
            if (C.q.peak) {
                atomicMax(&C.q.peak[q], *((volatile uint32_t *)&C.q.count[q]));
                if (q2 >= 0) atomicMax(&C.q.peak[q2], *((volatile uint32_t *)&C.q.count[q2]));
            }
            C.q.count[q] = 0;
            C.q.head[q] = 0;
            C.q.done[q] = 0;
            if (q2 >= 0) C.q.count[q2] = 0;
            __threadfence();
            if (finished) atomicAdd(finished, 1u);
        }
    }
}

// Queue a particle of a transport for a stage, or for the next wave as it
// stands (electrons with their step state), into `qid`.
template <bool ELEC>
__device__ __forceinline__ void queue_particle(const DevCtx &C, int qid, Part &p, const Rng &r, const EState &s)
{
    rng_store(r, p);
    if (qid < GX_NSTAGE) {
        p.status = (uint8_t)qid;
        trace_event(C, 0u, qid, p);
    }
    const uint32_t i = queue_place(C.q.count, qid);
    if (i < C.q.cap[qid]) {
        store_part(&C.q.buf[qid][i], p);
        if (ELEC && qid >= GX_Q_ECONT) C.q.estate[qid - GX_Q_ECONT][i] = pack_estate(s);
    } else {
        atomicOr(C.err, GX_ERR_QUEUE_FULL);
    }
}

__device__ __forceinline__ void block_stat_add(const DevCtx &C, int slot, unsigned long long v)
{
    // warp reduction then one atomic per warp
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&C.stats[slot], v);
}

// ---- source ------------------------------------------------------------------
__global__ void k_source(const __grid_constant__ DevCtx C, const SchedState *st)
{
    timeline_mark(C, TL_SOURCE, false);
    unsigned long long h0 = st->h0, h1 = st->h1;
    unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long h = h0 + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; h < h1; h += stride) {
        Part p;
        if (!make_primary(C, h, p)) { atomicOr(C.err, GX_ERR_SOURCE); continue; }
        push(C, p.charge == 0 ? ST_PHOTON : ST_ELECTRON, p);
    }
    if (C.timeline) {
        __syncthreads();
        timeline_mark(C, TL_SOURCE, true);
    }
}

// A warp goes back to its queue once this many of its lanes are idle. A refill
// runs at the speed of its loads (the claim, the record, the region: one after
// another some 2000 cycles) with only the new lanes active, so a refill per
// lane that ends holds the others up at nearly every step. Slab, 5M histories:
// 85.1 ms at 1, 78.1 at 4, 75.5 at 8, 75.8 at 16; CT head 5-field plan, 16M:
// 275.8, 263.4, 258.6, 256.1.
#ifndef GX_REFILL_IDLE
#define GX_REFILL_IDLE 12u
#endif

// ---- persistent consumers with warp regeneration ---------------------------
// A consumer drains the continuation queue of the previous wave (indices
// [0, n_cont)) and then its stage queue ([n_cont, n)) through one shared head
// counter `hq`; idle lanes of a warp are refilled with one atomic.
template <int Q, bool ELEC>
__device__ __forceinline__ bool refill(const DevCtx &C, int hq, uint32_t n_cont, uint32_t n, int qc, bool &exhausted,
                                       bool active, Part &p, Rng &r, EState &s, Vox &vx, float &gle, unsigned long long &taken)
{
    const uint32_t lane = threadIdx.x & 31u;
    unsigned need = __ballot_sync(0xffffffffu, !active);
    uint32_t cnt = __popc(need);
    if (cnt == 0u || exhausted || cnt < GX_REFILL_IDLE) return active;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&C.q.head[hq], cnt);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base + cnt >= n) exhausted = true;
    if (!active) {
        uint32_t idx = base + __popc(need & ((1u << lane) - 1u));
        if (idx < n) {
            const bool cont = idx < n_cont;
            p = load_part(cont ? &C.q.buf[qc][idx] : &C.q.buf[Q][idx - n_cont]);
            rng_load(r, p);
            vx = C.reg[p.region];
            if (!ELEC) gle = gx_log(p.e);
            if (cont) {
                if (ELEC) unpack_estate(C.q.estate[qc - GX_Q_ECONT][idx], s);
            } else {
                if (ELEC) estate_init(s);
                trace_event(C, 1u, Q, p);
                taken++;
            }
            return true;
        }
    }
    return active;
}

// Register caps of the transport consumers (minimum resident 256-thread
// blocks per SM); measured best on the CT 5-field plan.
#ifndef GX_PHOTON_MIN_BLOCKS
#define GX_PHOTON_MIN_BLOCKS 4
#endif
// the near-boundary electron passes: 128 registers (1.2 % faster than 80 on the
// CT head 5-field plan, 16M histories, 1.6 % at 1M)
#ifndef GX_ELECTRON_MIN_BLOCKS
#define GX_ELECTRON_MIN_BLOCKS 2
#endif
// the phantom electrons: 64 registers. Its step spills there (224 bytes of
// stores, 428 of loads; 160 and 224 at 80 registers), yet the fourth block per
// SM hides as much of the loads' latency: the same time at 3 blocks, 3.5 %
// slower at 5 (48 registers)
#ifndef GX_EPHANTOM_MIN_BLOCKS
#define GX_EPHANTOM_MIN_BLOCKS 4
#endif
// the jaws photons (and their long tracks) and the MLC photons hold a second
// step, the one the warp shares (share_steps): 80 and 128 registers. With 48 and
// 80 that step's registers spill in the other one too: CT of 161x117x87, 3
// fields, 3M histories (two plans) 148.4 ms against 136.0, CT head 5-field plan,
// 16M (two) 518.4 against 509.9; without the shared step 156.4 and 512.6.
#ifndef GX_PJAWS_MIN_BLOCKS
#define GX_PJAWS_MIN_BLOCKS 3
#endif
#ifndef GX_PMLC_MIN_BLOCKS
#define GX_PMLC_MIN_BLOCKS 2
#endif
// the first pass of the jaws and MLC electrons, without howfar: 80 registers
// (3 blocks; CT head 5-field plan, 16M histories: 1.8 % faster than 48, with
// fewer warps waiting for instructions, and 0.3 % than 64)
#ifndef GX_EHEAD_MIN_BLOCKS
#define GX_EHEAD_MIN_BLOCKS 3
#endif

// Transport consumer for photons (ELEC false) or electrons of one geometry
// class G. The three class kernels of a particle type run concurrently; the
// phantom kernel also takes the stage queue's new particles. A particle
// outside the class, or one whose step budget for this launch is spent, is
// re-queued with its state for the next wave (into its class's continuation
// queue), so the tally does not depend on where a track is split.
//
// Electrons in the jaws and the MLC run in two passes. The first hands every
// step that needs a boundary search (howfar, the costliest routine of these
// classes, wanted by few lanes of a warp at a time) to its class's
// near-boundary queue, as the step stood at its start; the second (NEAR) runs
// those steps again, whole, and carries its particles on while their steps
// need howfar, so that its warps search boundaries with most lanes at once. A
// step that does not goes back, as it stood, to the first pass of the next
// wave. For jaws photons the second form (NEAR) is the long-track kernel:
// it takes the photons still going when the photon phase ended and steps them
// beside the electron phase.
template <bool ELEC, int G, bool NEAR = false>
__device__ __forceinline__ void transport_consumer(const DevCtx &C)
{
    constexpr int Q = ELEC ? ST_ELECTRON : ST_PHOTON;
    constexpr int base = ELEC ? GX_Q_ECONT : GX_Q_PCONT;
    constexpr int cls = G - GX_GEOM_JAWS;                // 0 jaws, 1 MLC, 2 phantom
    constexpr bool FIRST = (G == GX_GEOM_PHANTOM);        // takes the new particles
    constexpr bool DEFER = ELEC && (G == GX_GEOM_JAWS || G == GX_GEOM_MLC) && !NEAR;
    // the photon jaws kernel's second form (NEAR): the long tracks, beside the electron phase
    constexpr bool LONG = !ELEC && G == GX_GEOM_JAWS && NEAR;
    constexpr int tl = LONG ? TL_PLONG : NEAR ? TL_ENEAR : (ELEC ? TL_ELECTRON : TL_PHOTON) + cls;
    const uint32_t par = *C.wave & 1u;
    const int qc_in = LONG ? GX_Q_PLONG : NEAR ? GX_Q_ENEAR + cls : base + 2 * cls + (int)par;
    const int qc_out = base + 2 * cls + (int)(par ^ 1u);
    const int hq = FIRST ? Q : qc_in;
    const uint32_t n_cont = queue_len(C, qc_in);
    const uint32_t n = n_cont + (FIRST ? queue_len(C, Q) : 0u);
    // the last kernel of each photon branch but the jaws (MLC, phantom), and of
    // each electron branch (jaws and MLC near-boundary passes, phantom)
    uint32_t *fin = (!ELEC && G != GX_GEOM_JAWS) ? C.photon_done
                  : (ELEC && (NEAR || G == GX_GEOM_PHANTOM)) ? C.electron_done : nullptr;
    // Only the blocks that have work take part: a launch of 888 blocks that found
    // nothing and counted themselves off took 10 to 25 us, now 3 to 4.
    const uint32_t blocks = min(gridDim.x, n / blockDim.x + (n % blockDim.x ? 1u : 0u));
    if (blockIdx.x >= blocks) {
        if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0 && fin) atomicAdd(fin, 1u);
        return;
    }
    timeline_mark(C, tl, false);
    if (!ELEC) stage_photon_tables(C);
    // Per-class budgets (measured on the CT 5-field plan): electrons take 2x their
    // budget in the phantom. A jaws photon takes a handful of steps, except the
    // rare one that runs almost parallel to a jaw face in tens of thousands of
    // tiny steps, and an MLC photon a few, except one in a million that goes
    // along a leaf gap for thousands, at 8 us each. Past its budget such a photon
    // keeps stepping while the other transport branches of the wave still run (up
    // to 64 budgets), so that its long track advances with the bulk of the work
    // and neither holds a wave up nor is left for the run's tail. The jaws take
    // 8x the photons' budget before that; the MLC 1x (8x: CT head 5-field plan,
    // 1M histories, one such photon added 2 ms to each of nine waves). Only when
    // the phase's kernels run concurrently (C.overlap).
    constexpr bool JAWS_PHOTON = !ELEC && G == GX_GEOM_JAWS;
    constexpr bool EXTEND = !ELEC && cls < 2;
    const uint32_t budget = (ELEC ? (cls < 2 ? C.electron_budget : 2u * C.electron_budget)
                                  : (JAWS_PHOTON || (cls < 2 && !C.overlap) ? 8u : 1u) * C.photon_budget)
                            << *C.budget_shift;
    // How many of the other branches have to be done for that to end: of both
    // particle types in the pipelined form, else of the photons; the MLC's own is
    // not among them, and it does not wait for the jaws photons, which wait for it.
    const volatile uint32_t *others_done = LONG ? C.electron_done : C.photon_done;
    const volatile uint32_t *others_done2 = C.electron_done;
    const uint32_t others = LONG ? 3u : (C.pipelined ? 5u : 2u) - (JAWS_PHOTON ? 0u : 1u);
    // in the serial persistent form, a jaws photon still going when the photon
    // phase ends moves on to the long-track kernel, which runs beside the
    // electron phase the same way
    const int q_limit = (JAWS_PHOTON && !LONG && C.overlap && !C.pipelined) ? GX_Q_PLONG : qc_out;
    Part p;
    Rng r;
    EState s;
    Vox vx;
    float gle = 0.0f;
    bool active = false, exhausted = false;
    unsigned long long taken = 0, steps = 0;
    uint32_t nst = 0;
    for (;;) {
        const bool was = active;
        active = refill<Q, ELEC>(C, hq, n_cont, n, qc_in, exhausted, active, p, r, s, vx, gle, taken);
        if (active && !was) nst = 0;
        if (!__any_sync(0xffffffffu, active)) break;
        // (compiled for these kernels alone, and the condition below spelt out twice:
        // a lambda for it made the phantom's kernels 7 % slower)
        if constexpr (EXTEND) if (exhausted) {
            const unsigned act = __ballot_sync(0xffffffffu, active);
            if (__popc(act) <= GX_SHARE_LANES) {
                int tq = -1, code = STEP_ON;
                const bool stepping = active && in_geom_class<G>(p);
                if (active && !stepping) tq = base + 2 * (geom_class_of(p.module) - GX_GEOM_JAWS) + (int)(par ^ 1u);
                if (stepping) {
                    steps++;
                    rng_window(C, r);
                }
                share_steps<G>(C, __ballot_sync(0xffffffffu, stepping), p, r, vx, gle, code, tq);
                if (stepping) {
                    if (code == STEP_DONE) active = false;
                    else if (code == STEP_ON && ++nst >= budget &&
                             (!EXTEND || !C.overlap || nst >= 64u * budget ||
                            (((nst - budget) & 15u) == 0u &&
                             *others_done + (C.pipelined && !LONG ? *others_done2 : 0u) >= others)))
                        tq = q_limit;
                }
                if (tq >= 0) {
                    queue_particle<false>(C, tq, p, r, s);
                    active = false;
                }
                continue;
            }
        }
        if (active) {
            int tq = -1;                          // the queue the particle leaves for
            if (!in_geom_class<G>(p)) tq = base + 2 * (geom_class_of(p.module) - GX_GEOM_JAWS) + (int)(par ^ 1u);
            else {
                steps++;
                rng_window(C, r);
                const uint32_t ctr0 = r.ctr;
                const EState s0 = s;
                const int code = ELEC ? electron_step<G, DEFER, ELEC && NEAR>(C, p, r, s, vx, tq) : photon_step<G, true>(C, p, r, vx, gle, tq);
                if (code == STEP_DONE) active = false;
                else if ((DEFER && code == STEP_NEAR) || (ELEC && NEAR && code == STEP_FAR)) {
                    // needs howfar (to the near-boundary pass) or, in that pass, does
                    // not (back to the first pass of the next wave): as it stood
                    r.ctr = ctr0;
                    s = s0;
                    tq = DEFER ? GX_Q_ENEAR + cls : qc_out;
                    steps--;
                } else if (code == STEP_ON && ++nst >= budget &&
                           (!EXTEND || !C.overlap || nst >= 64u * budget ||
                            (((nst - budget) & 15u) == 0u &&
                             *others_done + (C.pipelined && !LONG ? *others_done2 : 0u) >= others)))
                    tq = ELEC ? qc_out : q_limit;
            }
            if (tq >= 0) {
                queue_particle<ELEC>(C, tq, p, r, s);
                active = false;
            }
        }
    }
    if (FIRST) block_stat_add(C, Q, taken);
    block_stat_add(C, GX_NSTAGE + (ELEC ? 1 : 0), steps);
    // steps in the jaws and the MLC (slots 12-15; the phantom's are the rest)
    if (cls < 2) block_stat_add(C, GX_NSTAGE + 2 + 2 * (ELEC ? 1 : 0) + cls, steps);
    if (FIRST) consumer_done(C, blocks, Q, qc_in, fin);
    else consumer_done(C, blocks, qc_in, -1, fin);
    timeline_mark(C, tl, true);
}

__global__ void __launch_bounds__(256, GX_PJAWS_MIN_BLOCKS) k_photon_jaws(const __grid_constant__ DevCtx C)
{
    transport_consumer<false, GX_GEOM_JAWS>(C);
}

__global__ void __launch_bounds__(256, GX_PJAWS_MIN_BLOCKS) k_photon_jaws_long(const __grid_constant__ DevCtx C)
{
    transport_consumer<false, GX_GEOM_JAWS, true>(C);
}

__global__ void __launch_bounds__(256, GX_PMLC_MIN_BLOCKS) k_photon_mlc(const __grid_constant__ DevCtx C)
{
    transport_consumer<false, GX_GEOM_MLC>(C);
}

__global__ void __launch_bounds__(256, GX_PHOTON_MIN_BLOCKS) k_photon(const __grid_constant__ DevCtx C)
{
    transport_consumer<false, GX_GEOM_PHANTOM>(C);
}

__global__ void __launch_bounds__(256, GX_EHEAD_MIN_BLOCKS) k_electron_jaws(const __grid_constant__ DevCtx C)
{
    transport_consumer<true, GX_GEOM_JAWS>(C);
}

__global__ void __launch_bounds__(256, GX_EHEAD_MIN_BLOCKS) k_electron_mlc(const __grid_constant__ DevCtx C)
{
    transport_consumer<true, GX_GEOM_MLC>(C);
}

__global__ void __launch_bounds__(256, GX_ELECTRON_MIN_BLOCKS) k_electron_jaws_near(const __grid_constant__ DevCtx C)
{
    transport_consumer<true, GX_GEOM_JAWS, true>(C);
}

__global__ void __launch_bounds__(256, GX_ELECTRON_MIN_BLOCKS) k_electron_mlc_near(const __grid_constant__ DevCtx C)
{
    transport_consumer<true, GX_GEOM_MLC, true>(C);
}

__global__ void __launch_bounds__(256, GX_EPHANTOM_MIN_BLOCKS) k_electron(const __grid_constant__ DevCtx C)
{
    transport_consumer<true, GX_GEOM_PHANTOM>(C);
}

template <int Q>
__global__ void __launch_bounds__(256) k_interact(const __grid_constant__ DevCtx C)
{
    constexpr int tl = Q < ST_ELECTRON ? TL_PINT + (Q - ST_COMPTON) : TL_EINT + (Q - ST_MOLLER);
    const uint32_t n = queue_len(C, Q);
    const uint32_t blocks = min(gridDim.x, n / blockDim.x + (n % blockDim.x ? 1u : 0u));
    if (blockIdx.x >= blocks) return;
    timeline_mark(C, tl, false);
    unsigned long long taken = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        Part p = load_part(&C.q.buf[Q][i]);
        Rng r;
        rng_load(r, p);
        rng_window(C, r);
        trace_event(C, 1u, Q, p);
        run_interaction<Q>(C, p, r);
        taken += counted<Q>(p);
    }
    block_stat_add(C, Q, taken);
    consumer_done(C, blocks, Q);
    timeline_mark(C, tl, true);
}

// ---- plain form: per-thread pops, one stage per launch ---------------------
template <int Q>
__global__ void __launch_bounds__(256) k_plain(const __grid_constant__ DevCtx C)
{
    const uint32_t n = queue_len(C, Q);
    unsigned long long taken = 0, steps = 0;
    for (;;) {
        uint32_t idx = atomicAdd(&C.q.head[Q], 1u);
        if (idx >= n) break;
        Part p = load_part(&C.q.buf[Q][idx]);
        Rng r;
        rng_load(r, p);
        trace_event(C, 1u, Q, p);
        taken += counted<Q>(p);
        if (Q == ST_PHOTON || Q == ST_ELECTRON) {
            EState s;
            estate_init(s);
            Vox vx = C.reg[p.region];
            const float gle = gx_log(p.e);
            uint32_t nst = 0;
            int code, out = 0;
            do {
                code = Q == ST_PHOTON ? photon_step(C, p, r, vx, gle, out) : electron_step(C, p, r, s, vx, out);
                steps++;
                if (++nst > GX_STEP_BUDGET) { atomicOr(C.err, GX_ERR_STEP_BUDGET); break; }
            } while (code == STEP_ON);
            if (code == STEP_QUEUE) push_move(C, out, p, r);
        } else {
            run_interaction<Q>(C, p, r);
        }
    }
    block_stat_add(C, Q, taken);
    if (Q == ST_PHOTON) block_stat_add(C, GX_NSTAGE, steps);
    if (Q == ST_ELECTRON) block_stat_add(C, GX_NSTAGE + 1, steps);
    consumer_done(C, gridDim.x, Q);
}

// ---- planner: next wave's injection and the loop condition -----------------
// One warp: a lane per queue reads its count (one thread reading the 25 one
// after another took most of the 9 to 12 us between two waves).
__device__ __forceinline__ uint32_t plan_wave(const DevCtx &C, SchedState *st)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t count = lane < GX_NQ ? *((volatile uint32_t *)&C.q.count[lane]) : 0u;
    const bool is_main = lane == ST_PHOTON || lane == ST_ELECTRON || lane >= GX_Q_PCONT;
    const uint32_t inflight = __reduce_add_sync(0xffffffffu, count);
    const uint32_t main_q = __reduce_add_sync(0xffffffffu, is_main ? count : 0u);
    const uint32_t side_q = __reduce_add_sync(0xffffffffu, lane >= GX_Q_ENEAR ? count : 0u);   // empty between waves
    uint32_t pending = 0;
    if (lane == 0) {
        const uint32_t err = *((volatile uint32_t *)C.err);
        const unsigned long long remaining = st->end - st->next;
        unsigned long long inject = 0;
        // what is left is small: the drain kernel takes all of it, and the waves end
        st->drain = main_q + remaining > 0 && main_q == inflight && side_q == 0u && main_q + remaining <= st->drain_below && err == 0u;
        // once the population falls below `refill_below`, top it up to `batch`
        if (!st->drain && remaining > 0 && main_q < st->refill_below && main_q < st->batch) {
            inject = st->batch - main_q;
            if (inject > remaining) inject = remaining;
        }
        st->h0 = st->next;
        st->h1 = st->next + inject;
        st->next += inject;
        // The tail of a run: every history injected and few particles left. The
        // waves are then short and their fixed cost (launches, the step chains of
        // single particles) dominates; larger step budgets take fewer of them.
        st->budget_shift = (st->next >= st->end && main_q < st->batch / GX_TAIL_DIV) ? GX_TAIL_SHIFT : 0u;
        st->waves++;
        st->photon_done = 0u;
        st->electron_done = 0u;
        pending = (inflight > 0 || inject > 0 || st->next < st->end) ? 1u : 0u;
        if (pending && st->waves >= st->max_waves) {
            atomicOr(C.err, GX_ERR_STEP_BUDGET);
            pending = 0;
        }
        if ((err & GX_ERR_QUEUE_FULL) || st->drain) pending = 0;
        st->pending = pending;
    }
    return __shfl_sync(0xffffffffu, pending, 0);
}

__global__ void k_plan(const __grid_constant__ DevCtx C, SchedState *st)
{
    plan_wave(C, st);
}

// Planner of a host-driven loop that queues several waves between checks
// (gegs_run_noalloc): once a plan has ended the run (pending 0), later calls
// inject nothing and count no wave, so the run's wave count and injected
// histories are those of the graph form, which stops at that plan.
__global__ void k_plan_gated(const __grid_constant__ DevCtx C, SchedState *st)
{
    const uint32_t pending = *((volatile uint32_t *)&st->pending);
    __syncwarp();
    if (pending == 0u) {
        if (threadIdx.x == 0) st->h0 = st->h1 = st->next;
        return;
    }
    plan_wave(C, st);
}

// Behind the drain kernel: if it ran, the queues it emptied are reset (their
// peaks recorded) and the next wave is planned, for what it left in the event
// queues. Returns whether it left anything.
__device__ __forceinline__ uint32_t drain_end(const DevCtx &C, SchedState *st)
{
    const uint32_t drained = *((volatile uint32_t *)&st->drain);
    __syncwarp();
    if (drained == 0u) return 0u;
    if (threadIdx.x < 8u) {
        const int k = (int)threadIdx.x, q = k < 6 ? GX_Q_PCONT + 2 * k + (int)(*C.wave & 1u) : k == 6 ? ST_PHOTON : ST_ELECTRON;
        if (C.q.peak && C.q.count[q] > C.q.peak[q]) C.q.peak[q] = C.q.count[q];
        C.q.count[q] = 0;
        C.q.head[q] = 0;
    }
    if (threadIdx.x == 0) {
        st->next = st->end;
        st->drain_below = 0u;
        st->drain_hist = 0ull;
    }
    __syncwarp();
    const uint32_t left = plan_wave(C, st);
    if (threadIdx.x == 0) st->resume = left;
    return left;
}

__global__ void k_drain_end(const __grid_constant__ DevCtx C, SchedState *st)
{
    drain_end(C, st);
}

__global__ void k_drain_end_cond(const __grid_constant__ DevCtx C, SchedState *st, cudaGraphConditionalHandle handle)
{
    const uint32_t left = drain_end(C, st);
    if (threadIdx.x == 0) cudaGraphSetConditional(handle, left);
}

// Enters the wave loop: plans its first wave, unless that has been done (drain_end).
__global__ void k_plan_enter(const __grid_constant__ DevCtx C, SchedState *st, cudaGraphConditionalHandle handle)
{
    const uint32_t resume = *((volatile uint32_t *)&st->resume);
    __syncwarp();
    const uint32_t pending = resume ? 1u : plan_wave(C, st);
    if (threadIdx.x == 0) {
        st->resume = 0u;
        cudaGraphSetConditional(handle, pending);
    }
}

__global__ void k_plan_cond(const __grid_constant__ DevCtx C, SchedState *st, cudaGraphConditionalHandle handle)
{
    uint32_t pending = plan_wave(C, st);
    if (threadIdx.x == 0) cudaGraphSetConditional(handle, pending);
}

// ---- geometry probe (gegs_probe_geometry) ----------------------------------
__device__ __forceinline__ Part probe_part(const gegs_probe_state &s)
{
    Part p = {};
    p.region = s.region; p.charge = s.charge; p.leafIndex = s.leafIndex; p.bank = s.bank;
    p.module = s.module; p.field = s.field; p.status = s.status;
    p.wt = s.wt; p.e = s.e; p.x = s.x; p.y = s.y; p.z = s.z; p.u = s.u; p.v = s.v; p.w = s.w;
    return p;
}

__global__ void k_probe_geometry(const __grid_constant__ DevCtx C, uint32_t n, const gegs_probe_state *in,
                                 const float *t_in, uint32_t *far_region, float *far_t, gegs_probe_state *far_out,
                                 float *near_t)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const gegs_probe_state s = in[i];
    Part p = probe_part(s);
    float t = t_in[i];
    bool ok;
    far_region[i] = howfar(C, p, t, ok);
    far_t[i] = t;
    gegs_probe_state o = s;
    o.leafIndex = p.leafIndex; o.bank = p.bank; o.module = p.module;
    far_out[i] = o;
    Part q = probe_part(s);
    float tp = 0.0f;
    hownear(C, q, tp, ok);
    near_t[i] = tp;
}

// The forms of the same routines that only some steps take: howfar by the whole
// warp, one state after another (share_steps), and hownear as an electron step
// with tustep t_in and the given range (negative: no range rejection) uses it.
__global__ void k_probe_step_geometry(const __grid_constant__ DevCtx C, uint32_t n, const gegs_probe_state *in,
                                      const float *t_in, const float *range, uint32_t *far_region, float *far_t,
                                      gegs_probe_state *far_out, float *near_t)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool have = i < n;
    gegs_probe_state s = {};
    if (have) s = in[i];
    const Part p = probe_part(s);
    const float t = have ? t_in[i] : 0.0f;
    for (unsigned m = __ballot_sync(0xffffffffu, have); m; m &= m - 1u) {
        const int src = __ffs(m) - 1;
        Part q = part_of(p, src);
        float tq = __shfl_sync(0xffffffffu, t, src);
        bool ok;
        uint32_t region;
        switch (geom_class_of(q.module)) {
        case GX_GEOM_JAWS: region = howfar_g<GX_GEOM_JAWS, true>(C, q, tq, ok); break;
        case GX_GEOM_MLC: region = howfar_g<GX_GEOM_MLC, true>(C, q, tq, ok); break;
        default: region = howfar(C, q, tq, ok);
        }
        __syncwarp();
        if ((int)(threadIdx.x & 31u) == src) {
            far_region[i] = region;
            far_t[i] = tq;
            gegs_probe_state o = s;
            o.leafIndex = q.leafIndex; o.bank = q.bank; o.module = q.module;
            far_out[i] = o;
        }
    }
    if (!have) return;
    Part q = p;
    NearUse use;
    use.rr = range[i] >= 0.0f;
    use.range = range[i];
    use.tustep = t;
    float tp = 0.0f;
    bool ok;
    switch (geom_class_of(q.module)) {
    case GX_GEOM_JAWS: hownear_g<GX_GEOM_JAWS>(C, q, tp, ok, use); break;
    case GX_GEOM_MLC: hownear_g<GX_GEOM_MLC>(C, q, tp, ok, use); break;
    default: hownear(C, q, tp, ok);
    }
    near_t[i] = tp;
}

__global__ void k_dose(const unsigned long long *tally, const float *mass, double unit, double *out, uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        double m = (double)mass[i];
        if (m == 0.0) m = 1.0;
        out[i] = (double)(long long)tally[i] * 9.313225746154785e-10 / m * unit;
    }
}

// ---- batch statistics (the reference's GET_UNCERTAINTY, CUDA_EGS.cu:817-876) ----
// One batch ends: x = tally gained since the last fold (MeV), S1 += x, S2 += x^2.
__global__ void k_stat_fold(const unsigned long long *tally, unsigned long long *snap, double *s1, double *s2,
                            uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long t = tally[i];
        const double x = (double)(long long)(t - snap[i]) * 9.313225746154785e-10;
        snap[i] = t;
        s1[i] += x;
        s2[i] += x * x;
    }
}

// Batch mean and the relative standard error of the mean of n batches,
// sqrt((S2/n - (S1/n)^2) / (n - 1)) / (S1/n) (0 where nothing was deposited).
__global__ void k_stat_final(const double *s1, const double *s2, double n, double *mean, double *rel, uint64_t nv)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nv; i += (uint64_t)gridDim.x * blockDim.x) {
        const double m = s1[i] / n;
        const double v = s2[i] / n - m * m;
        mean[i] = m;
        rel[i] = m > 0.0 ? sqrt((v > 0.0 ? v : 0.0) / (n - 1.0)) / m : 0.0;
    }
}
