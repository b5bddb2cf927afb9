// The drain kernel: takes what is left of a run once it is small and transports
// it to its end in one launch.
//
// A wave of the persistent form costs some 100 us however few particles it
// moves: its kernels start and end one after another and the slowest particle
// of each holds the rest up. A run's tail is all such waves, and so is a run of
// few histories. Here each warp works by itself: it keeps a stack of particles
// per type (photons and electrons of each geometry class, the eight
// interactions), takes the type it has most of, runs up to 32 of them side by
// side, and what they make goes back on its own stacks, so that a warp still
// executes one kind of work at a time but waits for nobody. Warps that run low
// claim more from the event queues, or histories not yet started. There are no
// barriers and no waits: a warp ends when its stacks and the queues are empty, or
// after so many turns (C.drain_turns) that one of its particles may never end;
// then all it has goes to the event queues, and the waves' budget ends the run.
// A stack that is full sends the particle to the event queues, and the run goes
// on in waves behind the drain kernel, in the same launch (add_wave_loop). With
// the tables' own single bremsstrahlung photon no plan has been seen to need
// it; photons split more than 64 ways overflow at once.
//
// Bound by the longest cascade of one warp, step after step, and by fetching
// instructions (all stages in one kernel, 850 KB: on the CT head, 4000 histories,
// 16 cycles per issue, issue slots 14 % busy, 4 lanes active): that is why it
// takes the last few thousand particles only (drain_threshold). 80 registers,
// 24 warps per SM; 128 registers and 16 warps measured the same. At 80 each
// stage spills 0.2 to 1.0 KB of stores and 0.5 to 2.1 KB of loads.
#define GX_WARP_STACKS
#include "dev_run.cuh"
#include "drain.cuh"

namespace {

constexpr int kWarps = kDrainThreads / 32;

struct DrainWarp {
    uint32_t cnt[GX_DT_N];     // records on each stack
    uint32_t turns;            // turns that are left to the warp
    uint32_t taken[GX_NSTAGE]; // particles taken per stage
    uint32_t steps[2];         // photon, electron
    uint32_t head_steps[4];    // photon jaws, MLC, electron jaws, MLC
};

__shared__ DrainWarp g_warp[kWarps];
// The context, copied here by each block: the work of each type is a function
// of its own, and a function reads it from shared memory faster than through a
// pointer to the kernel's parameter. (Inlined into one kernel the stages spill as
// much and take the same time: water, 10 000 histories 2.13 and 2.14 ms, slab,
// 200 000 9.67 and 9.70.)
__shared__ DevCtx g_ctx;

__device__ __forceinline__ DrainWarp &warp_of() { return g_warp[threadIdx.x >> 5]; }
__device__ __forceinline__ size_t warp_index() { return (size_t)blockIdx.x * kWarps + (threadIdx.x >> 5); }

__device__ __forceinline__ Part *slot_part(const DevCtx &C, int type, uint32_t i)
{
    return C.drain_part + (warp_index() * GX_DT_N + (size_t)type) * GX_DRAIN_CAP + i;
}

__device__ __forceinline__ EStatePk *slot_estate(const DevCtx &C, int type, uint32_t i)
{
    return C.drain_estate + (warp_index() * 3 + (size_t)(type - GX_DT_E)) * GX_DRAIN_CAP + i;
}

// Stack of a particle queued for stage qid.
__device__ __forceinline__ int stack_of(int qid, const Part &p)
{
    if (qid == ST_PHOTON) return GX_DT_P + geom_class_of(p.module) - GX_GEOM_JAWS;
    if (qid == ST_ELECTRON) return GX_DT_E + geom_class_of(p.module) - GX_GEOM_JAWS;
    return GX_DT_I + qid - (qid < ST_ELECTRON ? ST_COMPTON : ST_MOLLER - 4);
}

// `status` of a record: its stage where it is new there, kGoesOn where its
// transport has begun (an electron's step state is then beside it).
constexpr uint8_t kGoesOn = 0xFF;

__device__ __forceinline__ EStatePk fresh_estate()
{
    EState s;
    estate_init(s);
    return pack_estate(s);
}

// A full stack: to the event queues, where the next wave finds it.
__device__ __noinline__ void spill(const DevCtx &C, int type, Part p, const EStatePk &k)
{
    int qid;
    if (type >= GX_DT_I) qid = type - GX_DT_I < 4 ? ST_COMPTON + type - GX_DT_I : ST_MOLLER + type - GX_DT_I - 4;
    else qid = (type < GX_DT_E ? GX_Q_PCONT + 2 * type : GX_Q_ECONT + 2 * (type - GX_DT_E)) + (int)((*C.wave & 1u) ^ 1u);
    const uint32_t i = atomicAdd(&C.q.count[qid], 1u);
    if (i >= C.q.cap[qid]) { atomicOr(C.err, GX_ERR_QUEUE_FULL); return; }
    if (type < GX_DT_I && p.status != kGoesOn) {      // queued as a continuation, so counted as taken here
        atomicAdd(&warp_of().taken[type < GX_DT_E ? ST_PHOTON : ST_ELECTRON], 1u);
        trace_event(C, 1u, type < GX_DT_E ? ST_PHOTON : ST_ELECTRON, p);
    }
    store_part(&C.q.buf[qid][i], p);
    if (type >= GX_DT_E && type < GX_DT_I) C.q.estate[qid - GX_Q_ECONT][i] = k;
}

__device__ __forceinline__ void stack_push(const DevCtx &C, int type, const Part &p, const EStatePk *k)
{
    const uint32_t i = atomicAdd(&warp_of().cnt[type], 1u);
    if (i < C.drain_cap) {
        store_part(slot_part(C, type, i), p);
        if (k) *slot_estate(C, type, i) = *k;
    } else spill(C, type, p, k ? *k : fresh_estate());
}

}  // namespace

__device__ __forceinline__ void push(const DevCtx &C, int qid, const Part &p)
{
    Part r = p;
    r.status = (uint8_t)qid;
    trace_event(C, 0u, qid, r);
    stack_push(C, stack_of(qid, r), r, nullptr);
}

namespace {

// A transport: up to 32 particles of one type, lanes refilled from the warp's
// stack, until the stack is empty and the lanes are done -- or few lanes are
// left and another stack has more to run.
template <bool ELEC, int G>
__device__ __noinline__ void drain_transport()
{
    const DevCtx &C = g_ctx;
    constexpr int cls = G - GX_GEOM_JAWS;
    constexpr int T = (ELEC ? GX_DT_E : GX_DT_P) + cls;
    constexpr int Q = ELEC ? ST_ELECTRON : ST_PHOTON;
    DrainWarp &w = warp_of();
    const uint32_t lane = threadIdx.x & 31u;
    Part p;
    Rng r;
    EState s;
    Vox vx;
    float gle = 0.0f;
    bool active = false;
    uint32_t steps = 0, taken = 0;
    __syncwarp();
    uint32_t turns = w.turns;
    for (;;) {
        __syncwarp();
        uint32_t act = __ballot_sync(0xffffffffu, active);
        const uint32_t have = min(w.cnt[T], C.drain_cap);
        if (have > 0 && __popc(act) <= 24) {
            const uint32_t take = min(32u - __popc(act), have);
            const uint32_t rank = __popc(~act & ((1u << lane) - 1u));
            if (!active && rank < take) {
                const uint32_t i = have - 1u - rank;
                p = load_part(slot_part(C, T, i));
                rng_load(r, p);
                vx = C.reg[p.region];
                if (!ELEC) gle = gx_log(p.e);
                active = true;
                if (p.status == kGoesOn) {
                    if (ELEC) unpack_estate(*slot_estate(C, T, i), s);
                } else {
                    if (ELEC) estate_init(s);
                    trace_event(C, 1u, Q, p);
                    taken++;
                }
            }
            __syncwarp();
            if (lane == 0) w.cnt[T] = have - take;
            __syncwarp();
            act = __ballot_sync(0xffffffffu, active);
        }
        if (act == 0u) break;
        bool leave = turns == 0u;
        if (!leave) turns--;
        if (__popc(act) <= 8) {
            const uint32_t other = lane < GX_DT_N && (int)lane != T ? w.cnt[lane] : 0u;
            leave |= __any_sync(0xffffffffu, other >= 16u);
        }
        const bool in_class = in_geom_class<G>(p);     // before the step, which may leave it
        int code = STEP_ON, shared = -1;
        const bool share = !ELEC && cls < 2 && !leave && __popc(act) <= GX_SHARE_LANES;
        if (share) {
            const bool stepping = active && in_class;
            if (stepping) rng_window(C, r);
            share_steps<G>(C, __ballot_sync(0xffffffffu, stepping), p, r, vx, gle, code, shared);
        }
        if (active) {
            int to = -1, out = 0;                 // the stack the particle leaves for; the stage it is new in there
            bool moved = true;
            if (leave) to = T;
            else if (!in_class) to = (ELEC ? GX_DT_E : GX_DT_P) + geom_class_of(p.module) - GX_GEOM_JAWS;
            else {
                steps++;
                if (share) out = shared;
                else {
                    rng_window(C, r);
                    code = ELEC ? electron_step<G>(C, p, r, s, vx, out) : photon_step<G>(C, p, r, vx, gle, out);
                }
                if (code == STEP_DONE) active = false;
                else if (code == STEP_QUEUE) { to = stack_of(out, p); moved = false; }
            }
            if (to >= 0) {
                rng_store(r, p);
                p.status = moved ? kGoesOn : (uint8_t)out;
                if (!moved) trace_event(C, 0u, out, p);
                EStatePk k = pack_estate(s);
                stack_push(C, to, p, ELEC && moved ? &k : nullptr);
                active = false;
            }
        }
        if (leave) break;
    }
    __syncwarp();
    steps = __reduce_add_sync(0xffffffffu, steps);
    taken = __reduce_add_sync(0xffffffffu, taken);
    if (lane == 0) {
        w.turns = turns;
        w.taken[Q] += taken;
        w.steps[ELEC ? 1 : 0] += steps;
        if (cls < 2) w.head_steps[(ELEC ? 2 : 0) + cls] += steps;
    }
}

// The transports of the jaws and the MLC; a beam line of the phantom alone has no such particle.
template <bool HEAD, bool ELEC, int G>
__device__ __forceinline__ void drain_head()
{
    if constexpr (HEAD) drain_transport<ELEC, G>();
    else if ((threadIdx.x & 31u) == 0u) {
        warp_of().cnt[(ELEC ? GX_DT_E : GX_DT_P) + G - GX_GEOM_JAWS] = 0u;
        atomicOr(g_ctx.err, GX_ERR_MODULE);
    }
}

template <int Q>
__device__ __noinline__ void drain_interaction()
{
    const DevCtx &C = g_ctx;
    constexpr int T = GX_DT_I + Q - (Q < ST_ELECTRON ? ST_COMPTON : ST_MOLLER - 4);
    DrainWarp &w = warp_of();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t have = min(w.cnt[T], C.drain_cap);
    const uint32_t take = min(32u, have);
    const bool active = lane < take;
    Part p;
    if (active) p = load_part(slot_part(C, T, have - 1u - lane));
    __syncwarp();
    if (lane == 0) w.cnt[T] = have - take;
    __syncwarp();
    uint32_t n = 0;
    if (active) {
        Rng r;
        rng_load(r, p);
        rng_window(C, r);
        trace_event(C, 1u, Q, p);
        n = counted<Q>(p);
        run_interaction<Q>(C, p, r);
    }
    __syncwarp();
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) w.taken[Q] += n;
}

// The event queues a drain begins with, the longest tracks first: photons
// under way, histories not yet started, new photons, electrons under way, new
// electrons.
constexpr int kPools = 9;

__device__ __forceinline__ int pool_queue(int k, uint32_t par)
{
    switch (k) {
    case 0: case 1: case 2: return GX_Q_PCONT + 2 * k + (int)par;
    case 3: return -1;                                   // histories
    case 4: return ST_PHOTON;
    case 5: case 6: case 7: return GX_Q_ECONT + 2 * (k - 5) + (int)par;
    default: return ST_ELECTRON;
    }
}

// Claim up to `per` particles of the first pool that has any onto the warp's
// stacks; false once all are empty (`pool` remembers the first that may not be).
__device__ __noinline__ bool claim(SchedState *st, uint32_t par, uint32_t per, int &pool)
{
    const DevCtx &C = g_ctx;
    const uint32_t lane = threadIdx.x & 31u;
    for (; pool < kPools; pool++) {
        const int q = pool_queue(pool, par);
        const unsigned long long n = q < 0 ? st->end - st->next : (unsigned long long)queue_len(C, q);
        if (n == 0) continue;
        unsigned long long base = 0;
        if (lane == 0) base = q < 0 ? atomicAdd(&st->drain_hist, (unsigned long long)per) : (unsigned long long)atomicAdd(&C.q.head[q], per);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) continue;
        const unsigned long long i = base + lane;
        if (lane < per && i < n) {
            Part p;
            if (q < 0) {
                if (make_primary(C, st->next + i, p)) push(C, p.charge == 0 ? ST_PHOTON : ST_ELECTRON, p);
                else atomicOr(C.err, GX_ERR_SOURCE);
            } else {
                p = load_part(&C.q.buf[q][i]);
                if (q == ST_PHOTON || q == ST_ELECTRON) stack_push(C, stack_of(q, p), p, nullptr);
                else {
                    p.status = kGoesOn;
                    const bool e = q >= GX_Q_ECONT;
                    EStatePk k;
                    if (e) k = C.q.estate[q - GX_Q_ECONT][i];
                    stack_push(C, stack_of(e ? ST_ELECTRON : ST_PHOTON, p), p, e ? &k : nullptr);
                }
            }
        }
        __syncwarp();
        return true;
    }
    return false;
}

// All that is on the warp's stacks goes to the event queues.
__device__ __noinline__ void spill_stacks()
{
    const DevCtx &C = g_ctx;
    DrainWarp &w = warp_of();
    const uint32_t lane = threadIdx.x & 31u;
    for (int type = 0; type < GX_DT_N; type++) {
        const uint32_t n = min(w.cnt[type], C.drain_cap);
        for (uint32_t i = lane; i < n; i += 32) {
            const Part p = load_part(slot_part(C, type, i));
            const bool state = type >= GX_DT_E && type < GX_DT_I && p.status == kGoesOn;
            spill(C, type, p, state ? *slot_estate(C, type, i) : fresh_estate());
        }
    }
    __syncwarp();
    if (lane < GX_DT_N) w.cnt[lane] = 0u;
    __syncwarp();
}

template <bool HEAD>
__global__ void __launch_bounds__(kDrainThreads, 6) k_drain(const __grid_constant__ DevCtx ctx, SchedState *st)
{
    if (*((volatile uint32_t *)&st->drain) == 0u) return;
    static_assert(sizeof(DevCtx) % 4 == 0, "copied by words");
    for (uint32_t i = threadIdx.x; i < sizeof(DevCtx) / 4; i += kDrainThreads)
        reinterpret_cast<uint32_t *>(&g_ctx)[i] = reinterpret_cast<const uint32_t *>(&ctx)[i];
    __syncthreads();
    const DevCtx &C = g_ctx;
    timeline_mark(C, TL_DRAIN, false);
    DrainWarp &w = warp_of();
    const uint32_t lane = threadIdx.x & 31u, par = *C.wave & 1u;
    for (uint32_t i = lane; i < sizeof(DrainWarp) / 4; i += 32) reinterpret_cast<uint32_t *>(&w)[i] = 0u;
    __syncwarp();
    if (lane == 0) w.turns = C.drain_turns;
    // an even share of what there is, so that a small run spreads over the SMs, up to a warp's width
    unsigned long long total = st->end - st->next;
    for (int k = 0; k < kPools; k++) {
        const int q = pool_queue(k, par);
        if (q >= 0) total += queue_len(C, q);
    }
    const unsigned long long warps = (unsigned long long)gridDim.x * kWarps;
    const uint32_t per = (uint32_t)min(32ull, (total + warps - 1) / warps);
    int pool = 0;
    for (;;) {
        __syncwarp();
        uint32_t c = 0;
        if (lane < GX_DT_N) {
            c = min(w.cnt[lane], C.drain_cap);
            w.cnt[lane] = c;
        }
        const uint32_t best = __reduce_max_sync(0xffffffffu, c * 32u + lane);
        const uint32_t all = __reduce_add_sync(0xffffffffu, c);
        const bool over = w.turns == 0u;
        __syncwarp();
        if (over) {
            if (all) spill_stacks();
            if (pool < kPools && claim(st, par, per, pool)) continue;
            break;
        }
        if (all < per && pool < kPools && claim(st, par, per, pool)) continue;
        if (all == 0u) break;
        if (lane == 0) w.turns--;
        switch (best & 31u) {
        case GX_DT_P + 2: drain_transport<false, GX_GEOM_PHANTOM>(); break;
        case GX_DT_E + 2: drain_transport<true, GX_GEOM_PHANTOM>(); break;
        case GX_DT_I + 0: drain_interaction<ST_COMPTON>(); break;
        case GX_DT_I + 1: drain_interaction<ST_PHOTO>(); break;
        case GX_DT_I + 2: drain_interaction<ST_RAYLEIGH>(); break;
        case GX_DT_I + 3: drain_interaction<ST_PAIR>(); break;
        case GX_DT_I + 4: drain_interaction<ST_MOLLER>(); break;
        case GX_DT_I + 5: drain_interaction<ST_BREMS>(); break;
        case GX_DT_I + 6: drain_interaction<ST_BHABHA>(); break;
        case GX_DT_I + 7: drain_interaction<ST_ANNIH>(); break;
        case GX_DT_P + 1: drain_head<HEAD, false, GX_GEOM_MLC>(); break;
        case GX_DT_E + 1: drain_head<HEAD, true, GX_GEOM_MLC>(); break;
        case GX_DT_P + 0: drain_head<HEAD, false, GX_GEOM_JAWS>(); break;
        case GX_DT_E + 0: drain_head<HEAD, true, GX_GEOM_JAWS>(); break;
        }
    }
    if (lane < GX_NSTAGE && w.taken[lane]) atomicAdd(&C.stats[lane], (unsigned long long)w.taken[lane]);
    if (lane < 2 && w.steps[lane]) atomicAdd(&C.stats[GX_NSTAGE + lane], (unsigned long long)w.steps[lane]);
    if (lane < 4 && w.head_steps[lane]) atomicAdd(&C.stats[GX_NSTAGE + 2 + lane], (unsigned long long)w.head_steps[lane]);
    if (C.timeline) {
        __syncthreads();
        timeline_mark(C, TL_DRAIN, true);
    }
}

}  // namespace

int drain_blocks_per_sm(bool head)
{
    int n = 0;
    cudaError_t c = head ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_drain<true>, kDrainThreads, 0)
                         : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_drain<false>, kDrainThreads, 0);
    return c == cudaSuccess && n > 0 ? n : 1;
}

size_t drain_frames(bool head)
{
    cudaFuncAttributes a;
    int device = 0, sms = 0, threads = 0;
    if ((head ? cudaFuncGetAttributes(&a, k_drain<true>) : cudaFuncGetAttributes(&a, k_drain<false>)) != cudaSuccess ||
        cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&threads, cudaDevAttrMaxThreadsPerMultiProcessor, device) != cudaSuccess)
        return (size_t)1 << 30;
    return a.localSizeBytes * (size_t)sms * (size_t)threads + ((size_t)64 << 20);
}

void launch_drain(const DevCtx &C, SchedState *st, bool head, int grid, cudaStream_t s)
{
    if (head) k_drain<true><<<grid, kDrainThreads, 0, s>>>(C, st);
    else k_drain<false><<<grid, kDrainThreads, 0, s>>>(C, st);
}
