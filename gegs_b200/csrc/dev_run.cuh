// What the transport kernels of a run share, whichever way they are launched:
// the scheduler state, the wave timeline stamps, the electron step state as it
// is stored, a history's primary, and the interaction of one particle.
#pragma once
#include "dev_electron.cuh"

struct SchedState {
    unsigned long long next, end;     // history cursor
    unsigned long long h0, h1;        // histories injected by the current wave
    uint32_t batch, waves, max_waves, pending;
    uint32_t refill_below;
    uint32_t photon_done;             // photon MLC and phantom consumers finished in this wave
    uint32_t electron_done;           // electron branches finished in this wave
    uint32_t drain_below;             // the drain kernel takes over at this many particles and histories left (0: never)
    uint32_t drain;                   // 1: it does, after this plan
    uint32_t resume;                  // 1: it left particles in the event queues, and the wave that takes them is planned
    unsigned long long drain_hist;    // histories it has claimed
    uint32_t budget_shift;            // step budgets of the next wave are shifted left by this (tail of a run)
};

// ---- wave timeline (tracing; off unless DevCtx::timeline is set) ------------
// Kernel ids: 0 source; 1-3 photon jaws / MLC / phantom; 4-7 Compton, photo,
// Rayleigh, pair; 8-10 electron jaws / MLC / phantom; 11-14 Moller, brems,
// Bhabha, annihilation. Each block's thread 0 lowers the kernel's start stamp
// of this wave when the block begins and raises its end stamp once the block
// is done (after the block's barrier).
enum : int { TL_SOURCE = 0, TL_PHOTON = 1, TL_PINT = 4, TL_ELECTRON = 8, TL_EINT = 11, TL_ENEAR = 15, TL_PLONG = 16, TL_DRAIN = 17 };

__device__ __forceinline__ void timeline_mark(const DevCtx &C, int kernel, bool end)
{
    if (C.timeline == nullptr || threadIdx.x != 0) return;
    uint32_t w = *((volatile const uint32_t *)C.wave);
    if (w >= C.timeline_waves) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    unsigned long long *slot = C.timeline + ((size_t)w * GX_TL_KERNELS + (size_t)kernel) * 2;
    if (end) atomicMax(slot + 1, t);
    else atomicMin(slot, t);
}

__device__ __forceinline__ EStatePk pack_estate(const EState &s)
{
    EStatePk k;
    k.elke = s.elke; k.demfp = s.demfp; k.sig0 = s.sig0; k.total_tstep = s.total_tstep;
    k.lelke = s.lelke;
    k.flags = (s.compute_tstep ? 1u : 0u) | (s.is_tstep ? 2u : 0u);
    k.pad0 = 0; k.pad1 = 0;
    return k;
}

__device__ __forceinline__ void unpack_estate(const EStatePk &k, EState &s)
{
    s.elke = k.elke; s.demfp = k.demfp; s.sig0 = k.sig0; s.total_tstep = k.total_tstep;
    s.lelke = k.lelke;
    s.compute_tstep = (k.flags & 1u) != 0;
    s.is_tstep = (k.flags & 2u) != 0;
}

// One step of each photon of the lanes `act` in turn, by the whole warp: for the
// few photons that are left when a queue has run out, which otherwise step at
// the speed of one lane (a photon that goes along a jaw face or a leaf gap for
// thousands of steps, 1.4 and 8 us each, one edge after another). Their polygon
// edges are tested side by side. Every lane's random window has been filled.
#define GX_SHARE_LANES 4
template <int G>
__device__ __forceinline__ void share_steps(const DevCtx &C, unsigned act, Part &p, Rng &r, Vox &vx, float gle, int &code, int &out)
{
    __syncwarp();
    for (unsigned m = act; m; m &= m - 1u) {
        const int src = __ffs(m) - 1;
        Part q = part_of(p, src);
        Vox v;
        v.med = (uint16_t)__shfl_sync(0xffffffffu, (uint32_t)vx.med, src);
        v.flags = (uint16_t)__shfl_sync(0xffffffffu, (uint32_t)vx.flags, src);
        v.rhof = __shfl_sync(0xffffffffu, vx.rhof, src);
        const float g = __shfl_sync(0xffffffffu, gle, src);
        Rng rq = {};
        rq.ctr = __shfl_sync(0xffffffffu, r.ctr, src);
        int to = -1;
        const int c = photon_step<G, false, true>(C, q, rq, v, g, to, (threadIdx.x & ~31u) + (uint32_t)src);
        if ((int)(threadIdx.x & 31u) == src) {
            p = q;
            vx = v;
            r.ctr = rq.ctr;
            code = c;
            out = to;
        }
    }
}

__device__ __forceinline__ uint32_t queue_len(const DevCtx &C, int q)
{
    uint32_t n = *((volatile uint32_t *)&C.q.count[q]);
    return n < C.q.cap[q] ? n : C.q.cap[q];
}

// ---- source: history index -> primary (CUDA_EGS.cu:52-131) -----------------
static __device__ bool make_primary(const DevCtx &C, unsigned long long h, Part &p)
{
    int f;
    for (f = 0; f < C.nfields; f++) {
        unsigned long long hb = C.fields[f].hist_begin, he = C.fields[f].hist_end;
        if (h >= hb && h < he) break;
    }
    if (f == C.nfields) return false;
    const gegs_field *F = &C.fields[f];
    unsigned long long j = (h - F->hist_begin) / (unsigned long long)(F->nrepeat + 1);
    const gegs_phsp_record *rec = &C.phsp[j % C.nphsp];
    uint32_t latch = __ldg(&rec->latch);
    float re = __ldg(&rec->e), rx = __ldg(&rec->x), ry = __ldg(&rec->y);
    float ru = __ldg(&rec->u), rv = __ldg(&rec->v), rwt = __ldg(&rec->wt);
    int q;
    if (latch & 0x40000000u) q = -1;
    else if (latch & 0x20000000u) q = 1;
    else q = 0;
    float w2 = 1.0f - ru * ru - rv * rv;
    float w = sqrtf(w2 > 0.0f ? w2 : 0.0f);
    float wt = rwt;
    if (wt < 0.0f) { w = -w; wt = -wt; }
    p.charge = (int8_t)q;
    p.e = re < 0.0f ? -re : re;
    p.wt = wt;
    p.region = 0;
    p.leafIndex = GX_OUTMLC;
    p.bank = -1;
    p.module = (uint8_t)C.module_order[0];
    p.field = (uint8_t)f;
    p.x = rx; p.y = ry; p.z = C.z_phsp;
    p.u = ru; p.v = rv; p.w = w;
    p.hist_lo = (uint32_t)h;
    p.hist_hi = (uint32_t)(h >> 32);
    p.sid_lo = 0; p.sid_hi = 0; p.ctr = 0;
    p.status = 0;
    // beamlet: the bixel of the isocentre plane on the primary's straight line
    p.beamlet = GX_NO_BEAMLET;
    if (C.bl_nx > 0 && w > 0.0f) {
        float t = (C.sid - C.z_phsp) / w;
        float xi = rx + ru * t, yi = ry + rv * t;
        float fx = (xi - C.bl_x0) / C.bl_dx, fy = (yi - C.bl_y0) / C.bl_dy;
        if (fx >= 0.0f && fy >= 0.0f && fx < (float)C.bl_nx && fy < (float)C.bl_ny) {
            int b = f * C.bl_nx * C.bl_ny + (int)fy * C.bl_nx + (int)fx;
            p.beamlet = (uint16_t)b;
            if (C.bl_weight) p.wt = wt * __ldg(&C.bl_weight[b]);
        }
    }
    return true;
}

template <int Q>
__device__ __forceinline__ void run_interaction(const DevCtx &C, const Part &p, Rng &r)
{
    if (Q == ST_COMPTON) compton(C, p, r);
    else if (Q == ST_PHOTO) photo(C, p, r);
    else if (Q == ST_RAYLEIGH) rayleigh(C, p, r);
    else if (Q == ST_PAIR) pair(C, p, r);
    else if (Q == ST_MOLLER) moller(C, p, r);
    else if (Q == ST_BREMS) brems(C, p, r);
    else if (Q == ST_BHABHA) bhabha(C, p, r);
    else if (Q == ST_ANNIH) {
        if (at_rest_mark(p)) {
            Part q = p;
            annih_at_rest(C, q, region_info(C, q.region), r);
        } else annih(C, p, r);
    }
}

// Entries an interaction kernel counts as processed: all but the positrons that
// stopped in the electron transport (`processed` counts annihilations in flight).
template <int Q>
__device__ __forceinline__ unsigned counted(const Part &p)
{
    return (Q == ST_ANNIH && at_rest_mark(p)) ? 0u : 1u;
}

