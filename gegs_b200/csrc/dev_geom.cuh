// Device geometry: beam->patient transform and one-plane voxel DDA
// (howfar_phantom, geom.cu:54-307), isotropic distance to the voxel walls
// (hownear_phantom, geom.cu:1422-1543), DYNVMLC leaf tracking (howfar_MLC /
// hownear_MLC, geom.cu:310-790, 1152-1286) and the secondary jaws
// (geom.cu:793-1035, 1288-1374).  The reference's behaviour is kept, including
// its hownear voxel decode (region - 5, selectable) and the dis_yz step of
// howfar_SecJawsX inside the tungsten.
#pragma once
#include "dev_common.cuh"

struct P6 { float x, y, z, u, v, w; };

__device__ __forceinline__ P6 to_patient(const DevCtx &C, const Part &p0)
{
    const gegs_field *F = &C.fields[p0.field];
    float ca = __ldg(&F->cos_angle), sa = __ldg(&F->sin_angle);
    P6 p;
    if (C.change_xyz) {
        p.x = p0.y; p.y = p0.z - C.sid; p.z = p0.x;
        p.u = p0.v; p.v = p0.w; p.w = p0.u;
    } else {
        p.x = p0.x; p.y = p0.y; p.z = p0.z - C.sid;
        p.u = p0.u; p.v = p0.v; p.w = p0.w;
    }
    float tx = p.x * ca - p.y * sa;
    float ty = p.x * sa + p.y * ca;
    p.x = tx; p.y = ty;
    tx = p.u * ca - p.v * sa;
    ty = p.u * sa + p.v * ca;
    p.u = tx; p.v = ty;
    p.x = p.x + C.iso0;
    p.y = p.y + C.iso1;
    p.z = p.z + C.iso2;
    return p;
}

__device__ __forceinline__ int is_where(float p, uint32_t nreg, const float *bounds)
{
    if ((p < __ldg(&bounds[0])) || (p > __ldg(&bounds[nreg]))) return -1;
    if (nreg == 1) return 0;
    int ml = 0, mu = (int)nreg;
    while (mu - ml > 1) {
        int mav = (ml + mu) / 2;
        if (p <= __ldg(&bounds[mav])) mu = mav; else ml = mav;
    }
    return mu - 1;
}

static __device__ uint32_t howfar_phantom(const DevCtx &C, const Part &p0, float &t)
{
    const float *xb = C.xb, *yb = C.yb, *zb = C.zb;
    uint32_t Nx = (uint32_t)C.nx, Ny = (uint32_t)C.ny, Nz = (uint32_t)C.nz;
    P6 p = to_patient(C, p0);
    uint32_t region = p0.region;
    if (region >= GX_VAC_AND_OTH) {
        uint32_t ir = region - GX_VAC_AND_OTH;
        int iz = (int)fastdiv(C.div_nxny, ir);
        ir -= (uint32_t)iz * Nx * Ny;
        int iy = (int)fastdiv(C.div_nx, ir);
        int ix = (int)(ir - (uint32_t)iy * Nx);
        uint32_t inew = region;
        if (p.u > 0.0f) {
            float d = (__ldg(&xb[ix + 1]) - p.x) / p.u;
            if (d <= t) { t = d; if ((uint32_t)(++ix) < Nx) inew = region + 1; else inew = 0; }
        } else if (p.u < 0.0f) {
            float d = (__ldg(&xb[ix]) - p.x) / p.u;
            if (d <= t) { t = d; if (--ix >= 0) inew = region - 1; else inew = 0; }
        }
        if (p.v > 0.0f) {
            float d = (__ldg(&yb[iy + 1]) - p.y) / p.v;
            if (d <= t) { t = d; if ((uint32_t)(++iy) < Ny) inew = region + Nx; else inew = 0; }
        } else if (p.v < 0.0f) {
            float d = (__ldg(&yb[iy]) - p.y) / p.v;
            if (d <= t) { t = d; if (--iy >= 0) inew = region - Nx; else inew = 0; }
        }
        if (p.w > 0.0f) {
            float d = (__ldg(&zb[iz + 1]) - p.z) / p.w;
            if (d <= t) { t = d; if ((uint32_t)(++iz) < Nz) inew = region + Nx * Ny; else inew = 0; }
        } else if (p.w < 0.0f) {
            float d = (__ldg(&zb[iz]) - p.z) / p.w;
            if (d <= t) { t = d; if (--iz >= 0) inew = region - Nx * Ny; else inew = 0; }
        }
        if (t < 0) t = GX_EPSTEP;
        return inew;
    }
    int ix, iy, iz;
    float t1 = 0.0f;
    ix = -1;
    if ((p.x <= __ldg(&xb[0])) && (p.u > 0.0f)) { t1 = (__ldg(&xb[0]) - p.x) / p.u; ix = 0; }
    else if ((p.x >= __ldg(&xb[Nx])) && (p.u < 0.0f)) { t1 = (__ldg(&xb[Nx]) - p.x) / p.u; ix = (int)Nx - 1; }
    if ((ix >= 0) && (t1 <= t)) {
        float y1 = p.y + p.v * t1;
        iy = is_where(y1, Ny, yb);
        if (iy >= 0) {
            float z1 = p.z + p.w * t1;
            iz = is_where(z1, Nz, zb);
            if (iz >= 0) { t = t1; return (uint32_t)ix + (uint32_t)iy * Nx + (uint32_t)iz * Nx * Ny + GX_VAC_AND_OTH; }
        }
    }
    iy = -1;
    if ((p.y <= __ldg(&yb[0])) && (p.v > 0.0f)) { t1 = (__ldg(&yb[0]) - p.y) / p.v; iy = 0; }
    else if ((p.y >= __ldg(&yb[Ny])) && (p.v < 0.0f)) { t1 = (__ldg(&yb[Ny]) - p.y) / p.v; iy = (int)Ny - 1; }
    if ((iy >= 0) && (t1 <= t)) {
        float x1 = p.x + p.u * t1;
        ix = is_where(x1, Nx, xb);
        if (ix >= 0) {
            float z1 = p.z + p.w * t1;
            iz = is_where(z1, Nz, zb);
            if (iz >= 0) { t = t1; return (uint32_t)ix + (uint32_t)iy * Nx + (uint32_t)iz * Nx * Ny + GX_VAC_AND_OTH; }
        }
    }
    iz = -1;
    if ((p.z <= __ldg(&zb[0])) && (p.w > 0.0f)) { t1 = (__ldg(&zb[0]) - p.z) / p.w; iz = 0; }
    else if ((p.z >= __ldg(&zb[Nz])) && (p.w < 0.0f)) { t1 = (__ldg(&zb[Nz]) - p.z) / p.w; iz = (int)Nz - 1; }
    if ((iz >= 0) && (t1 <= t)) {
        float x1 = p.x + p.u * t1;
        ix = is_where(x1, Nx, xb);
        if (ix >= 0) {
            float y1 = p.y + p.v * t1;
            iy = is_where(y1, Ny, yb);
            if (iy >= 0) { t = t1; return (uint32_t)ix + (uint32_t)iy * Nx + (uint32_t)iz * Nx * Ny + GX_VAC_AND_OTH; }
        }
    }
    return 0;
}

static __device__ void hownear_phantom(const DevCtx &C, const Part &p0, float &tperp)
{
    const float *xb = C.xb, *yb = C.yb, *zb = C.zb;
    uint32_t Nx = (uint32_t)C.nx, Ny = (uint32_t)C.ny, Nz = (uint32_t)C.nz;
    P6 p = to_patient(C, p0);
    uint32_t off = (uint32_t)C.hownear_off;
    tperp = GX_INFI_DIST;
    if (p0.region > off - 1u) {
        uint32_t ir = p0.region - off;
        int iz = (int)fastdiv(C.div_nxny, ir);
        ir -= (uint32_t)iz * Nx * Ny;
        int iy = (int)fastdiv(C.div_nx, ir);
        int ix = (int)(ir - (uint32_t)iy * Nx);
        float tx, ty, tz, tmp;
        tmp = __ldg(&xb[ix + 1]) - p.x; tx = p.x - __ldg(&xb[ix]); if (tmp < tx) tx = tmp;
        tmp = __ldg(&yb[iy + 1]) - p.y; ty = p.y - __ldg(&yb[iy]); if (tmp < ty) ty = tmp;
        // the reference decode maps the last voxel to iz = nz: the missing plane is the last plane
        tmp = __ldg(&zb[(uint32_t)(iz + 1) <= Nz ? iz + 1 : (int)Nz]) - p.z; tz = p.z - __ldg(&zb[iz]); if (tmp < tz) tz = tmp;
        if (tx < ty) tperp = tx; else tperp = ty;
        if (tperp > tz) tperp = tz;
    } else {
        float p1x = __ldg(&xb[0]), p1y = __ldg(&yb[0]), p1z = __ldg(&zb[0]);
        float p2x = __ldg(&xb[Nx]), p2y = __ldg(&yb[Ny]), p2z = __ldg(&zb[Nz]);
        if (p.x - p1x > 0 && p.x - p2x > 0) {} else if (p.x - p1x < 0 && p.x - p2x < 0) p2x = p1x; else p2x = p.x;
        if (p.y - p1y > 0 && p.y - p2y > 0) {} else if (p.y - p1y < 0 && p.y - p2y < 0) p2y = p1y; else p2y = p.y;
        if (p.z - p1z > 0 && p.z - p2z > 0) {} else if (p.z - p1z < 0 && p.z - p2z < 0) p2z = p1z; else p2z = p.z;
        tperp = sqrtf((p.x - p2x) * (p.x - p2x) + (p.y - p2y) * (p.y - p2y) + (p.z - p2z) * (p.z - p2z));
    }
}

// ---- polygons (2-D points as float2) ----------------------------------------
// The instruction cache is the scarcest resource of the beam-line kernels: with
// each polygon test inlined and unrolled where it is used they took 80 to 280 KB
// of code and waited for instructions first of all. So each routine has one
// loop over its polygons, the loops over edges stay rolled and without
// branches, and what only few edges need (the divisions) follows for those
// edges alone, picked out by a bit mask. The photon kernels of the jaws and the
// MLC went from 97 and 83 KB to 30 and 33 KB, 50 and 62 KB with the second step
// that the warp shares (share_steps; times: electron_step).
__device__ __forceinline__ float2 ld2(const float2 *a) { return __ldg(a); }

static __device__ __noinline__ int point_in_polygon(float px, float py, const float2 *poly, int n)
{
    uint32_t cross = 0;
    float2 b = ld2(&poly[n - 1]);
#pragma unroll 2
    for (int i = 0; i < n; i++) {
        const float2 a = ld2(&poly[i]);
        if ((a.y < py) != (b.y < py) && (a.y >= py || b.y >= py) && (a.x <= px || b.x <= px)) cross |= 1u << i;
        b = a;
    }
    int odd = 0;
    while (cross) {
        const int i = __ffs(cross) - 1;
        cross &= cross - 1u;
        const float2 a = ld2(&poly[i]), c = ld2(&poly[i ? i - 1 : n - 1]);
        odd ^= (a.x + (py - a.y) / (c.y - a.y) * (c.x - a.x) < px);
    }
    return odd;
}

// The warp's way with one particle: every lane holds the same point (and ray)
// and takes one edge, so that a polygon costs one edge's time instead of the
// loop's. All 32 lanes call it; n is at most 30.
__device__ __forceinline__ int point_in_polygon_warp(float px, float py, const float2 *poly, int n)
{
    const int i = (int)(threadIdx.x & 31u);
    bool left = false;
    if (i < n) {
        const float2 a = ld2(&poly[i]), b = ld2(&poly[i ? i - 1 : n - 1]);
        if ((a.y < py) != (b.y < py) && (a.y >= py || b.y >= py) && (a.x <= px || b.x <= px))
            left = a.x + (py - a.y) / (b.y - a.y) * (b.x - a.x) < px;
    }
    return __popc(__ballot_sync(0xffffffffu, left)) & 1;
}

template <bool WARP>
__device__ __forceinline__ int in_polygon(float px, float py, const float2 *poly, int n)
{
    return WARP ? point_in_polygon_warp(px, py, poly, n) : point_in_polygon(px, py, poly, n);
}

__device__ __forceinline__ const float2 *endnode_of(const DevCtx &C, int field, int leaf)
{
    return reinterpret_cast<const float2 *>(&C.fields[field].endnode[leaf][0][0]);
}

template <bool WARP = false>
static __device__ int point_in_leaf(float2 p, const float2 *endn)
{
    int bank = 0;
    if (in_polygon<WARP>(p.x, p.y, endn, 17)) bank = 1;
    else if (in_polygon<WARP>(p.x, p.y, endn + 17, 17)) bank = 2;
    return bank;
}

template <bool WARP = false>
static __device__ __noinline__ int index_of_leaf(const DevCtx &C, float2 p)
{
    int i = GX_OUTMLC, index = GX_OUTMLC;
    float x = p.x / p.y * C.mlc_zmin;
    float z = p.y - C.mlc_zmin;
    if (z < 0 || z > C.mlc_zthick) return index;
    if (x < C.mlc_x_start || x > C.mlc_x_end) return index;
    float wt = C.mlc_wt, gap = C.mlc_air_gap;
    if (x < C.mlc_x_start + wt) i = 0;
    else if (x < C.mlc_x_mid_1 + wt) i = (int)((x - C.mlc_x_start - wt) / (C.mlc_wl_full + gap));
    else if (x < C.mlc_x_mid_2 + wt) {
        i = (int)((x - C.mlc_x_mid_1 - wt) / (C.mlc_wl_target + C.mlc_wl_isocenter + gap * 2));
        if (x - C.mlc_x_mid_1 - wt - (C.mlc_wl_target + C.mlc_wl_isocenter + gap * 2) * (float)i < C.mlc_wl_target + gap)
            i = 10 + i * 2;
        else
            i = 11 + i * 2;
    } else if (x < C.mlc_x_end - C.mlc_wl_full)
        i = (int)((x - C.mlc_x_mid_2 - wt) / (C.mlc_wl_full + gap)) + 50;
    else if (x <= C.mlc_x_end)
        i = 58;
    if (i >= 0) {
        if (in_polygon<WARP>(p.x, p.y, C.crossXZ + i * 16, 14)) index = i;
        else if (i < 59) {
            if (in_polygon<WARP>(p.x, p.y, C.crossXZ + (i + 1) * 16, 14)) index = i + 1;
            else index = -(i + 1);
        } else index = GX_OUTMLC;
    }
    return index;
}

// An edge's terms in the ray's intersection with it: the edge parameter is
// num / den, the distance dn / den (rayIntersectPolygon, geom.cu; the
// differences are taken the other way round, which changes no rounding).
__device__ __forceinline__ void ray_edge(float2 p0, float2 v, float2 a, float2 b, float &num, float &den, float &dn)
{
    const float ex = b.x - a.x, ey = b.y - a.y, dx = a.x - p0.x, dy = a.y - p0.y;
    den = v.x * ey - v.y * ex;
    num = dx * v.y - dy * v.x;
    dn = ey * dx - ex * dy;
}

// The nearest edge in front of the ray, and the parity of the edges hit. An
// edge is hit where u = fl(num / den) lies in [0, 1) and fl(dn / den) >= 0.
// First the edges for which that is possible, from the signs and sizes of num,
// den and dn alone: with d = |den| and the others carrying den's sign, n >= d
// makes u >= 1, and n or m below -d * 1e-30 makes a quotient negative that does
// not round to zero. Then the quotients of those edges, one or two of a
// polygon; u only where n is not certainly below d (1 - 2^-20).
__device__ __forceinline__ float ray_intersect_polygon(float2 p0, float2 v, const float2 *poly, int n, int &inside)
{
    uint32_t hit = 0;
    const float2 first = ld2(poly);
    float2 a = first;
#pragma unroll 2
    for (int i = 0; i < n; i++) {
        const float2 b = i + 1 < n ? ld2(&poly[i + 1]) : first;
        float num, den, dn;
        ray_edge(p0, v, a, b, num, den, dn);
        const uint32_t sign = __float_as_uint(den) & 0x80000000u;
        const float d = fabsf(den), least = d * -1e-30f;
        const float u = __uint_as_float(__float_as_uint(num) ^ sign), m = __uint_as_float(__float_as_uint(dn) ^ sign);
        if (u >= least && u < d && m >= least) hit |= 1u << i;
        a = b;
    }
    float minDist = GX_INFI_DIST + 1;
    int count = 0;
    while (hit) {
        const int i = __ffs(hit) - 1;
        hit &= hit - 1u;
        float num, den, dn;
        ray_edge(p0, v, ld2(&poly[i]), i + 1 < n ? ld2(&poly[i + 1]) : first, num, den, dn);
        const float d = fabsf(den);
        const float u = den > 0.0f ? num : -num;
        if (!(u >= 0.0f && u <= d * 0.99999904632568359375f)) {
            const float q = num / den;
            if (!(q >= 0 && q < 1)) continue;
        }
        const float dist = dn / den;
        if (dist >= 0) {
            count++;
            if (dist < minDist) minDist = dist;
        }
    }
    inside = count & 1;
    return minDist;
}

// The same by the warp: each lane decides its edge as the loop would.
__device__ __forceinline__ float ray_intersect_polygon_warp(float2 p0, float2 v, const float2 *poly, int n, int &inside)
{
    const int i = (int)(threadIdx.x & 31u);
    float dist = GX_INFI_DIST + 1;
    bool hit = false;
    if (i < n) {
        float num, den, dn;
        ray_edge(p0, v, ld2(&poly[i]), ld2(&poly[i + 1 < n ? i + 1 : 0]), num, den, dn);
        if (den != 0.0f) {
            const float q = num / den, d = dn / den;
            hit = q >= 0 && q < 1 && d >= 0;
            if (hit) dist = fabsf(d);
        }
    }
    inside = __popc(__ballot_sync(0xffffffffu, hit)) & 1;
    // distances are not negative: they order as their bits
    const float m = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(dist)));
    return m < GX_INFI_DIST + 1 ? m : GX_INFI_DIST + 1;
}

template <bool WARP>
__device__ __forceinline__ float ray_polygon(float2 p0, float2 v, const float2 *poly, int n, int &inside)
{
    return WARP ? ray_intersect_polygon_warp(p0, v, poly, n, inside) : ray_intersect_polygon(p0, v, poly, n, inside);
}

template <bool WARP = false>
static __device__ uint32_t inwhere_mlc(const DevCtx &C, int field, float qx, float qy, float qz, int &index, int &bank)
{
    uint32_t inew = 1;
    float2 p = make_float2(qx, qz);
    if (index == GX_OUTMLC) index = index_of_leaf<WARP>(C, p);
    p.x = qy;
    if (index >= 0) {
        bank = point_in_leaf<WARP>(p, endnode_of(C, field, index));
        if (bank > 0) inew = 3; else inew = 1;
    }
    return inew;
}

template <bool WARP = false>
static __device__ uint32_t howfar_mlc(const DevCtx &C, Part &p0, float &t)
{
    const Part p = p0;
    uint32_t inew = p.region;
    int bank = p.bank;
    int index = p.leafIndex;
    if (p.y < -C.mlc_rmax || p.y > C.mlc_rmax) return 0;
    const float2 p1 = make_float2(p.x, p.z), p2 = make_float2(p.y, p.z);
    const float2 dir1 = make_float2(p.u, p.w), dir2 = make_float2(p.v, p.w);
    // One polygon per turn of one loop, so that lanes with different polygons
    // intersect together and the code is there once: the MLC's bounds in XZ and
    // in YZ; then, inside them, in a leaf the leaf's XZ cross section and its
    // YZ leaf-end outline; in an air gap the XZ cross sections of the leaves
    // that the ray walks through, from the nearest, until one is hit or the
    // walk leaves the limits (each lane keeps the reference's polygons, points
    // and order).
    float dis_xz = 0.0f, dis_yz = 0.0f, minBoundaryDist = 0.0f, temp1 = GX_INFI_DIST + 1;
    float leaf_xz = 0.0f;
    int limit1 = 0, limit2 = 60, sx = 1, i = 0, inside_xz = 0;
    bool leaf = false, to_new_region = false;
    const float2 *poly = C.mlc_bounds, *yzp = nullptr;
    int n = 4, nvyz = 17;
    bool yz = false;
    for (int turn = 0;; turn++) {
        int ins;
        const float d = ray_polygon<WARP>(yz ? p2 : p1, yz ? dir2 : dir1, poly, n, ins);
        if (turn == 0) {
            dis_xz = d;
            inside_xz = ins;
            poly = C.mlc_bounds + 4;
            yz = true;
        } else if (turn == 1) {
            dis_yz = d;
            if (dis_xz >= GX_INFI_DIST || dis_yz >= GX_INFI_DIST) return 0;
            minBoundaryDist = dis_xz < dis_yz ? dis_xz : dis_yz;
            if (!(inside_xz && ins)) {
                if (!(t > minBoundaryDist)) return 0;
                inew = 0;
                t = minBoundaryDist + GX_EPSTEP;
                to_new_region = true;
                break;
            }
            if (p.leafIndex <= -60) index = index_of_leaf<WARP>(C, p1);
            if (index <= -60) break;
            leaf = index >= 0;
            yz = false;
            n = 14;
            if (leaf) {
                poly = C.crossXZ + index * 16;
                yzp = endnode_of(C, p.field, index);
                if (p.bank == 0) { yzp += 2; nvyz = 30; }
                else if (p.bank == 2) yzp += 17;
            } else {
                // the leaf (or gap) where the ray leaves the MLC; in double, as geom.cu:591
                const float2 p3 = make_float2(p1.x + dis_xz * dir1.x, p1.y + (dis_xz - 0.001) * dir1.y);
                limit1 = index_of_leaf<WARP>(C, p3);
                if (limit1 < 0) limit1 = -limit1;
                if (dir1.x < 0) { sx = -1; if (limit1 > 0) limit1 -= 1; limit2 = -index + 1; }
                else { limit2 = limit1; limit1 = -index - 1; }
                i = -index - sx;
                if (limit1 < 0) limit1 = 0;
                if (limit2 > 59) limit2 = 59;
                if (i < 0) i = 0;
                if (i > 59) i = 59;
                poly = C.crossXZ + i * 16;
            }
        } else if (leaf) {
            if (turn == 3) { dis_xz = leaf_xz; dis_yz = d; break; }
            leaf_xz = d;
            poly = yzp;
            n = nvyz;
            yz = true;
        } else {
            temp1 = d;
            i += sx;
            poly += 16 * sx;
            if (!(i >= limit1 && i <= limit2 && temp1 >= GX_INFI_DIST)) break;
            if (WARP) {
                // the rest of the walk, a leaf to a lane: the first that is hit ends it
                for (; i >= limit1 && i <= limit2; i += 32 * sx) {
                    const int j = i + sx * (int)(threadIdx.x & 31u);
                    float dj = GX_INFI_DIST + 1;
                    if (j >= limit1 && j <= limit2) dj = ray_intersect_polygon(p1, dir1, C.crossXZ + 16 * j, 14, ins);
                    const unsigned hit = __ballot_sync(0xffffffffu, dj < GX_INFI_DIST);
                    if (hit) {
                        const int k = __ffs(hit) - 1;
                        temp1 = __shfl_sync(0xffffffffu, dj, k);
                        i += sx * (k + 1);
                        break;
                    }
                }
                break;
            }
        }
    }
    if (!to_new_region) {
        if (index > -60) {
            if (leaf) {
                if (dis_yz > dis_xz) {
                    if (dir1.x < 0 && index > 0) index = -index;
                    else if (index < 59) index = -(index + 1);
                }
            } else if (temp1 < dis_xz) {
                dis_xz = temp1;
                index = i - sx;
            } else {
                index = GX_PASSMLC;
                p0.module = (uint8_t)C.module_order[GEGS_M_VARMLC];
            }
        }
        float minDist = dis_xz < dis_yz ? dis_xz : dis_yz;
        bool steppingOut = false;
        if ((minDist + GX_EPSTEP) >= minBoundaryDist) { minDist = minBoundaryDist; steppingOut = true; }
        if (t > minDist) {
            t = minDist + GX_EPSTEP;
            if (steppingOut) {
                p0.leafIndex = GX_PASSMLC;
                p0.module = (uint8_t)C.module_order[GEGS_M_VARMLC];
                return 1;
            }
        } else return inew;
    }
    float qx = p.x + t * p.u, qy = p.y + t * p.v, qz = p.z + t * p.w;
    inew = inwhere_mlc<WARP>(C, p.field, qx, qy, qz, index, bank);
    p0.leafIndex = (int8_t)index;
    p0.bank = (int8_t)bank;
    return inew;
}

__device__ __forceinline__ const float2 *fpoly(const float (*a)[2]) { return reinterpret_cast<const float2 *>(a); }

// The polygons of one pair of jaws: bounding polygons, and the opening with the
// two jaws around it (the opening is the polygon from vertex 2, the jaws those
// from vertices 0 and 4).
struct JawPolys { const float2 *bmax, *bmin, *geom; };

__device__ __forceinline__ JawPolys jaw_polys(const DevCtx &C, int field, bool xjaw)
{
    const gegs_field *F = &C.fields[field];
    JawPolys j;
    j.bmax = fpoly(xjaw ? F->boundMaxX : F->boundMaxY);
    j.bmin = fpoly(xjaw ? F->boundMinX : F->boundMinY);
    j.geom = fpoly(xjaw ? F->jawsGeomX : F->jawsGeomY);
    return j;
}

// howfar_SecJawsY and howfar_SecJawsX (geom.cu:793-1035) in one: the Y jaws
// open in x, the X jaws in y. The reference's X routine steps to the opening
// from the tungsten by the distance to the bounds in YZ; kept.
template <bool WARP = false>
static __device__ uint32_t howfar_secjaws(const DevCtx &C, Part &p, float &t)
{
    const bool xjaw = p.module == GEGS_M_SECJAWX;
    const JawPolys J = jaw_polys(C, p.field, xjaw);
    const float2 p1 = make_float2(p.y, p.z), p2 = make_float2(p.x, p.z);
    const float2 dir1 = make_float2(p.v, p.w), dir2 = make_float2(p.u, p.w);
    const float2 q = xjaw ? p1 : p2, dq = xjaw ? dir1 : dir2;
    float dis_xz = 0.0f, dis_yz = 0.0f, minBoundaryDist = 0.0f, jaw0 = 0.0f, d;
    int inside_xz = 0, ins;
    bool open = false;
    // outside the bounds: to them, and what lies behind
    auto from_outside = [&]() -> uint32_t {
        if (!(t > minBoundaryDist)) return 1;
        t = minBoundaryDist + GX_EPSTEP;
        const float y = p.y + t * p.v, x = p.x + t * p.u;
        if (!in_polygon<WARP>(y, x, J.bmin, 4)) return 0;
        return in_polygon<WARP>(xjaw ? y : x, p.z + t * p.w, J.geom + 2, 4) ? 1 : 2;
    };
    if (WARP) {
        // all polygons at once, four lanes to each: the bounds seen from (y, z) and
        // from (x, z), the two jaws, the opening, and the point in the opening
        const int k = (int)(threadIdx.x & 31u) >> 2, i = (int)threadIdx.x & 3;
        const float2 o = k == 0 ? p1 : k == 1 ? p2 : q, v = k == 0 ? dir1 : k == 1 ? dir2 : dq;
        const float2 *poly = k < 2 ? J.bmax : J.geom + (k == 2 ? 0 : k == 3 ? 4 : 2);
        const float2 a = ld2(&poly[i]), b = ld2(&poly[(i + 1) & 3]);
        float num, den, dn, dist = GX_INFI_DIST + 1;
        ray_edge(o, v, a, b, num, den, dn);
        bool hit = false;
        if (k == 5) {
            if ((a.y < q.y) != (b.y < q.y) && (a.y >= q.y || b.y >= q.y) && (a.x <= q.x || b.x <= q.x))
                hit = b.x + (q.y - b.y) / (a.y - b.y) * (a.x - b.x) < q.x;   // the edge that ends at b, as point_in_polygon takes it
        } else if (k < 5 && den != 0.0f) {
            const float u = num / den, e = dn / den;
            hit = u >= 0 && u < 1 && e >= 0;
            if (hit) dist = fminf(fabsf(e), GX_INFI_DIST + 1);
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        dist = fminf(dist, __shfl_xor_sync(0xffffffffu, dist, 1));
        dist = fminf(dist, __shfl_xor_sync(0xffffffffu, dist, 2));
        dis_xz = __shfl_sync(0xffffffffu, dist, 0);
        dis_yz = __shfl_sync(0xffffffffu, dist, 4);
        if (dis_xz >= GX_INFI_DIST || dis_yz >= GX_INFI_DIST) return 0;
        minBoundaryDist = dis_xz < dis_yz ? dis_xz : dis_yz;
        if (!((__popc(hits & 0xfu) & 1) && (__popc(hits & 0xf0u) & 1))) return from_outside();
        open = __popc(hits & 0xf00000u) & 1;
        jaw0 = __shfl_sync(0xffffffffu, dist, 8);
        d = open ? __shfl_sync(0xffffffffu, dist, 12) : __shfl_sync(0xffffffffu, dist, 16);
    } else {
        // one polygon per turn: the bounds seen from (y, z) and from (x, z); then
        // from the opening the two jaws around it, from a jaw the opening
        float2 o = p1, v = dir1;
        const float2 *poly = J.bmax;
        for (int turn = 0;; turn++) {
            d = ray_intersect_polygon(o, v, poly, 4, ins);
            if (turn == 0) {
                dis_xz = d;
                inside_xz = ins;
                o = p2;
                v = dir2;
            } else if (turn == 1) {
                dis_yz = d;
                if (dis_xz >= GX_INFI_DIST || dis_yz >= GX_INFI_DIST) return 0;
                minBoundaryDist = dis_xz < dis_yz ? dis_xz : dis_yz;
                if (!(inside_xz && ins)) return from_outside();
                open = point_in_polygon(q.x, q.y, J.geom + 2, 4);
                o = q;
                v = dq;
                poly = open ? J.geom : J.geom + 2;
            } else if (turn == 2 && open) {
                jaw0 = d;
                poly = J.geom + 4;
            } else break;
        }
    }
    if (open) {
        const float jaw = jaw0 < GX_INFI_DIST ? jaw0 : d;
        if (jaw < GX_INFI_DIST) {
            if (t > jaw) { t = jaw + GX_EPSTEP; return 2; }
        } else if (t > minBoundaryDist) {
            t = minBoundaryDist + GX_EPSTEP;
            p.module = (uint8_t)C.module_order[xjaw ? GEGS_M_SECJAWX : GEGS_M_SECJAWY];
        }
        return 1;
    }
    if (d < GX_INFI_DIST) {
        if (t > d) { t = (xjaw ? dis_yz : d) + GX_EPSTEP; return 1; }
    } else if (t > minBoundaryDist) {
        t = minBoundaryDist + GX_EPSTEP;
        return 0;
    }
    return 2;
}

// ---- hownear -----------------------------------------------------------------
__device__ __forceinline__ float dist2p(float2 v, float2 w) { return (v.x - w.x) * (v.x - w.x) + (v.y - w.y) * (v.y - w.y); }

// Squared distance whose sqrtf is point_dist_to_segment(p, v, w), term for term.
__device__ __forceinline__ float point_dist2_to_segment(float2 p, float2 v, float2 w)
{
    float l2 = dist2p(v, w);
    if (l2 == 0) return dist2p(p, v);
    float tn = (p.x - v.x) * (w.x - v.x) + (p.y - v.y) * (w.y - v.y);
    // t = fl(tn / l2) with l2 > 0: certainly negative (and not rounded to zero)
    // below -l2 * 1e-30, certainly above 1 beyond l2 * (1 + 2^-20); only the
    // projection case needs the quotient itself
    if (tn < -l2 * 1e-30f) return dist2p(p, v);
    if (tn > l2 * 1.00000095367431640625f) return dist2p(p, w);
    float t = tn / l2;
    if (t < 0) return dist2p(p, v);
    if (t > 1) return dist2p(p, w);
    float2 a = make_float2(v.x + t * (w.x - v.x), v.y + t * (w.y - v.y));
    return dist2p(p, a);
}

// What an electron step does with hownear: compares it with the range (where
// range rejection is on) and with the step tustep, which it limits when it is
// smaller. A value known to within a slack often decides that, and then stands
// in for the exact one.
struct NearUse { bool rr; float range, tustep; };

__device__ __forceinline__ NearUse near_exactly()
{
    NearUse u;
    u.rr = false; u.range = 0.0f; u.tustep = __int_as_float(0x7f800000);
    return u;
}

// lo <= hownear <= hi: is the step's outcome (beyond the range; or within it
// and beyond tustep) certain?
__device__ __forceinline__ bool near_decided(const NearUse &u, float lo, float hi)
{
    return u.rr ? lo > u.range || (lo > u.tustep && hi < u.range) : lo > u.tustep;
}

// Squared distances to the polygon's edges, without their roundings: lowers
// `best` to the smallest and marks the edges that come within `slack` (cm) of
// the smallest found so far, which include every edge whose exact distance can
// be the smallest. (sqrt(m) + s)^2 <= m (1 + s) + s + s^2.
__device__ __forceinline__ void near_edges(float2 p0, const float2 *poly, int n, float slack, float &best, uint32_t &cand)
{
    cand = 0;
    const float grow = 1.0f + slack, add = slack + slack * slack;
    const float2 first = ld2(poly);
    float2 a = first;
#pragma unroll 2
    for (int i = 0; i < n; i++) {
        const float2 b = i + 1 < n ? ld2(&poly[i + 1]) : first;
        const float ex = b.x - a.x, ey = b.y - a.y, dx = p0.x - a.x, dy = p0.y - a.y;
        const float t = __saturatef(__fdividef(__fmaf_rn(dx, ex, dy * ey), __fmaf_rn(ex, ex, ey * ey)));
        const float rx = __fmaf_rn(-t, ex, dx), ry = __fmaf_rn(-t, ey, dy);
        const float d2 = __fmaf_rn(rx, rx, ry * ry);
        if (d2 <= __fmaf_rn(best, grow, add)) cand |= 1u << i;
        best = fminf(best, d2);
        a = b;
    }
}

// Exact distance to the polygon (pointMinDistToPolygon, geom.cu:1175-1191,
// capped at 1e9) from its marked edges; infinite without any. sqrtf is
// correctly rounded and monotonic, so the root of the smallest square is the
// smallest root.
__device__ __forceinline__ float near_exact(float2 p0, const float2 *poly, int n, uint32_t cand)
{
    float min2 = __int_as_float(0x7f800000);
    while (cand) {
        const int i = __ffs(cand) - 1;
        cand &= cand - 1u;
        const float d2 = point_dist2_to_segment(p0, ld2(&poly[i]), ld2(&poly[i + 1 < n ? i + 1 : 0]));
        if (d2 < min2) min2 = d2;
    }
    const float d = sqrtf(min2);
    return d < 1e9f ? d : 1e9f;
}

// How far near_edges can be from the exact distance, as computed in float: some
// 1e-6 of the coordinates and of the polygons' extent (C.near_slack holds 10 um
// and 1e-5 of the latter).
__device__ __forceinline__ float near_error(const DevCtx &C, const Part &p)
{
    return C.near_slack + 1e-5f * (fabsf(p.x) + fabsf(p.y) + fabsf(p.z));
}

static __device__ void hownear_mlc(const DevCtx &C, Part &p, float &tperp, const NearUse &use)
{
    const float2 p1 = make_float2(p.x, p.z), p2 = make_float2(p.y, p.z);
    const float err = near_error(C, p);
    // Two polygons in every case, one per turn, so that the lanes of all cases
    // share the loops: outside the MLC its bounds in XZ and in YZ; in a leaf
    // column the leaf's XZ cross section and its YZ leaf-end outline; in an air
    // gap the XZ cross sections of the leaves on either side.
    const float2 *poly0 = C.mlc_bounds, *poly1 = C.mlc_bounds + 4;
    int n0 = 4, n1 = 4;
    bool second_yz = true, gap = false;
    bool inside = true;
    if (p.leafIndex < -60)
        inside = point_in_polygon(p1.x, p1.y, C.mlc_bounds, 4) && point_in_polygon(p2.x, p2.y, C.mlc_bounds + 4, 4);
    if (inside) {
        int index;
        if (p.leafIndex > GX_PASSMLC) index = p.leafIndex;
        else { index = index_of_leaf(C, p1); p.leafIndex = (int8_t)index; }
        if (index <= -60) { tperp = GX_INFI_DIST + 1; return; }
        if (index >= 0) {
            const float2 *yzp = endnode_of(C, p.field, index);
            if (p.bank < 0) p.bank = (int8_t)point_in_leaf(p2, yzp);
            poly0 = C.crossXZ + index * 16;
            poly1 = yzp + (p.bank == 0 ? 2 : p.bank == 2 ? 17 : 0);
            n1 = p.bank == 0 ? 30 : 17;
        } else {
            gap = true;
            second_yz = false;
            poly0 = C.crossXZ + -index * 16;
            poly1 = C.crossXZ + (-index - 1) * 16;
            n1 = 14;
        }
        n0 = 14;
    }
    float best = 1e30f;
    uint32_t cand0 = 0, cand1 = 0;
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        cand0 = cand1;
        near_edges(k && second_yz ? p2 : p1, k ? poly1 : poly0, k ? n1 : n0, 2.0f * err, best, cand1);
    }
    const float d = sqrtf(best);
    if (near_decided(use, d - err, d + err)) { tperp = d - err; return; }
    tperp = gap ? GX_INFI_DIST + 1 : __int_as_float(0x7f800000);
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const float e = near_exact(k && second_yz ? p2 : p1, k ? poly1 : poly0, k ? n1 : n0, k ? cand1 : cand0);
        if (e < tperp) tperp = e;
    }
}

// hownear_SecJawsY and hownear_SecJawsX (geom.cu:1288-1374) in one: distances to
// the bounding polygon seen from (y, z) and from (x, z), and to the opening.
static __device__ void hownear_secjaws(const DevCtx &C, const Part &p, float &tperp)
{
    const bool xjaw = p.module == GEGS_M_SECJAWX;
    const JawPolys J = jaw_polys(C, p.field, xjaw);
    const float err = near_error(C, p);
    const float2 p1 = make_float2(p.y, p.z), p2 = make_float2(p.x, p.z);
    float d0 = 0.0f, d1 = 0.0f, d2 = 0.0f;
    int in0 = 0, in1 = 0, in2 = 0;
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
        const float2 o = k == 0 || (k == 2 && xjaw) ? p1 : p2;
        const float2 *poly = k < 2 ? J.bmax : J.geom + 2;
        float best = 1e30f;
        uint32_t cand;
        near_edges(o, poly, 4, 2.0f * err, best, cand);
        d0 = d1; d1 = d2; d2 = near_exact(o, poly, 4, cand);
        in0 = in1; in1 = in2; in2 = point_in_polygon(o.x, o.y, poly, 4);
    }
    const float along = xjaw ? d1 : d0, across = xjaw ? d0 : d1;
    if (in0 && in1) {
        float d = d2;
        if (!in2 && d > across) d = across;
        tperp = d < along ? d : along;
    } else tperp = d0 < d1 ? d0 : d1;
}

// Lower bound on hownear_secjaws: its result is a minimum over
// distances to some of three (point, polygon) pairs -- the bounding polygon
// seen from (y, z) and from (x, z), and the jaw opening seen from (x, z) for
// the Y jaws or from (y, z) for the X jaws -- and a distance to a polygon is
// at least the distance to the line of its nearest edge. 10 um covers the
// rounding of both sides at coordinates up to 100 cm (a few 1e-5 cm). Every
// lane evaluates the same twelve lines, so a warp whose steps are all shorter
// than the bound skips the exact polygon distances as a whole.
__device__ __forceinline__ float jaws_near_lower_bound(const DevCtx &C, const Part &p)
{
    const bool xjaw = p.module == GEGS_M_SECJAWX;
    const float4 *L = C.jaw_lines + ((size_t)p.field * 2 + (xjaw ? 1 : 0)) * 8;
    float m = __int_as_float(0x7f7fffff);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float4 l = __ldg(&L[k]);
        m = fminf(m, fabsf(l.x * p.y + l.y * p.z - l.z));
        m = fminf(m, fabsf(l.x * p.x + l.y * p.z - l.z));
    }
    const float qx = xjaw ? p.y : p.x;
#pragma unroll
    for (int k = 4; k < 8; k++) {
        const float4 l = __ldg(&L[k]);
        m = fminf(m, fabsf(l.x * qx + l.y * p.z - l.z));
    }
    return m - 1e-3f;
}

// dispatch on the particle's module (photon.cu:142-158, electron.cu:1491-1508)
__device__ __forceinline__ uint32_t howfar(const DevCtx &C, Part &p, float &t, bool &ok)
{
    ok = true;
    switch (p.module) {
    case GEGS_M_PHANTOM: return howfar_phantom(C, p, t);
    case GEGS_M_VARMLC: return howfar_mlc(C, p, t);
    case GEGS_M_SECJAWY:
    case GEGS_M_SECJAWX: return howfar_secjaws(C, p, t);
    default: ok = false; return 0;
    }
}

__device__ __forceinline__ void hownear(const DevCtx &C, Part &p, float &tperp, bool &ok)
{
    ok = true;
    switch (p.module) {
    case GEGS_M_PHANTOM: hownear_phantom(C, p, tperp); return;
    case GEGS_M_VARMLC: hownear_mlc(C, p, tperp, near_exactly()); return;
    case GEGS_M_SECJAWY:
    case GEGS_M_SECJAWX: hownear_secjaws(C, p, tperp); return;
    default: ok = false; tperp = 0; return;
    }
}

// Geometry classes: a consumer kernel compiled for one class contains only that
// class's geometry code -- the secondary jaws, the MLC, or the phantom voxels --
// which keeps the code a divergent warp runs small. Classes are numbered in beam
// order; a particle whose module is outside the class is handed to the other
// class's kernel between steps. GX_GEOM_ALL compiles every module (plain form).
#define GX_GEOM_ALL 0
#define GX_GEOM_JAWS 1
#define GX_GEOM_MLC 2
#define GX_GEOM_PHANTOM 3

// class of a module (unsupported modules fall in the jaws class, whose
// geometry dispatch reports them)
__device__ __forceinline__ int geom_class_of(uint8_t module)
{
    if (module == GEGS_M_PHANTOM) return GX_GEOM_PHANTOM;
    if (module == GEGS_M_VARMLC) return GX_GEOM_MLC;
    return GX_GEOM_JAWS;
}

template <int G>
__device__ __forceinline__ bool in_geom_class(const Part &p)
{
    return G == GX_GEOM_ALL || geom_class_of(p.module) == G;
}

template <int G, bool WARP = false>
__device__ __forceinline__ uint32_t howfar_g(const DevCtx &C, Part &p, float &t, bool &ok)
{
    if (G == GX_GEOM_ALL) return howfar(C, p, t, ok);
    ok = true;
    if (G == GX_GEOM_PHANTOM) {
        if (p.module == GEGS_M_PHANTOM) return howfar_phantom(C, p, t);
    } else if (G == GX_GEOM_MLC) {
        if (p.module == GEGS_M_VARMLC) return howfar_mlc<WARP>(C, p, t);
    } else {
        if (p.module == GEGS_M_SECJAWY || p.module == GEGS_M_SECJAWX) return howfar_secjaws<WARP>(C, p, t);
    }
    ok = false;
    return 0;
}

// Distance to the nearest boundary, as far as `use` needs it.
template <int G>
__device__ __forceinline__ void hownear_g(const DevCtx &C, Part &p, float &tperp, bool &ok, const NearUse &use)
{
    if (G == GX_GEOM_ALL) { hownear(C, p, tperp, ok); return; }
    ok = true;
    if (G == GX_GEOM_PHANTOM) {
        if (p.module == GEGS_M_PHANTOM) { hownear_phantom(C, p, tperp); return; }
    } else if (G == GX_GEOM_MLC) {
        if (p.module == GEGS_M_VARMLC) { hownear_mlc(C, p, tperp, use); return; }
    } else {
        if (p.module == GEGS_M_SECJAWY || p.module == GEGS_M_SECJAWX) {
            tperp = jaws_near_lower_bound(C, p);
            if (near_decided(use, tperp, __int_as_float(0x7f800000))) return;
            hownear_secjaws(C, p, tperp);
            return;
        }
    }
    ok = false;
    tperp = 0;
}
