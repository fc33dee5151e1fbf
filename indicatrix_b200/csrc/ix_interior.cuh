// ix_interior.cuh -- the slab scan of a ray that starts inside the stone, for a converged
// warp: four 8-lane groups, each with its own ray.
#pragma once

#include "ix_transport.cuh"

namespace ix {

// ------------------------------------------------------------------------------------
// A ray whose origin is strictly inside every plane (each one after a path's entry): no
// plane can make an entry or a miss, so the hit is the smallest t = -side / denom over the
// planes with denom > 1e-7, and only the winner needs its IEEE quotient.  Each plane gets
// u = denom * rcp(side), about -1 / t, whose low 7 mantissa bits then carry the plane's
// index, so one minimum finds value and plane at once (receding planes are positive and
// never count).  The second smallest is kept beside it: a winner ahead of it by two units
// of 2^-16 relative -- the reciprocal, the product and the replaced bits err by less than
// one -- is the plane the exact scan keeps, whatever the rounding.  Everything else (a
// closer second, an origin on, outside or within 1e-20 of a plane, no candidate, a winner the
// exact scan would pass over) is undecided and takes the exact scan.  The 1e-20 keeps every
// key finite for normals up to 1e18: nearer than that the reciprocal overflows (a subnormal
// side is flushed before it), and infinity with an index in its low bits is a NaN that the
// minimum passes over.
//
// The planes come as pairs (i, i + 8) of a block of 16 in shared memory, lane c reading
// pair c of each block, so that the packed f32x2 units form both planes' dot products:
// about 10 instructions a plane and no branch, against 20 to 30 of the exact scan, whose
// lanes divide under a branch.  Padding planes (0, 0, 0, -1e30) have u = 0.
// ------------------------------------------------------------------------------------
constexpr int PAIR_WORDS = 8;  // x, x', y, y', z, z', w, w'
constexpr int PLANE_PAIR_VECS = IX_MAX_PLANES / 2 * PAIR_WORDS / 4;  // float4s of a full set
static_assert(IX_MAX_PLANES <= 128, "7 index bits");

// A plane's n . d in the reference's order, every rounding written out as the exact scan's
// source compiles: the fast build fuses where the compiler's contraction does.
IX_DEV float plane_denom(float4 p, V3 d) {
#if IX_EXACT
    return __fadd_rn(__fadd_rn(__fmul_rn(p.x, d.x), __fmul_rn(p.y, d.y)), __fmul_rn(p.z, d.z));
#else
    return fmaf(p.z, d.z, fmaf(p.x, d.x, __fmul_rn(p.y, d.y)));
#endif
}
IX_DEV float plane_side(float4 p, V3 o) { return __fadd_rn(p.w, plane_denom(p, o)); }

#if IX_EXACT
#define IX_F2(op) op ".rn.f32x2"
#else
#define IX_F2(op) op ".rn.ftz.f32x2"
#endif
typedef unsigned long long F2;
IX_DEV F2 f2_both(float v) {
    F2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
IX_DEV void f2_split(F2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a)); }
IX_DEV F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm(IX_F2("mul") " %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
IX_DEV F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm(IX_F2("add") " %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
IX_DEV F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm(IX_F2("fma") " %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// plane_denom of two planes, with its roundings.
IX_DEV F2 f2_denom(F2 px, F2 py, F2 pz, F2 x, F2 y, F2 z) {
#if IX_EXACT
    return f2_add(f2_add(f2_mul(px, x), f2_mul(py, y)), f2_mul(pz, z));
#else
    return f2_fma(pz, z, f2_fma(px, x, f2_mul(py, y)));
#endif
}
IX_DEV float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Writes planes [0, n) into `rows` and as padded pairs into `pairs`, `nt` threads together.
IX_DEV void stage_planes(const float4* __restrict__ src, int n, float4* rows, float4* pairs, int tid, int nt) {
    const int padded = (n + 15) & ~15;
    for (int i = tid; i < padded; i += nt) {
        const float4 p = i < n ? src[i] : make_float4(0.0f, 0.0f, 0.0f, -1e30f);
        if (i < n) rows[i] = p;
        float* f = reinterpret_cast<float*>(pairs) + ((i >> 4) * 8 + (i & 7)) * PAIR_WORDS + ((i >> 3) & 1);
        f[0] = p.x;
        f[2] = p.y;
        f[4] = p.z;
        f[6] = p.w;
    }
}
// The whole warp calls it, converged.  False: undecided.
IX_DEV bool warp_interior_hit(const float4* __restrict__ rows, const float4* __restrict__ pairs, int n, V3 o, V3 d,
                              Hit& hit) {
    const int c = (int)(threadIdx.x & 7u);
    const F2 ox = f2_both(o.x), oy = f2_both(o.y), oz = f2_both(o.z);
    const F2 dx = f2_both(d.x), dy = f2_both(d.y), dz = f2_both(d.z);
    float u1 = 0.0f, u2 = 0.0f;  // the two smallest keys
    float most = -1.0f;          // the largest side
    const ulonglong2* q = reinterpret_cast<const ulonglong2*>(pairs) + 2 * c;
    auto key = [](float u, uint32_t i) { return __uint_as_float((__float_as_uint(u) & ~127u) | i); };
#pragma unroll 2
    for (uint32_t i = 0; i < (uint32_t)n; i += 16, q += 16) {
        const ulonglong2 xy = q[0], zw = q[1];
        const F2 side = f2_add(zw.y, f2_denom(xy.x, xy.y, zw.x, ox, oy, oz));
        const F2 denom = f2_denom(xy.x, xy.y, zw.x, dx, dy, dz);
        float s0, s1, n0, n1;
        f2_split(side, s0, s1);
        f2_split(denom, n0, n1);
        most = fmaxf(most, fmaxf(s0, s1));
        const float a = key(n0 * rcp_approx(s0), i), b = key(n1 * rcp_approx(s1), i + 8u);
        const float lo = fminf(a, b), hi = fmaxf(a, b);
        u2 = fminf(fminf(u2, hi), fmaxf(u1, lo));
        u1 = fminf(u1, lo);
    }
    u1 = most < -1e-20f ? __uint_as_float(__float_as_uint(u1) | (uint32_t)c) : -INFINITY;
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) {
        const float o1 = __shfl_xor_sync(WARP_MASK, u1, m), o2 = __shfl_xor_sync(WARP_MASK, u2, m);
        u2 = fminf(fminf(u2, o2), fmaxf(u1, o1));
        u1 = fminf(u1, o1);
    }
    const uint32_t k1 = __float_as_uint(u1) & 0x7FFFFFFFu, k2 = __float_as_uint(u2) & 0x7FFFFFFFu;
    if (!(u1 < -1e-30f && u1 > -1e30f) || (k1 >> 7) - (k2 >> 7) < 2u) return false;
    const int idx = (int)(k1 & 127u);
    const float4 p = rows[idx];
    const float denom = plane_denom(p, d), side = plane_side(p, o);
    if (!(denom > 1e-7f) || !(side < 0.0f)) return false;
    const float t = __fdiv_rn(-side, denom);
    hit.facet = t > 1e-4f ? idx : -1;
    hit.t = t > 1e-4f ? t : 0.0f;
    return true;
}
// The exact scan of four rays (group_intersect under the full mask).
IX_DEV Hit warp_exact_hit(const float4* __restrict__ rows, int n, V3 o, V3 d) {
    return group_intersect(warp_group(), rows, n, o, d);
}

}  // namespace ix
