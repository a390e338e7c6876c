// rt_traverse.cuh - ray traversal of the compressed 8-wide BVH.
//
// Replaces optixTrace (core/cuda/devicePrograms.cu:258-269 closest hit,
// :303-319 terminate-on-first-hit shadow rays).  Traversal follows Ylitie,
// Karras and Laine, "Efficient Incoherent Ray Traversal on GPUs Through
// Compressed Wide BVHs" (HPG 2017): a node is read as five 16-byte loads, its
// eight quantised child boxes are tested at once, and the hits become a
// 32-bit group mask (bits 24..31 internal children in near-to-far order,
// bits 0..23 triangles) kept on a short per-thread stack.  Triangles use the
// watertight test of Woop, Benthin and Wald (JCGT 2013).
#pragma once

#include <cuda_fp16.h>

#include "rt_device.cuh"

namespace rtd {

struct TravRay {
    v3 o, d;
    float tmin, tmax;
    v3 idir;        // 1 / d with tiny components clamped
    uint32_t oct;   // bit a set when d[a] < 0 (as idir[a] is): slot index of the nearest child
    int kx, ky, kz; // watertight shear axes
    float Sx, Sy, Sz;
};

RT_D void prepare_ray(TravRay& r) {
    const float tiny = 1e-20f;
    float dx = fabsf(r.d.x) > tiny ? r.d.x : (r.d.x < 0.0f ? -tiny : tiny);
    float dy = fabsf(r.d.y) > tiny ? r.d.y : (r.d.y < 0.0f ? -tiny : tiny);
    float dz = fabsf(r.d.z) > tiny ? r.d.z : (r.d.z < 0.0f ? -tiny : tiny);
    r.idir = v3(1.0f / dx, 1.0f / dy, 1.0f / dz);
    r.oct = (r.d.x < 0.0f ? 1u : 0u) | (r.d.y < 0.0f ? 2u : 0u) | (r.d.z < 0.0f ? 4u : 0u);
    float ax = fabsf(r.d.x), ay = fabsf(r.d.y), az = fabsf(r.d.z);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz == 2 ? 0 : kz + 1;
    int ky = kx == 2 ? 0 : kx + 1;
    float dkz = r.d[kz];
    if (dkz < 0.0f) {
        int t = kx;
        kx = ky;
        ky = t;
    }
    r.kx = kx;
    r.ky = ky;
    r.kz = kz;
    r.Sx = __fdiv_rn(r.d[kx], dkz);
    r.Sy = __fdiv_rn(r.d[ky], dkz);
    r.Sz = __fdiv_rn(1.0f, dkz);
}

RT_D float comp(v3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

// Watertight ray/triangle test.  Products are rounded individually (no FMA
// contraction) so the edge functions match a plain FP32 evaluation.  The
// distance range is tested on the unnormalised T against tmin/tmax * |det|;
// the one division happens only for an accepted hit.
RT_D bool intersect_tri(const TravRay& r, float4 a, float4 b, float4 c, float tmax, float& t, float& b1, float& b2) {
    v3 A = v3(a.x, a.y, a.z) - r.o, B = v3(b.x, b.y, b.z) - r.o, C = v3(c.x, c.y, c.z) - r.o;
    float Akz = comp(A, r.kz), Bkz = comp(B, r.kz), Ckz = comp(C, r.kz);
    float Ax = __fsub_rn(comp(A, r.kx), __fmul_rn(r.Sx, Akz)), Ay = __fsub_rn(comp(A, r.ky), __fmul_rn(r.Sy, Akz));
    float Bx = __fsub_rn(comp(B, r.kx), __fmul_rn(r.Sx, Bkz)), By = __fsub_rn(comp(B, r.ky), __fmul_rn(r.Sy, Bkz));
    float Cx = __fsub_rn(comp(C, r.kx), __fmul_rn(r.Sx, Ckz)), Cy = __fsub_rn(comp(C, r.ky), __fmul_rn(r.Sy, Ckz));
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    float Az = __fmul_rn(r.Sz, Akz), Bz = __fmul_rn(r.Sz, Bkz), Cz = __fmul_rn(r.Sz, Ckz);
    float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    const float adet = fabsf(det);
    const float sT = det < 0.0f ? -T : T;
    if (!(sT > 0.99999f * r.tmin * adet && sT < 1.00001f * tmax * adet)) return false;
    float inv = __fdiv_rn(1.0f, det);
    float tt = __fmul_rn(T, inv);
    if (!(tt > r.tmin && tt < tmax)) return false;
    t = tt;
    b1 = __fmul_rn(V, inv);
    b2 = __fmul_rn(W, inv);
    return true;
}

// Three-input minimum / maximum (PTX ISA 8.8, sm_100).
RT_D float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
RT_D float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Two half-precision lanes in a register.
RT_D uint32_t half2_of(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
RT_D uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
RT_D uint32_t hfma2_relu(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
RT_D uint32_t hle2_mask(uint32_t a, uint32_t b) {  // 0xFFFF in the lanes with a <= b
    return __hle2_mask(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
}

// Tests the eight children of `node` against the ray over [r.tmin, tmax];
// returns the mask of the slots it may meet (bit s: slot s).
//
// Two children at a time in half precision.  The planes' distances are taken
// relative to t0, where the ray enters the node (or tmin), and scaled by a
// power of two k, so that the longest of the three slabs spans 0.25..0.5: a
// plane byte q is the subnormal half q * 2^-24 as it stands, and its distance
// one fma with S = 2^24 k s (s: distance of one quantisation step) and
// C = k c (c: distance of the node's origin from t0).  The near distances are
// compared as 16-bit integers, in which non-negative halves order like their
// values and any negative one is below them; the x distance is clamped at 0
// (the entry), which is what makes the nearest of three non-negative.
//
// Conservative: S, C and the fma round to 11 bits, of at most |q S| <= 255 |s|,
// |C| <= 255 |s| and the result, 3 * 255 * 2^-11 = 0.374 quantisation steps
// together (plus 2^-25 each where they are subnormal); the single-precision
// distances are off by at most 2^-21 (|t0| + 255 |s|).  So near planes move in
// and far planes out by E = 0.4 |s| k + 2^-21 |t0| k + 2^-23.
// An axis along which the ray hardly moves has a slab so long that the other
// two would lose their precision: past 2^10 times the shortest, its distances
// are scaled down to that length.  That keeps every box the ray meets: signs
// stay, near planes only come nearer, and a far plane ahead by 0.25 steps or
// more, which is added to E there, stays beyond the shortest slab's end, where
// the ray has left the node.  (c / |s| comes first there: lim / |s| can fall
// below the smallest float.)  Distances beyond 1e30 report every slot.
// Long directions (queries ask for no unit length) make short distances: k is
// bounded (mx >= 2^-102), so that 2^24 k stays a float and a step below 2^-126,
// which single precision flushes to zero, puts a plane off by at most
// 255 * 2^-126 k = 2^-26, within E.  Slabs of less than 2^-114 lose precision
// for it, and below 2^-115 every slot is reported: at 2^-118 the flushed steps
// leave nothing to tell the planes apart by.
RT_D uint32_t intersect_children(const CwNode* nodes, uint32_t idx, const TravRay& r, float tmax, uint32_t& child_base,
                                 uint32_t& tri_base, uint32_t& imask, uint32_t& meta_lo, uint32_t& meta_hi) {
    const float4* q = reinterpret_cast<const float4*>(nodes + idx);
    const float4 n0 = __ldg(q + 0), n1 = __ldg(q + 1);
    const uint4 qx = __ldg(reinterpret_cast<const uint4*>(q) + 2), qy = __ldg(reinterpret_cast<const uint4*>(q) + 3),
                qz = __ldg(reinterpret_cast<const uint4*>(q) + 4);
    const uint32_t e = __float_as_uint(n0.w);
    imask = e >> 24;
    child_base = __float_as_uint(n1.x);
    tri_base = __float_as_uint(n1.y);
    meta_lo = __float_as_uint(n1.z), meta_hi = __float_as_uint(n1.w);
    // per axis: t = q * (2^e * idir) + (p - o) * idir
    float sx = __uint_as_float((e & 0xFFu) << 23) * r.idir.x, sy = __uint_as_float((e & 0xFF00u) << 15) * r.idir.y,
          sz = __uint_as_float((e & 0xFF0000u) << 7) * r.idir.z;
    float cx = (n0.x - r.o.x) * r.idir.x, cy = (n0.y - r.o.y) * r.idir.y, cz = (n0.z - r.o.z) * r.idir.z;
    const float t0 = max3f(fminf(cx, fmaf(255.0f, sx, cx)), fminf(cy, fmaf(255.0f, sy, cy)),
                           fmaxf(fminf(cz, fmaf(255.0f, sz, cz)), r.tmin));
    cx -= t0, cy -= t0, cz -= t0;
    float mx = max3f(fabsf(sx), fabsf(sy), fabsf(sz));
    const float lim =
        1024.0f * max3f(min3f(fabsf(sx), fabsf(sy), fabsf(sz)), fabsf(t0) * 0x1p-28f, 0x1p-112f);
    float wide = 0.4f * 0x1p-24f;
    const bool far_out = !(fmaxf(mx, fabsf(t0)) < 1e30f);
    if (mx > lim) {
        wide = 0.65f * 0x1p-24f;
        mx = lim;
        if (fabsf(sx) > lim) cx = cx / fabsf(sx) * lim, sx = copysignf(lim, sx);
        if (fabsf(sy) > lim) cy = cy / fabsf(sy) * lim, sy = copysignf(lim, sy);
        if (fabsf(sz) > lim) cz = cz / fabsf(sz) * lim, sz = copysignf(lim, sz);
    }
    mx = fmaxf(mx, 0x1p-102f);
    const uint32_t kb = (244u << 23) - (__float_as_uint(mx) & 0x7F800000u);  // k mx in [2^-10, 2^-9)
    const float k = __uint_as_float(kb), k24 = __uint_as_float(kb + (24u << 23));
    sx *= k24, sy *= k24, sz *= k24;
    cx *= k, cy *= k, cz *= k;
    const float b = fmaf(fabsf(t0) * k, 0x1p-21f, 0x1p-23f);
    const float ex = fmaf(fabsf(sx), wide, b), ey = fmaf(fabsf(sy), wide, b), ez = fmaf(fabsf(sz), wide, b);
    const uint32_t hsx = half2_of(sx, sx), hsy = half2_of(sy, sy), hsz = half2_of(sz, sz);
    const uint32_t nx = half2_of(cx - ex, cx - ex), ny = half2_of(cy - ey, cy - ey), nz = half2_of(cz - ez, cz - ez);
    const uint32_t fx = half2_of(cx + ex, cx + ex), fy = half2_of(cy + ey, cy + ey), fz = half2_of(cz + ez, cz + ez);
    const float te = fmaf(tmax - t0, k * (1.0f + 0x1p-10f), b);
    const uint32_t tend = half2_of(te, te);
    const uint32_t wx[4] = {qx.x, qx.y, qx.z, qx.w}, wy[4] = {qy.x, qy.y, qy.z, qy.w}, wz[4] = {qz.x, qz.y, qz.z, qz.w};
    const uint32_t selx = r.oct & 1u ? 0x4341u : 0x4240u, sely = r.oct & 2u ? 0x4341u : 0x4240u,
                   selz = r.oct & 4u ? 0x4341u : 0x4240u;
    uint32_t m[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t tnx = hfma2_relu(__byte_perm(wx[i], 0u, selx), hsx, nx);
        const uint32_t tny = hfma2(__byte_perm(wy[i], 0u, sely), hsy, ny);
        const uint32_t tnz = hfma2(__byte_perm(wz[i], 0u, selz), hsz, nz);
        const uint32_t tfx = hfma2(__byte_perm(wx[i], 0u, selx ^ 0x0101u), hsx, fx);
        const uint32_t tfy = hfma2(__byte_perm(wy[i], 0u, sely ^ 0x0101u), hsy, fy);
        const uint32_t tfz = hfma2(__byte_perm(wz[i], 0u, selz ^ 0x0101u), hsz, fz);
        m[i] = hle2_mask(__vimax3_s16x2(tnx, tny, tnz), __vmins2(__vimin3_s16x2(tfx, tfy, tfz), tend));
    }
    // one bit per slot: bits 0..3 and 4..7 sit in different bits of the four bytes
    const uint32_t lo = __byte_perm(m[0], m[1], 0x6420u), hi = __byte_perm(m[2], m[3], 0x6420u);
    const uint32_t hits = (((lo & 0x08040201u) | (hi & 0x80402010u)) * 0x01010101u) >> 24;
    return far_out ? 0xFFu : hits;
}

// Byte `byte` of w as the float 2^15 + byte, by one byte permute: the byte
// lands in mantissa bits 8..15 of 2^15 (0x47000000), where one unit is 1.
RT_D float u8f15(uint32_t w, int byte) {
    const uint32_t sel = 4u | (uint32_t(byte) << 4) | (5u << 8) | (7u << 12);
    return __uint_as_float(__byte_perm(w, 0x47000000u, sel));
}

// The same for scenes of few nodes, in single precision: their nodes are large
// beside their flat leaves, so half a quantisation step of margin would make
// most rays test the surface they leave again.  Distances carry 1/128 step and
// 1.6e-6 relative margin: t = (2^15 + q) s + (o - 2^15 s); the folded offset
// carries a rounding error of at most |2^15 s| * 2^-24 = |s| / 512 per rounding,
// plus an |o|-relative part.
RT_D uint32_t intersect_children_f32(const CwNode* nodes, uint32_t idx, const TravRay& r, float tmax,
                                     uint32_t& child_base, uint32_t& tri_base, uint32_t& imask, uint32_t& meta_lo,
                                     uint32_t& meta_hi) {
    const float4* q = reinterpret_cast<const float4*>(nodes + idx);
    const float4 n0 = __ldg(q + 0), n1 = __ldg(q + 1);
    const uint4 qx = __ldg(reinterpret_cast<const uint4*>(q) + 2), qy = __ldg(reinterpret_cast<const uint4*>(q) + 3),
                qz = __ldg(reinterpret_cast<const uint4*>(q) + 4);
    const uint32_t e = __float_as_uint(n0.w);
    imask = e >> 24;
    child_base = __float_as_uint(n1.x);
    tri_base = __float_as_uint(n1.y);
    meta_lo = __float_as_uint(n1.z), meta_hi = __float_as_uint(n1.w);
    const float sx = __uint_as_float((e & 0xFFu) << 23) * r.idir.x, sy = __uint_as_float((e & 0xFF00u) << 15) * r.idir.y,
                sz = __uint_as_float((e & 0xFF0000u) << 7) * r.idir.z;
    const float ox = (n0.x - r.o.x) * r.idir.x, oy = (n0.y - r.o.y) * r.idir.y, oz = (n0.z - r.o.z) * r.idir.z;
    const float cx = fmaf(-32768.0f, sx, ox), cy = fmaf(-32768.0f, sy, oy), cz = fmaf(-32768.0f, sz, oz);
    const float ex = fabsf(sx) * (1.0f / 128.0f), ey = fabsf(sy) * (1.0f / 128.0f), ez = fabsf(sz) * (1.0f / 128.0f);
    const float cxn = cx - ex, cxf = cx + ex, cyn = cy - ey, cyf = cy + ey, czn = cz - ez, czf = cz + ez;
    // the near plane of each slot's pair first
    const uint32_t kx = r.oct & 1u ? 0x2301u : 0x3210u, ky = r.oct & 2u ? 0x2301u : 0x3210u,
                   kz = r.oct & 4u ? 0x2301u : 0x3210u;
    const uint32_t wx[4] = {qx.x, qx.y, qx.z, qx.w}, wy[4] = {qy.x, qy.y, qy.z, qy.w}, wz[4] = {qz.x, qz.y, qz.z, qz.w};
    uint32_t hits = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t x = __byte_perm(wx[i], 0u, kx), y = __byte_perm(wy[i], 0u, ky), z = __byte_perm(wz[i], 0u, kz);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float tx0 = fmaf(u8f15(x, 2 * j), sx, cxn), tx1 = fmaf(u8f15(x, 2 * j + 1), sx, cxf);
            const float ty0 = fmaf(u8f15(y, 2 * j), sy, cyn), ty1 = fmaf(u8f15(y, 2 * j + 1), sy, cyf);
            const float tz0 = fmaf(u8f15(z, 2 * j), sz, czn), tz1 = fmaf(u8f15(z, 2 * j + 1), sz, czf);
            const float tn = max3f(tx0, ty0, fmaxf(tz0, r.tmin));
            const float tf = min3f(tx1, ty1, fminf(tz1, tmax));
            if (tn <= tf * 1.0000016f) hits |= 1u << (2 * i + j);
        }
    }
    return hits;
}

// The nearest internal child of node group g (bits 24..31: children to visit,
// bits 0..7: the parent's internal slots): takes it out of g and returns its
// node index.
RT_D uint32_t take_nearest(uint2& g, const TravRay& r) {
    uint32_t y = g.y & 0xFF000000u, z = y & (r.oct & 4u ? 0xF0000000u : 0x0F000000u);
    y = z ? z : y;
    z = y & (r.oct & 2u ? 0xCC000000u : 0x33000000u);
    y = z ? z : y;
    z = y & (r.oct & 1u ? 0xAA000000u : 0x55000000u);
    y = z ? z : y;
    g.y ^= y;  // one bit is left
    return g.x + __popc(g.y & ((y >> 24) - 1u));
}

// The triangle bits (0..23) of the leaf slots in `leaves`.  A leaf's meta byte
// is (unary mask of its triangles << 5) | index of the first; an empty slot's
// is 0 and adds none.
RT_D uint32_t triangle_bits(uint32_t leaves, uint32_t meta_lo, uint32_t meta_hi) {
    uint32_t bits = 0;
    while (leaves) {
        const uint32_t m = __byte_perm(meta_lo, meta_hi, __ffs(leaves) - 1) & 0xFFu;
        leaves &= leaves - 1u;
        bits |= (m >> 5) << (m & 31u);
    }
    return bits;
}

// Returns the index of the closest hit triangle (or -1) in [tmin, tmax).
// `nodes_visited` / `tris_tested` are only updated when Stats is true.
// `overflows` counts node groups that found the stack full (their subtrees
// are not visited); the renderer rejects BVHs deeper than the stack, so it
// stays zero unless that check is broken, and callers report it as an error.
template <bool AnyHit, bool Stats>
RT_D int traverse(const SceneView& sc, TravRay& r, float& t_hit, float& b1, float& b2, uint32_t& nodes_visited,
                  uint32_t& tris_tested, uint32_t& overflows) {
    int hit_tri = -1;
    float tmax = r.tmax;
    if (sc.num_nodes <= 0) return -1;
    uint2 stack[kStackSize];
    int sp = 0;
    // node group: x = base node index, y = internal hit bits (24..31) | parent imask (0..7)
    uint2 g = make_uint2(0u, 1u << 24);
    // Invariant at the top of the loop: g holds at least one internal-child bit.
    while (true) {
        const uint32_t idx = take_nearest(g, r);
        if (g.y & 0xFF000000u) {
            if (sp < kStackSize)
                stack[sp++] = g;
            else
                overflows++;
        }
        uint32_t cb, tb, im, mlo, mhi;
        const uint32_t hits = intersect_children_f32(sc.nodes, idx, r, tmax, cb, tb, im, mlo, mhi);
        if (Stats) nodes_visited++;
        g = make_uint2(cb, (hits & im) << 24 | im);
        uint32_t tbits = triangle_bits(hits & ~im, mlo, mhi);
        while (tbits) {
            uint32_t b = __ffs(tbits) - 1u;
            tbits &= ~(1u << b);
            uint32_t ti = tb + b;
            const float4* tv = sc.tri_v + size_t(ti) * 3;
            float4 a = __ldg(tv), bb = __ldg(tv + 1), c = __ldg(tv + 2);
            if (Stats) tris_tested++;
            float t, u, v;
            if (intersect_tri(r, a, bb, c, tmax, t, u, v)) {
                hit_tri = int(ti);
                tmax = t;
                t_hit = t;
                b1 = u;
                b2 = v;
                if (AnyHit) return hit_tri;
            }
        }
        while (!(g.y & 0xFF000000u)) {
            if (sp == 0) return hit_tri;
            g = stack[--sp];
        }
    }
    return hit_tri;
}

// ------------------------------------------------------------------ persistent traversal
// Lane-refill ("while-while with dynamic fetch", Aila and Laine, HPG 2009):
// every lane traverses its own ray one wide node at a time; when enough lanes
// of a warp have finished, they take new rays from the queue with a single
// warp-aggregated atomicAdd, so a warp never waits for its slowest ray while
// work remains.  `src.load(i, ray, scene)` fetches queue entry i;
// `src.finish(fin, i, tri, t, b1, b2, tri_v)` is called by the whole warp and
// stores the result of the lanes whose `fin` is set.
//
// Triangles are tested by the whole warp: a lane that meets a leaf appends its
// triangles to the warp's list in shared memory and walks on; when the list
// holds about a warp's worth, every lane tests one triangle of whichever ray
// (its origin and shear are in shared memory too).  A ray's triangles are
// tested in the order in which it met them, and of equal distances the first
// counts, so the answer is that of traverse().
// Bound by issue slots.  Tested by its own lane at once, a triangle had 2.9 of
// 32 lanes for company, and a node step of 26 lanes brought 4 such passes of
// 100 instructions against 250 for the node.  On the 2.59M-triangle scene,
// with the half-precision node test: 2^22 rays leaving its surfaces 2.71 ->
// 1.76 ms, k_extend 67.8 -> 56.5 and k_shadow 19.7 -> 15.6 ms a 1080p frame of
// 64 spp (the half-precision boxes' share: k_extend 64.5 -> 58.6, k_shadow
// 18.8 -> 16.1 ms).  k_extend at other settings: a test at 20 or 32 listed
// triangles +1%, refill at 8 / 12 idle lanes +5% / +1%; a list of 64 costs the
// media scene's k_extend 6% (its rays meet 1.8 triangles a node, 46 a step),
// and testing in the owning lanes there, as traverse_queue_few does, costs the
// large scene 2%; 9 or 7 blocks per SM instead of 8 +4%.
constexpr int kRefillLanesClosest = 14;
constexpr int kRefillLanesAny = 8;
constexpr int kTestAt = 28;      // listed triangles that start a test
constexpr int kDrainLanes = 16;  // lanes waiting only for listed triangles that start one too
constexpr int kListMax = 128;    // room of the list; a lane whose triangles do not fit keeps the rest for the next step
// Threads per block of the persistent traversal kernels.
constexpr int kTravBlock = 128;

// Whether `total` queue items leave nothing for the calling warp of a
// persistent kernel: the warps before it in the grid take one batch of 32
// each.  It ends at once then; at the last bounces' few paths all 4736 warps
// of a launch otherwise queue for the fetch counter's address.  A viewer's
// frame (1080p, 1 spp, 25 bounces) 3.78 -> 3.54 ms.
RT_D bool no_work(int total) { return int(blockIdx.x) * int(blockDim.x) + int(threadIdx.x & ~31u) >= total; }

// The per-thread traversal stack (local memory; a shared-memory stack
// measured no faster).
struct TravStack {
    uint2 e[kStackSize];
    int sp;
    RT_D void push(uint2 v) { e[sp++] = v; }
    RT_D uint2 pop() { return e[--sp]; }
};

// What the lanes of a warp know of each other's rays.
struct TravWarp {
    float ox[32], oy[32], oz[32], sx[32], sy[32], sz[32], tmin[32];
    int axes[32];  // kx | ky << 2 | kz << 4
    // Closest hit: order-preserving bits of the nearest distance so far (at
    // first tmax) in the high word, its place in the list in the low word.
    // Any hit: the place of the first in the list, or ~0.
    unsigned long long best[32];
    float t[32], b1[32], b2[32];  // of the hit (any hit: t is tmax before it)
    const float4* tri[32];        // of the hit, or null
    unsigned long long list[kListMax];  // address of the triangle | lane of its ray << 56
    int count;  // entries of the list, counting those that found no room
};

// Bits that order like the floats, and back.
RT_D uint32_t order_bits(float f) {
    const uint32_t u = __float_as_uint(f);
    return u ^ (uint32_t(int32_t(u) >> 31) | 0x80000000u);
}
RT_D float from_order_bits(uint32_t u) { return __uint_as_float(u ^ (~uint32_t(int32_t(u) >> 31) | 0x80000000u)); }

// The whole warp tests one triangle each, `tv` (null: none) against the ray of
// lane `own`; of several for one ray the lowest `place` counts first.
template <bool AnyHit>
RT_D void test_triangles(TravWarp& w, int own, const float4* tv, int place) {
    bool hit = false;
    float t = 0.f, b1 = 0.f, b2 = 0.f;
    unsigned long long key = 0;
    if (tv != nullptr) {
        const float4 a = __ldg(tv), b = __ldg(tv + 1), c = __ldg(tv + 2);
        TravRay r;
        r.o = v3(w.ox[own], w.oy[own], w.oz[own]);
        r.tmin = w.tmin[own];
        r.Sx = w.sx[own], r.Sy = w.sy[own], r.Sz = w.sz[own];
        const int ax = w.axes[own];
        r.kx = ax & 3, r.ky = (ax >> 2) & 3, r.kz = ax >> 4;
        const float tmax = AnyHit ? w.t[own] : from_order_bits(uint32_t(w.best[own] >> 32));
        hit = intersect_tri(r, a, b, c, tmax, t, b1, b2);
    }
    __syncwarp();
    if (hit) {
        key = (AnyHit ? 0ull : static_cast<unsigned long long>(order_bits(t)) << 32) | unsigned(place);
        atomicMin(&w.best[own], key);
    }
    __syncwarp();
    if (hit && w.best[own] == key) {
        w.t[own] = t;
        w.b1[own] = b1;
        w.b2[own] = b2;
        w.tri[own] = tv;
    }
    __syncwarp();
}

template <bool AnyHit, bool Stats, class Src>
RT_D void traverse_queue(Src& src, int* fetch_counter, int total, uint32_t& nodes_visited, uint32_t& tris_tested,
                         uint32_t& rays, uint32_t& overflows) {
    constexpr int kRefillLanes = AnyHit ? kRefillLanesAny : kRefillLanesClosest;
    if (no_work(total)) return;
    __shared__ TravWarp s_warp[kTravBlock / 32];
    const int lane = threadIdx.x & 31;
    TravWarp& w = s_warp[threadIdx.x >> 5];
    if (lane == 0) w.count = 0;
    __syncwarp();
    TravStack st;
    st.sp = 0;
    TravRay r;
    const CwNode* nodes = nullptr;
    const float4* tri_v = nullptr;
    uint2 g = make_uint2(0u, 0u);
    float tmax = 0.0f;
    uint32_t tb = 0, tbits = 0;  // triangles met and not yet listed
    int item = -1;
    bool active = false, exhausted = false;
    bool more = false;    // the ray has nodes to visit: g holds at least one
    bool listed = false;  // the ray has triangles in the list
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && idle && (__popc(idle) >= kRefillLanes || idle == 0xffffffffu)) {
            int leader = __ffs(idle) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(fetch_counter, __popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (base + __popc(idle) >= total) exhausted = true;
            if (!active) {
                int my = base + __popc(idle & ((1u << lane) - 1u));
                if (my < total) {
                    item = my;
                    const SceneView* sc = nullptr;
                    src.load(item, r, sc);
                    prepare_ray(r);
                    nodes = sc->nodes;
                    tri_v = sc->tri_v;
                    tmax = r.tmax;
                    st.sp = 0;
                    g = make_uint2(0u, 1u << 24);
                    rays++;
                    active = true;
                    more = sc->num_nodes > 0;  // an empty scene: a miss
                    w.ox[lane] = r.o.x, w.oy[lane] = r.o.y, w.oz[lane] = r.o.z;
                    w.sx[lane] = r.Sx, w.sy[lane] = r.Sy, w.sz[lane] = r.Sz;
                    w.tmin[lane] = r.tmin;
                    w.axes[lane] = r.kx | r.ky << 2 | r.kz << 4;
                    w.best[lane] = AnyHit ? ~0ull : static_cast<unsigned long long>(order_bits(tmax)) << 32;
                    w.t[lane] = tmax;
                    w.tri[lane] = nullptr;
                }
            }
        }
        if (more && tbits == 0) {
            const uint32_t idx = take_nearest(g, r);
            if (g.y & 0xFF000000u) {
                if (st.sp < kStackSize)
                    st.push(g);
                else
                    overflows++;
            }
            uint32_t cb, im, mlo, mhi;
            const uint32_t hits = intersect_children(nodes, idx, r, tmax, cb, tb, im, mlo, mhi);
            if (Stats) nodes_visited++;
            g = make_uint2(cb, (hits & im) << 24 | im);
            tbits = triangle_bits(hits & ~im, mlo, mhi);
            if (!(g.y & 0xFF000000u)) {
                if (st.sp == 0)
                    more = false;
                else
                    g = st.pop();
            }
        }
        if (tbits) {
            int pos = atomicAdd(&w.count, __popc(tbits));
            listed = listed || pos < kListMax;
            for (; tbits && pos < kListMax; pos++) {
                const uint32_t b = __ffs(tbits) - 1u;
                tbits &= tbits - 1u;
                if (Stats) tris_tested++;
                w.list[pos] = reinterpret_cast<unsigned long long>(tri_v + size_t(tb + b) * 3) |
                              static_cast<unsigned long long>(lane) << 56;
            }
        }
        __syncwarp();
        const int n = min(w.count, kListMax);
        __syncwarp();  // every lane has the same n before any lists for the next step (a ballot orders no memory)
        const unsigned walking = __ballot_sync(0xffffffffu, more && tbits == 0);
        const unsigned waiting = __ballot_sync(0xffffffffu, !more && listed);
        if (n > 0 && (n >= kTestAt || walking == 0u || __popc(waiting) >= kDrainLanes)) {
            for (int i = lane; i - lane < n; i += 32) {
                const unsigned long long e = i < n ? w.list[i] : 0ull;
                test_triangles<AnyHit>(w, int(e >> 56), reinterpret_cast<const float4*>(e & 0x00FFFFFFFFFFFFFFull), i);
            }
            if (lane == 0) w.count = 0;
            listed = false;
            if (AnyHit) {
                if (active && w.tri[lane] != nullptr) more = false, tbits = 0;
            } else if (active) {
                tmax = from_order_bits(uint32_t(w.best[lane] >> 32));
            }
            __syncwarp();
        }
        const bool fin = active && !more && tbits == 0 && !listed;
        if (__ballot_sync(0xffffffffu, fin)) {
            int tri = -1;
            float t = 0.f, b1 = 0.f, b2 = 0.f;
            if (fin) {
                const float4* tv = w.tri[lane];
                if (tv != nullptr) tri = int(uint32_t(tv - tri_v) / 3u);
                t = w.t[lane], b1 = w.b1[lane], b2 = w.b2[lane];
                active = false;
            }
            src.finish(fin, item, tri, t, b1, b2, tri_v);
        }
        if (exhausted && __ballot_sync(0xffffffffu, active) == 0u) break;
    }
}

// The loop for scenes of few nodes: nearly every lane meets triangles at every
// node there, so each tests its own.  Same contract as traverse_queue.
//
// Triangle postponing (Ylitie et al. 2017): when fewer than kPostpone percent
// of the lanes in a step still test triangles, the rest of a lane's group goes
// on its stack (flagged in bit 31 of x) and the lane returns to node traversal
// with the others.  It changes the order in which a ray meets its triangles,
// so ray queries go without (0).  Groups are postponed only while some lane of
// the warp still visits a node, so every step makes progress, and fill the
// stack only up to kStackSize - BVH depth: node groups (at most one per level
// of the current path) always find room.
constexpr uint32_t kTriGroup = 0x80000000u;
constexpr int kPostponePercentClosest = 12;
constexpr int kPostponePercentAny = 30;

template <bool AnyHit, bool Stats, int kPostpone, class Src>
RT_D void traverse_queue_few(Src& src, int* fetch_counter, int total, uint32_t& nodes_visited, uint32_t& tris_tested,
                             uint32_t& rays, uint32_t& overflows) {
    if (no_work(total)) return;
    constexpr int kRefillLanes = AnyHit ? kRefillLanesAny : kRefillLanesClosest;
    const int lane = threadIdx.x & 31;
    TravStack st;
    st.sp = 0;
    TravRay r;
    const CwNode* nodes = nullptr;
    const float4* tri_v = nullptr;
    int tri_room = 0;
    uint2 g = make_uint2(0u, 0u);
    float tmax = 0.f, t = 0.f, b1 = 0.f, b2 = 0.f;
    int item = -1, hit = -1;
    bool active = false, exhausted = false;
    while (true) {
        bool fin = false;
        const unsigned idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && idle && (__popc(idle) >= kRefillLanes || idle == 0xffffffffu)) {
            int leader = __ffs(idle) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(fetch_counter, __popc(idle));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (base + __popc(idle) >= total) exhausted = true;
            if (!active) {
                int my = base + __popc(idle & ((1u << lane) - 1u));
                if (my < total) {
                    item = my;
                    const SceneView* sc = nullptr;
                    src.load(item, r, sc);
                    prepare_ray(r);
                    nodes = sc->nodes;
                    tri_v = sc->tri_v;
                    tri_room = kStackSize - sc->bvh_depth;
                    tmax = r.tmax;
                    hit = -1;
                    st.sp = 0;
                    g = make_uint2(0u, 1u << 24);
                    rays++;
                    active = sc->num_nodes > 0;
                    fin = !active;  // an empty scene: a miss
                }
            }
        }
        const bool visits = active && !(kPostpone > 0 && (g.x & kTriGroup));
        const int n_step = kPostpone > 0 ? __popc(__ballot_sync(0xffffffffu, active)) : 0;
        const bool may_postpone = kPostpone > 0 && __ballot_sync(0xffffffffu, visits) != 0u;
        if (active) {
            uint32_t tb, tbits;
            if (!visits) {
                tb = g.x & ~kTriGroup;
                tbits = g.y;
                g = make_uint2(0u, 0u);
            } else {
                const uint32_t idx = take_nearest(g, r);
                if (g.y & 0xFF000000u) {
                    if (st.sp < kStackSize)
                        st.push(g);
                    else
                        overflows++;
                }
                uint32_t cb, im, mlo, mhi;
                const uint32_t hits = intersect_children_f32(nodes, idx, r, tmax, cb, tb, im, mlo, mhi);
                if (Stats) nodes_visited++;
                g = make_uint2(cb, (hits & im) << 24 | im);
                tbits = triangle_bits(hits & ~im, mlo, mhi);
            }
            while (tbits) {
                if (may_postpone && __popc(__activemask()) * 100 < kPostpone * n_step && st.sp < tri_room) {
                    st.push(make_uint2(tb | kTriGroup, tbits));
                    break;
                }
                const uint32_t ti = tb + __ffs(tbits) - 1u;
                tbits &= tbits - 1u;
                const float4* tv = tri_v + size_t(ti) * 3;
                const float4 a = __ldg(tv), b = __ldg(tv + 1), c = __ldg(tv + 2);
                if (Stats) tris_tested++;
                float tt, u, v;
                if (intersect_tri(r, a, b, c, tmax, tt, u, v)) {
                    hit = int(ti);
                    tmax = t = tt;
                    b1 = u;
                    b2 = v;
                    if (AnyHit) {
                        fin = true;
                        break;
                    }
                }
            }
            if (!fin && !(kPostpone > 0 && (g.x & kTriGroup)) && !(g.y & 0xFF000000u)) {
                if (st.sp == 0)
                    fin = true;
                else
                    g = st.pop();
            }
            active = !fin;
        }
        src.finish(fin, item, hit, t, b1, b2, tri_v);
        if (exhausted && __ballot_sync(0xffffffffu, active) == 0u) break;
    }
}

}  // namespace rtd
