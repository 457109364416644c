// walk_nodes.h — the 64-byte nodes that large trees are walked through: how
// the device derives them from the full-precision nodes (bvh.h) and how a ray
// tests them. Shared by the kernels and by host checks of both.
//
// A walk node holds the child boxes rounded outward to 8-bit offsets in the
// node's frame, like a quantized node, but tested without decoding the planes.
// Word 0 = (origin.xyz, Sx), word 1 = links, words 2-3 = (lo.x, hi.x, lo.y,
// hi.y), (lo.z, hi.z, Sy, Sz), one byte per child, S = 2^15 x the step s of the
// axis (a power of two).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "aq_math.h"

namespace aq {

// a - b = diff + the returned rest, exactly (Knuth's two-sum; no overflow here).
AQ_HD double diff_exact(double a, double b, double& diff) {
    diff = a - b;
    const double t = diff - a;
    return (a - (diff - t)) - (b + t);
}

// One axis of a walk node from the child planes lo[c], hi[c] and the links: the
// decoded planes origin + q s bound the children's exactly. A difference of two
// floats need not fit a double, but its rounding can only hide that it lies just
// below or above a multiple of the step, which the rest shows. (Products with and
// quotients by a power of two are exact.)
AQ_HD void walk_axis(const float* plo, const float* phi, const int32_t* link, float& origin, float& step,
                     uint32_t& lo_bytes, uint32_t& hi_bytes) {
    float lo = INFINITY, hi = -INFINITY;
    for (int c = 0; c < 4; ++c)
        if (link[c] != ~0) {
            lo = fminf(lo, plo[c]);
            hi = fmaxf(hi, phi[c]);
        }
    if (!(lo <= hi)) lo = hi = 0.0f;  // no children (not produced by the builder)
    int e = -100;
    double d, rest;
    if (hi > lo) {  // smallest step whose 255 multiples reach hi
        rest = diff_exact(hi, lo, d);
        const int k = ilogb(d / 255.0);
        e = k > -100 ? k : -100;
        const double reach = ldexp(255.0, e);
        if (reach < d || (reach == d && rest > 0.0)) ++e;
    }
    const double s = ldexp(1.0, e);
    origin = lo;
    step = (float)ldexp(1.0, e + 15);
    lo_bytes = hi_bytes = 0;
    for (int c = 0; c < 4; ++c) {
        uint32_t ql = 255, qh = 0;  // empty slot: an inverted box
        if (link[c] != ~0) {
            rest = diff_exact(plo[c], lo, d);
            ql = (uint32_t)floor(d / s);
            if (rest < 0.0 && (double)ql * s == d) --ql;
            rest = diff_exact(phi[c], lo, d);
            qh = (uint32_t)ceil(d / s);
            if (rest > 0.0 && (double)qh * s == d) ++qh;
        }
        lo_bytes |= ql << (8 * c);
        hi_bytes |= qh << (8 * c);
    }
}

// The frame and the planes of a walk node.
struct WalkBoxes {
    float ox, oy, oz, sx, sy, sz;  // origin and S
    uint32_t lx, hx, ly, hy, lz, hz;
};

// 1 + q 2^-15 of child k's byte q.
AQ_HD float walk_byte(uint32_t word, int k) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(__byte_perm(word, 0x3F800000u, 0x7604u | ((uint32_t)k << 4)));
#else
    const uint32_t bits = 0x3F800000u | (((word >> (8 * k)) & 0xffu) << 8);
    float f;
    memcpy(&f, &bits, 4);
    return f;
#endif
}

// Entry distances of the four child boxes (INFINITY = missed). One byte
// permute makes the float 1 + q 2^-15, and with b = (origin - o) / d and
// A = S / d one multiply-add gives the distance to the plane:
//   (1 + q 2^-15) A + (b - A) = b + q s / d.
// The rounding errors of a plane's distance stay below
// 5 x 2^-24 (|b| + |A|); near planes are moved back and far planes forward
// by 8 x 2^-24 (|b| + |A|) (1/64 of a step at least, more from far away), which
// also covers the rounding of slab_entry on the exact planes. So every box that
// slab_entry accepts is accepted here, at no later distance, and a walk whose hits
// are confirmed (walk_confirmed) finds what the full-precision walk finds. An
// empty slot is accepted too where the node is flat or the ray's origin lies
// some 10^5 node extents away: its leaf holds no triangle, but the walk may
// push all four slots of a node (walk_stack_fits).
// The ray's signs choose the near and far words, six selections per node
// instead of two min/max per plane pair and child: the arithmetic costs what
// the full-precision node's does, from 64 bytes and two loads instead of 112
// bytes and four. The walk of large trees is bound by its node fetches
// (L1 data pipe 71% busy on the 1.15M-triangle interior): 2.07M rays against
// it 540 -> 520 us, its 1080p render at 8 spp 49.1 -> 43.9 ms.
AQ_HD void walk_entries(const WalkBoxes& w, const RayPre& rp, float tfar, float* t) {
    constexpr float kPad = 4.76837158203125e-7f;  // 2^-21
    const float bx = mul_rn(sub_rn(w.ox, rp.o.x), rp.invd.x), by = mul_rn(sub_rn(w.oy, rp.o.y), rp.invd.y),
                bz = mul_rn(sub_rn(w.oz, rp.o.z), rp.invd.z);
    const float ax = mul_rn(w.sx, rp.invd.x), ay = mul_rn(w.sy, rp.invd.y), az = mul_rn(w.sz, rp.invd.z);
    const float mx = add_rn(fabsf(bx), fabsf(ax)), my = add_rn(fabsf(by), fabsf(ay)), mz = add_rn(fabsf(bz), fabsf(az));
    const float dx = sub_rn(bx, ax), dy = sub_rn(by, ay), dz = sub_rn(bz, az);
    const float bnx = fmaf(-kPad, mx, dx), bfx = fmaf(kPad, mx, dx), bny = fmaf(-kPad, my, dy),
                bfy = fmaf(kPad, my, dy), bnz = fmaf(-kPad, mz, dz), bfz = fmaf(kPad, mz, dz);
    const bool ix = rp.invd.x < 0.0f, iy = rp.invd.y < 0.0f, iz = rp.invd.z < 0.0f;
    const uint32_t qnx = ix ? w.hx : w.lx, qfx = ix ? w.lx : w.hx, qny = iy ? w.hy : w.ly, qfy = iy ? w.ly : w.hy,
                   qnz = iz ? w.hz : w.lz, qfz = iz ? w.lz : w.hz;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int k = 0; k < 4; ++k) {
        const float n = fmaxf(fmaxf(fmaf(walk_byte(qnx, k), ax, bnx), fmaf(walk_byte(qny, k), ay, bny)),
                              fmaxf(fmaf(walk_byte(qnz, k), az, bnz), rp.tmin));
        const float f = fminf(fminf(fmaf(walk_byte(qfx, k), ax, bfx), fmaf(walk_byte(qfy, k), ay, bfy)),
                              fminf(fmaf(walk_byte(qfz, k), az, bfz), tfar));
        t[k] = n <= mul_rn(f, kSlabFarScale) ? n : INFINITY;
    }
}

}  // namespace aq
