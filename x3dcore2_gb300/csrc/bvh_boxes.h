// Box arithmetic shared by the host builders (bvh.cpp, bvh_wide.cpp) and the device refit
// (refit.cu), so a refit of an unchanged scene writes the bytes the host build wrote.
//
// Every stored box is the exact union of the triangles below it, pushed outwards by
// |v| * 1e-6 + eps with eps = 1e-6 * (largest extent of the scene's box). The eight-wide layout
// then quantizes the pushed-out boxes of a node's children on a per-node grid.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <math.h>

#if defined(__CUDACC__)
#define E8G_BOX_HD __host__ __device__ __forceinline__
#else
#define E8G_BOX_HD inline
#endif

namespace e8g {

E8G_BOX_HD uint32_t box_f2u(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
#endif
}

E8G_BOX_HD float inflate_lo(float v, float eps) { return v - (fabsf(v) * 1.0e-6f + eps); }
E8G_BOX_HD float inflate_hi(float v, float eps) { return v + (fabsf(v) * 1.0e-6f + eps); }

// eps of a scene whose exact box is [lo, hi].
E8G_BOX_HD float scene_eps(float const lo[3], float const hi[3]) {
    float diag = 0;
    for (int a = 0; a < 3; a++) {
        float d = hi[a] - lo[a];
        diag = diag < d ? d : diag;
    }
    return diag * 1.0e-6f;
}

// Smallest grid step of the quantized layout: 2^-18 of the largest coordinate the scene and the
// rays reach (far above the rounding of the slab arithmetic, so one step of outward rounding
// keeps every box conservative), and at least 2^-100.
E8G_BOX_HD double wide_step_min(float max_abs) {
    double s = static_cast<double>(max_abs) * ldexp(1.0, -18);
    double floor_step = ldexp(1.0, -100);
    return s > floor_step ? s : floor_step;
}

// Smallest e in [-126, 127] with 2^e >= want (want > 0), computed without log2 so the host and
// the device agree exactly.
E8G_BOX_HD int wide_exponent(double want) {
    int x;
    double m = frexp(want, &x); // want = m * 2^x, m in [0.5, 1)
    int e = m == 0.5 ? x - 1 : x;
    return e < -126 ? -126 : (e > 127 ? 127 : e);
}

// floor and ceil of (v - org) * inv, with inv a power of two, from the exact difference: s + err
// = v - org exactly (Knuth's TwoSum in single precision), s * inv is exact, and a float quotient
// is at least one of its ulps away from the next integer, so only an integer quotient can move,
// by the sign of err. The same result as the double-precision expression whenever v - org is
// exact in double (exponents within 29 of each other), without double arithmetic (slow on this
// GPU).
E8G_BOX_HD void wide_grid_floor_ceil(float v, float org, float inv, float &fl, float &cl) {
    float s = v - org;
    float bb = s - v;
    float err = (v - (s - bb)) + (-org - bb);
    float q = s * inv;
    fl = floorf(q);
    cl = ceilf(q);
    if (fl == q && err < 0.0f)
        fl -= 1.0f;
    if (cl == q && err > 0.0f)
        cl += 1.0f;
}

E8G_BOX_HD float box_u2f(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}

// One axis of a node's quantization grid from the children's union: the grid starts one step below it and
// 253 steps cover it, so no child box is clamped to the grid's ends and every quantized plane lies at
// least one step outside the (already pushed-out) child box: the slack absorbs the rounding of the
// traversal's plane arithmetic. inv_step: 2^-e (dividing by the step 2^e is this exact product); returns
// the exponent byte. step_min: wide_step_min's, e_min its exponent.
E8G_BOX_HD uint32_t wide_grid_axis_double(float u_lo, float u_hi, double step_min, float &org, float &inv_step) {
    double ext = static_cast<double>(u_hi) - static_cast<double>(u_lo);
    double want = ext / 251.0;
    want = want > step_min ? want : step_min;
    int e = wide_exponent(want);
    inv_step = ldexpf(1.0f, -e);
    double l = static_cast<double>(u_lo) - ldexp(1.0, e);
    float f = static_cast<float>(l);
    if (static_cast<double>(f) > l)
        f = nextafterf(f, -INFINITY);
    org = f;
    return static_cast<uint32_t>(e + 127);
}

// The same result in single precision (the double form's divisions and differences run at about two a
// cycle on each SM: 100 of the 247 us that the 1.3M-triangle scene's eight-wide emission took). The
// exponent follows from the single-precision quotient unless its mantissa lies within 16 ulps, several times its rounding, of a
// power of two; the origin is the difference rounded down, from its exact error (Knuth's TwoSum), equal
// to the double form's while the difference is exact in double (exponents close enough). Anything else
// takes the double form.
E8G_BOX_HD uint32_t wide_grid_axis(float u_lo, float u_hi, double step_min, int e_min, float &org, float &inv_step) {
    const uint32_t w = box_f2u((u_hi - u_lo) * (1.0f / 251.0f)), m = w & 0x7FFFFFu, ew = w >> 23;
    int e = static_cast<int>(ew) - 126;
    e = e < e_min ? e_min : e;
    const uint32_t lb = box_f2u(u_lo) & 0x7FFFFFFFu;
    const int el = static_cast<int>(lb >> 23) - 127;
    if (ew < 30 || ew > 220 || m < 16 || m > 0x7FFFFFu - 16 || e < -90 || e > 90 ||
        (lb != 0 && (el < e - 29 || el > e + 40)))
        return wide_grid_axis_double(u_lo, u_hi, step_min, org, inv_step);
    const float step = box_u2f(static_cast<uint32_t>(e + 127) << 23);
    inv_step = box_u2f(static_cast<uint32_t>(127 - e) << 23);
    const float f = u_lo - step;
    const float bb = f - u_lo;
    const float err = (u_lo - (f - bb)) + (-step - bb);
    const uint32_t fb = box_f2u(f);
    org = err < 0.0f ? box_u2f(fb & 0x80000000u ? fb + 1 : fb - 1) : f; // the float below
    return static_cast<uint32_t>(e + 127);
}

// The quantized planes of one child box on one axis.
E8G_BOX_HD void wide_grid_planes(float lo, float hi, float org, float inv_step, uint32_t &qlo, uint32_t &qhi) {
    float fl, cl, unused;
    wide_grid_floor_ceil(lo, org, inv_step, fl, unused);
    wide_grid_floor_ceil(hi, org, inv_step, unused, cl);
    float ql = fl - 1.0f, qh = cl + 1.0f;
    ql = ql < 0.0f ? 0.0f : (ql > 255.0f ? 255.0f : ql);
    qh = qh < 0.0f ? 0.0f : (qh > 255.0f ? 255.0f : qh);
    qlo = static_cast<uint32_t>(ql);
    qhi = static_cast<uint32_t>(qh);
}

// Fills a node's grid and quantized child boxes: words[0..2] (grid origin), the exponent bytes of
// words[3] (the interior mask byte is left alone) and words[8..19]. lo/hi hold the pushed-out
// boxes of the eight slots; only slots in `present` are used.
E8G_BOX_HD void wide_quantize(float const lo[8][3], float const hi[8][3], uint32_t present, double step_min,
                          uint32_t words[24]) {
    float u_lo[3] = {INFINITY, INFINITY, INFINITY}, u_hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int s = 0; s < 8; s++) {
        if (!(present >> s & 1))
            continue;
        for (int a = 0; a < 3; a++) {
            u_lo[a] = lo[s][a] < u_lo[a] ? lo[s][a] : u_lo[a];
            u_hi[a] = u_hi[a] < hi[s][a] ? hi[s][a] : u_hi[a];
        }
    }
    float inv_step[3], org[3];
    uint32_t ebytes = 0;
    const int e_min = wide_exponent(step_min);
    for (int a = 0; a < 3; a++) {
        ebytes |= wide_grid_axis(u_lo[a], u_hi[a], step_min, e_min, org[a], inv_step[a]) << (8 * a);
        words[a] = box_f2u(org[a]);
    }
    words[3] = (words[3] & 0xFF000000u) | ebytes;
    uint32_t qb[12] = {0};
    for (int s = 0; s < 8; s++) {
        if (!(present >> s & 1))
            continue;
        for (int a = 0; a < 3; a++) {
            uint32_t ql, qh;
            wide_grid_planes(lo[s][a], hi[s][a], org[a], inv_step[a], ql, qh);
            // byte s of plane a (lo) and plane 3 + a (hi); 8 bytes per plane, little endian
            qb[2 * a + (s >> 2)] |= ql << (8 * (s & 3));
            qb[2 * (3 + a) + (s >> 2)] |= qh << (8 * (s & 3));
        }
    }
    for (int k = 0; k < 12; k++)
        words[8 + k] = qb[k];
}

} // namespace e8g
