// xpr_pixel.cuh -- the filtered pixel rule: detector pixels of a brick's voxels from a few
// single-precision operations each, with the contract's own arithmetic (xpr_math.cuh) only
// where those operations cannot tell which side of a pixel border a voxel lies on.
//
// A pixel is a rounding decision on the coordinate u = n_u / n_w (v alike).  Within a brick
// the numerators are affine in the voxel index, so with brick-relative coefficients (the
// matrix rows shifted to the window's first pixel and scaled by the voxel, formed in double
// once per brick and projection) a voxel's window coordinate costs one fused multiply-add
// per voxel of a column, plus a handful of operations per column:
//
//     U' = u - l + 1/2 + 128 + E / 2^16,  the pixel relative to l being floor(U') - 128.
//
// U' of an in-window voxel lies in [128, 256), where a float's ulp is 2^-16: the low 16 bits
// of its representation are its fraction.  E / 2^16 bounds the distance between U' as the
// kernel computes it and the coordinate as the contract rounds it (both errors, below), so a
// fraction >= 2 E / 2^16 proves that both lie between the same two pixel borders.  A smaller
// fraction is decided by the contract's operations.  The decision is therefore always the
// contract's; only its cost changes (a few voxels in ten thousand take the long way).
//
// Plain C++ (no intrinsics outside the bit casts), so the CPU can check the bound.
#pragma once

#include <cstdint>
#include <cstring>

namespace xpr {

#ifdef __CUDACC__
#define XPR_PIX __host__ __device__ inline
#else
#define XPR_PIX inline
#endif

constexpr float kPixBias = 128.0f;       // window coordinates live in [128, 256)
constexpr int kPixWindow = 126;          // largest window (pixels per axis) the filter takes
constexpr float kPixMaxE = 1024.0f;      // largest error bound (2^-16 px) the filter takes
constexpr float kPixU = 5.9604644775390625e-08f;  // 2^-24, the unit roundoff

XPR_PIX uint32_t pix_bits_of(float x)
{
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}
XPR_PIX float pix_float_of(uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}
XPR_PIX float pix_abs(float x) { return x < 0.0f ? -x : x; }
XPR_PIX float pix_max(float a, float b) { return a > b ? a : b; }

// Largest rounding error of a single-precision result of magnitude <= x: half an ulp of
// x's binade (with a margin for x itself being a rounded bound).
XPR_PIX float half_ulp(float x) { return pix_float_of(pix_bits_of(x * 1.0001f) & 0x7f800000u) * kPixU; }

// What the bound needs to know of one (brick, projection) pair.
struct PixBrick {
    float vox[3], org[3];     // voxel size and origin as the contract reads them
    int idx0[3], ext[3];      // first voxel index and extent (voxels) per axis
    float row_off;            // method_2's row offset, subtracted from v
    float wmin, wmax;         // range of n_w over the brick's corners, positive
    int l, r, b, t;           // window [l, r) x [b, t)
};

// Coefficients of one (brick, projection) pair: n_r(i, j, k) ~ c0 + cx i + cz j + cy k.
struct PixRow {
    float c0, cx, cz, cy;
};

// Row c of the matrix shifted by s pixels (c - s * cw), relative to the brick's first
// voxel (n: the row's numerator there, nw: n_w there) and scaled by the voxel size.
XPR_PIX PixRow pix_row(const float *c, const float *cw, double n, double nw, double s, const float *vox)
{
    PixRow o;
    o.c0 = (float)(n - s * nw);
    o.cx = (float)(((double)c[0] - s * (double)cw[0]) * (double)vox[0]);
    o.cy = (float)(((double)c[1] - s * (double)cw[1]) * (double)vox[1]);
    o.cz = (float)(((double)c[2] - s * (double)cw[2]) * (double)vox[2]);
    return o;
}

// Per-axis magnitudes of the brick's positions: P = max |p|, D = error of the contract's
// position against idx * vox + org.
struct PixAxes {
    float P[3], D[3];
};
XPR_PIX PixAxes pix_axes(const PixBrick &k, bool strict)
{
    PixAxes a;
    for (int i = 0; i < 3; ++i) {
        const float hi = (float)(k.idx0[i] + k.ext[i] - 1);
        const float p0 = pix_abs((float)k.idx0[i] * k.vox[i] + k.org[i]);
        const float p1 = pix_abs(hi * k.vox[i] + k.org[i]);
        a.P[i] = pix_max(p0, p1) * 1.0001f + 4.0f * kPixU * pix_abs(k.org[i]);
        // STRICT rounds idx * vox and the sum, FAST fuses them
        a.D[i] = half_ulp(a.P[i]) + (strict ? half_ulp(hi * pix_abs(k.vox[i])) : 0.0f);
    }
    return a;
}

// Error of the contract's numerator of row c, |n| <= nmax (STRICT: the whole numerator
// ((c.x px + c.y py) + c.z pz) + c.w; FAST: its column part fma(c.x, px, c.w) + c.z pz).
XPR_PIX float pix_num_err(const float *c, const PixAxes &a, float nmax, bool strict)
{
    const float Tx = pix_abs(c[0]) * a.P[0], Ty = pix_abs(c[1]) * a.P[1], Tz = pix_abs(c[2]) * a.P[2];
    const float pos = pix_abs(c[0]) * a.D[0] + pix_abs(c[1]) * a.D[1] + pix_abs(c[2]) * a.D[2];
    if (strict)
        return pos + half_ulp(Tx) + half_ulp(Ty) + half_ulp(Tz) + (Ty > 0.0f ? half_ulp(Tx + Ty) : 0.0f) +
               half_ulp(Tx + Ty + Tz) + half_ulp(nmax);
    const float w = pix_abs(c[3]);
    return pos + half_ulp(Tx + w) + half_ulp(Tz) + half_ulp(Tx + Tz + w);
}

// Distance between the contract's coordinate and the real one, for coordinates of magnitude
// <= q inside the window (q counts the row offset in).
XPR_PIX float pix_contract_err(const float *c, const float *cw, const PixBrick &k, const PixAxes &a, float q,
                               bool strict)
{
    const float rw = 1.0001f / k.wmin;
    if (strict) {
        const float ew = pix_num_err(cw, a, k.wmax, true);
        // the quotient's rounding; subtracting the row offset is exact inside the window
        return (pix_num_err(c, a, q * k.wmax, true) + q * ew) * rw + half_ulp(q);
    }
    const float ew = pix_num_err(cw, a, 0.0f, false) + (cw[1] != 0.0f ? half_ulp(k.wmax) : 0.0f);
    const float rel = kPixU + ew * rw;  // of the reciprocal
    const float C = pix_abs(c[0]) * a.P[0] + pix_abs(c[2]) * a.P[2] + pix_abs(c[3]);
    const float Ty = pix_abs(c[1]) * a.P[1];
    return pix_num_err(c, a, 0.0f, false) * rw + (rel * (C + Ty) + kPixU * Ty) * rw +
           half_ulp(C * rw + k.row_off + 1.0f) + half_ulp(q + 1.0f);
}

// Distance between the kernel's window coordinate and the real one, for coordinates within
// `span` pixels of the window's first: two fused multiply-adds per numerator on rounded
// coefficients, a reciprocal good to 2^-23 (a hardware approximation good to 2^-22 and one
// Newton step), the products with it, and three roundings at 128 .. 256.  When n_w has a
// y-coefficient the coordinate is walked as a quadratic in the column's layer index.
XPR_PIX float pix_kernel_err(const PixRow &r, const PixRow &w, const PixBrick &k, float span)
{
    const float ex = (float)k.ext[0], ey = (float)k.ext[1], ez = (float)k.ext[2];
    const float rw = 1.0001f / k.wmin;
    const float S = pix_abs(r.c0) + ex * pix_abs(r.cx) + ez * pix_abs(r.cz);
    const float Sw = pix_abs(w.c0) + ex * pix_abs(w.cx) + ez * pix_abs(w.cz);
    const float rel = kPixU * (2.0f + 4.0f * Sw * rw);
    const float rise = ey * pix_abs(r.cy) * rw;
    float e = 4.0f * kPixU * S * rw + rel * span + (rel + 2.0f * kPixU) * rise + 3.0f * 128.0f * kPixU;
    if (w.cy != 0.0f) {
        // n_w changes by `bend` (relative) along the column: the quadratic's coefficients, its
        // third-order remainder, and the roundings of its Horner steps
        const float bend = ey * pix_abs(w.cy) * rw;
        if (!(bend < 0.05f)) return 1.0f;
        const float lin = rise + span * bend;
        e += 4.0f * kPixU * lin + 3.0f * (rel + 4.0f * kPixU) * (span + lin) * bend + 1.2f * lin * bend * bend +
             128.0f * kPixU;
    } else {
        e += 4.0f * kPixU * rise;
    }
    return e;
}

// The bound E in units of 2^-16 px (an integer), or 0 when the pair is not to be filtered.
// cu, cv, cw: the matrix rows; u, v, w: their brick-relative coefficients.
XPR_PIX int pix_bound(const float *cu, const float *cv, const float *cw, const PixRow &u, const PixRow &v,
                      const PixRow &w, const PixBrick &k, bool strict)
{
    if (!(k.wmin > 0x1p-60f && k.wmax < 0x1p60f)) return 0;
    if (k.r - k.l > kPixWindow || k.t - k.b > kPixWindow) return 0;
    const PixAxes a = pix_axes(k, strict);
    const float qu = (float)k.r + 1.0f, qv = (float)k.t + 1.0f + k.row_off;
    const float eu = pix_contract_err(cu, cw, k, a, qu, strict) + pix_kernel_err(u, w, k, (float)(k.r - k.l) + 2.0f);
    const float ev = pix_contract_err(cv, cw, k, a, qv, strict) + pix_kernel_err(v, w, k, (float)(k.t - k.b) + 2.0f);
    const float e = pix_max(eu, ev) * 1.02f * 65536.0f;
    // NaN and infinities compare false
    if (!(eu < 1.0f && ev < 1.0f && e < kPixMaxE)) return 0;
    return (int)e + 2;
}

}  // namespace xpr
