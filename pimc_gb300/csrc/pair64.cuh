// pair64.cuh -- the FP64 pair evaluation of the plain form's kernels.
#pragma once

#include "pgb_device.cuh"

namespace pgb {

// ---------------------------------------------------------------------------
// One FP64 pair with about twenty FP64 instructions.  The FP64 pipe of this
// GPU takes 16 clocks of an SM for a warp instruction (64 of one
// sub-partition), so a pair kernel's time is its FP64 instruction count; the
// direct form (gradV64: three min_image, sqrt, r / dr, T / r) has about ninety.
//   * The image index floor(x / L + 1/2) is 0 or +-1 for beads in the box and
//     comes from FP32 box fractions; the separation x - index L is then the
//     same FP64 value as min_image's.
//   * 1/r is the hardware's 20-bit reciprocal root refined by one step of
//     Householder's third-order iteration, y (1 + e/2 + 3 e^2/8) with
//     e = 1 - r^2 y^2; the series leaves 5 e^3 / 16 < 2^-54.
//   * The table index int(r / dr) is read off the bits of r (1/dr) + 1.5 2^32,
//     whose last place is 2^-20.
// A pair whose FP32 fraction lies within kImageEdge of an image boundary, or
// whose quotient lies within 2 2^-20 of an integer, takes the direct form
// (about 1e-5 of the pairs), and so does any pair that is not finite or not
// near the box: the separation and the index are the direct form's always.
// ---------------------------------------------------------------------------
struct Pair64 {
    double dx, dy, dz, y;        // separation, 1/r
    double r2;
    int k;                       // table index, 0: outside the table (value 0)
};

// A box fraction (FP32 position times FP32 1/L) is within 3 2^-24 for |u| <= 1,
// the difference of two within 4.2e-7: below the edge.
constexpr float kImageEdge = 1.0e-6f;

// 1 / sqrt(d), 2^-960 <= d < 2^960, within 2^-52 of it: half an ulp of e, the
// last rounding, and the series' remainder
__device__ __forceinline__ double inv_root64(double d) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = __fma_rn(-(d * y), y, 1.0);
    return __fma_rn(y * e, __fma_rn(0.375, e, 0.5), y);
}

// x / L for the image screen; NaN outside the range where its error bound holds
__device__ __forceinline__ float box_fraction(float x, float Linv) {
    const float u = x * Linv;
    return fabsf(u) <= 1.0f ? u : __int_as_float(0x7fffffff);
}

// the direct form, for the pairs the fast form leaves out
static __device__ __noinline__ Pair64 pair64_direct(double x, double y, double z, double Lx, double Ly, double Lz,
                                             double Lix, double Liy, double Liz, double dr, int len) {
    Pair64 p;
    p.dx = min_image(x, Lx, Lix); p.dy = min_image(y, Ly, Liy); p.dz = min_image(z, Lz, Liz);
    p.r2 = dot3(make_double3(p.dx, p.dy, p.dz), make_double3(p.dx, p.dy, p.dz));
    const double r = sqrt(p.r2), q = r / dr;
    p.k = (q < (double)len) ? (int)q : 0;          // also catches NaN
    p.y = 1.0 / r;
    return p;
}

// x - L floor(x / L + 1/2) given x / L in FP32 as du; ok is cleared near an
// image boundary
__device__ __forceinline__ double image64(double x, float du, double L, bool& ok) {
    const float t = fabsf(fabsf(du) - 0.5f);
    ok = ok && (t > kImageEdge) && (t < 0.999f);
    const bool w = fabsf(du) > 0.5f;
    const int hi = w ? (__double2hiint(L) ^ (__float_as_int(du) & 0x80000000)) : 0;
    return x - __hiloint2double(hi, w ? __double2loint(L) : 0);
}

// separation (x, y, z) = r_a - r_b before the images, with the FP32
// differences of the box fractions
__device__ __forceinline__ Pair64 pair64(const PathView& v, double invdr, double x, double y, double z, float ux,
                                         float uy, float uz) {
    Pair64 p;
    bool ok = true;
    p.dx = image64(x, ux, v.side[0], ok);
    p.dy = image64(y, uy, v.side[1], ok);
    p.dz = image64(z, uz, v.side[2], ok);
    p.r2 = dot3(make_double3(p.dx, p.dy, p.dz), make_double3(p.dx, p.dy, p.dz));
    p.y = inv_root64(p.r2);
    const double t = __fma_rn(p.r2 * p.y, invdr, 6442450944.0);      // 1.5 2^32
    const long long b = __double_as_longlong(t);
    const unsigned frac = (unsigned)b & 0xFFFFFu;
    // exponent of [2^32, 2^33): finite and below 2^31 table steps
    ok = ok && ((unsigned)(b >> 52) == 0x41Fu) && (frac - 2u < 0xFFFFDu);
    p.k = (int)((unsigned)(b >> 20) - 0x80000000u);
    p.k = (unsigned)p.k < (unsigned)v.tableLength ? p.k : 0;
    if (!ok)
        p = pair64_direct(x, y, z, v.side[0], v.side[1], v.side[2], v.sideInv[0], v.sideInv[1], v.sideInv[2], v.dr,
                          v.tableLength);
    return p;
}

// table value at a pair's index: extremal values 0 (potential.h:249-260)
__device__ __forceinline__ double table64(const double* T, int k) { return k > 0 ? __ldg(T + k) : 0.0; }

}  // namespace pgb
