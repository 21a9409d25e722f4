// gp.cu -- the Gaussian-process external potential on the device.
//
// GaussianProcessPotential::GP (src/potential.cpp:330-392) with the Matern
// kernel of MaternKernel::K (src/gpkernel.cpp:97-108, include/gpkernel.h:
// 61-72): for an inference point r, normalised as (r - offset) / scale,
//     V(r) = mean_d + std_d (mu + sigma2 sum_k K(r, x_k) w_k),
//     K    = k_nu(|putInBC(x_k - r) / ell|),  w_k = (K^-1 Y)_k.
// The CPU kernel applies the container's boundary conditions to the
// separation; the reference's GPU kernel (potential_gpu.cu:4-54) leaves them
// out and divides by ell instead of multiplying by 1/ell.  This file follows
// the CPU form, so both precisions agree with the reference's CPU path.
//
// FP64 kernel (compiled with -fmad=false): one thread per inference point
// and chunk of training points, streamed through shared memory in index
// order; the chunk sums are added in chunk order.  Chunks exist only to fill
// the GPU when a call has few points: from about 155 k points on there is one
// chunk and every sum has the CPU form's order; the exponential
// and the root may differ by an ulp from the host's.  With several chunks the sum is
// regrouped, a relative change of order 1e-16 of sum_k |K w_k|.
// Mixed kernel: the separations and kernel values in FP32 and the sum in a
// double-float pair (TwoSum), about 1e-7 of sum_k |K w_k| off the FP64 value.
//
// GPHeBenzenePotential::V (src/potential.cpp:5610-5681): points are folded
// into the 30-degree wedge of the ring's symmetry on the device, passed
// through the GP, then switched to the long-range form beyond the core.
#include "pair64.cuh"

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace pgb {

struct GpDev {
    double off[3], scale[3], invell[3], pside[3], sideInv[3];
    double standard_mean, standard_std, mu, sigma2;
    double reach[3];  // largest |training coordinate| / side, 0 where not periodic
    double perInv[3]; // 1 / side, 0 where not periodic
    int nu2;          // 2 nu: 1, 3 or 5
    int n;            // training points
};

// No separation from a point can reach half a box, so the periodic images
// change nothing: inputs are normalised to order one and the box is not.
__device__ __forceinline__ bool gp_inside(const GpDev& g, double r0, double r1, double r2) {
    return g.reach[0] + fabs(r0) * g.perInv[0] < 0.4999 && g.reach[1] + fabs(r1) * g.perInv[1] < 0.4999 &&
           g.reach[2] + fabs(r2) * g.perInv[2] < 0.4999;
}

constexpr int kGpBlock = 256;           // inference points a CTA
constexpr int kGpTile = 256;            // training points per shared-memory tile

// x / 3, correctly rounded (Markstein's division by a constant)
__device__ __forceinline__ double third(double x) {
    const double k = 1.0 / 3.0, q = x * k;
    return __fma_rn(__fma_rn(-3.0, q, x), k, q);
}

// sqrt(d) for 2^-960 <= d < 2^960: r = d / sqrt(d) and one step of Newton's
// iteration for the root, r + (d - r^2) / 2 r, with the reciprocal root in the
// place of 1 / r and the residual exact (P. W. Markstein, IBM J. Res. Dev. 34,
// 1990).  Half an ulp and 2^-100: correctly rounded but for near ties; 9 FP64
// instructions
__device__ __forceinline__ double root64(double d) {
    const double y = inv_root64(d), r = d * y;
    return __fma_rn(__fma_rn(-r, r, d), 0.5 * y, r);
}

// exp(-x), x >= 0, by Tang's table method (ACM TOMS 15, 1989): with
// n = round(-64 x / ln 2), exp(-x) = 2^(n/64) exp(-x - n ln 2 / 64), the first
// factor from the 64 tabulated 2^(j/64), the second, whose argument is below
// ln 2 / 128, from six Taylor terms (relative remainder 3e-20).  Eleven FP64
// instructions where exp() takes about forty.  Half an ulp of the table, half
// an ulp of the last rounding and a hundredth for the argument and the series:
// within 1.01 ulp, and from 700 on (and for NaN) exp() itself.
constexpr int kExpTable = 64;
__device__ __forceinline__ double exp_neg64(double x, const double* T) {
    if ((unsigned)__double2hiint(x) >= 0x4085E000u) return exp(-x);     // 700 and up, NaN
    const double magic = 6755399441055744.0;                         // 1.5 2^52
    const double t = __fma_rn(x, -92.332482616893657, magic);         // 64 / ln 2
    const int n = __double2loint(t);
    const double f = t - magic;
    // ln 2 / 64 in two parts, those of fdlibm's exp (Sun Microsystems, 1993) a
    // 64th; f times the first is exact
    double r = __fma_rn(f, -6.93147180369123816490e-01 / 64.0, -x);
    r = __fma_rn(f, -1.90821492927058770002e-10 / 64.0, r);
    const double q = __fma_rn(r, __fma_rn(r, __fma_rn(r, __fma_rn(r, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5);
    const double p = __fma_rn(r * r, q, r);
    const double s = T[n & (kExpTable - 1)];
    const double y = __fma_rn(s, p, s);
    return __hiloint2double(__double2hiint(y) + ((n >> 6) << 20), __double2loint(y));
}

// the three functions and the reciprocal root by themselves, for their test
__global__ void k_gp_math(const double* __restrict__ x, int n, int what, const double* __restrict__ table,
                          double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = what == 0 ? root64(x[i]) : what == 1 ? third(x[i]) : what == 2 ? exp_neg64(x[i], table) : inv_root64(x[i]);
}

template <int NU2>
__device__ __forceinline__ double matern64(double r, const double* T) {
    const double kSqrt3 = 1.7320508075688772935, kSqrt5 = 2.2360679774997896964;
    if (NU2 == 1) return exp_neg64(r, T);
    if (NU2 == 3) { const double x = kSqrt3 * r; return (1.0 + x) * exp_neg64(x, T); }
    const double x = kSqrt5 * r;
    return (1.0 + x + third(x * x)) * exp_neg64(x, T);
}

template <int NU2>
__device__ __forceinline__ float matern32(float r) {
    const float kSqrt3 = 1.7320508f, kSqrt5 = 2.2360680f;
    if (NU2 == 1) return expf(-r);
    if (NU2 == 3) { const float x = kSqrt3 * r; return (1.0f + x) * expf(-x); }
    const float x = kSqrt5 * r;
    return (1.0f + x + x * x * (1.0f / 3.0f)) * expf(-x);
}

// The normalised points, once a call: every chunk's CTA dividing for itself
// would take the FP64 pipe longer than its share of the kernel values.  w is 1
// where no image is needed (gp_inside).
template <typename T4>
__global__ void k_gp_points(GpDev g, const double* __restrict__ pos, int count, T4* __restrict__ r) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const double x = (pos[3 * (size_t)i] - g.off[0]) / g.scale[0];
    const double y = (pos[3 * (size_t)i + 1] - g.off[1]) / g.scale[1];
    const double z = (pos[3 * (size_t)i + 2] - g.off[2]) / g.scale[2];
    T4 o;
    o.x = x; o.y = y; o.z = z; o.w = gp_inside(g, x, y, z) ? 1 : 0;
    r[i] = o;
}

__device__ __forceinline__ double gp_value(const GpDev& g, double acc) {
    return g.standard_mean + g.standard_std * (g.mu + g.sigma2 * acc);
}

// The last CTA of a block of points to arrive (its counter returns to 0)
__device__ __forceinline__ bool gp_last(unsigned* arrived) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(arrived + blockIdx.x, gridDim.y - 1) == gridDim.y - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Grid: x over blocks of kGpBlock inference points, y over chunks of `chunk`
// training points.  Each thread sums its chunk in index order; with several
// chunks the last CTA of a block of points adds the partial sums in chunk
// order.  With one chunk the FP64 sum is the CPU form's sequential sum.
//
// FP64 bound: the FP64 pipe (16 clocks of an SM a warp instruction), about 40
// instructions a kernel value.  2048 training points, 1500 points, nu = 5/2:
// 2424 us with images always, IEEE root, division by three, exp() and chunks
// of 512; 311 us here.  200 and 200: 836 and 33 us.
template <int NU2, bool kWrap>
__device__ __forceinline__ double gp_sum64(const GpDev& g, const double4* __restrict__ tile, const double* T, int nt,
                                           double r0, double r1, double r2, double acc) {
    for (int k = 0; k < nt; ++k) {
        const double4 t = tile[k];
        double s0 = t.x - r0, s1 = t.y - r1, s2 = t.z - r2;
        if (kWrap) {
            s0 -= g.pside[0] * floor(s0 * g.sideInv[0] + 0.5);
            s1 -= g.pside[1] * floor(s1 * g.sideInv[1] + 0.5);
            s2 -= g.pside[2] * floor(s2 * g.sideInv[2] + 0.5);
        }
        s0 = s0 * g.invell[0]; s1 = s1 * g.invell[1]; s2 = s2 * g.invell[2];
        double d2 = 0.0;
        d2 += s0 * s0; d2 += s1 * s1; d2 += s2 * s2;
        // 2^-960 .. 2^959 by the exponent bits: a comparison in FP64 costs as much as a product
        const bool normal = (unsigned)__double2hiint(d2) - 0x03F00000u < 0x77F00000u;
        const double r = normal ? root64(d2) : sqrt(d2);
        acc += matern64<NU2>(r, T) * t.w;
    }
    return acc;
}

template <int NU2>
__global__ void __launch_bounds__(kGpBlock)
k_gp64(GpDev g, const double4* __restrict__ train, const double4* __restrict__ points, int count,
       int chunk, unsigned* __restrict__ arrived, double* __restrict__ part, double* __restrict__ out) {
    __shared__ double4 tile[kGpTile];
    __shared__ double T[kExpTable];
    const int i = blockIdx.x * kGpBlock + threadIdx.x;
    const int kb = blockIdx.y * chunk, ke = min(g.n, kb + chunk);
    double4 r = make_double4(0.0, 0.0, 0.0, 1.0);
    if (i < count) r = points[i];
    if (threadIdx.x < kExpTable) T[threadIdx.x] = reinterpret_cast<const double*>(train + g.n)[threadIdx.x];
    const bool inside = __all_sync(0xffffffffu, r.w != 0.0);
    double acc = 0.0;
    for (int k0 = kb; k0 < ke; k0 += kGpTile) {
        const int nt = min(kGpTile, ke - k0);
        __syncthreads();
        for (int k = threadIdx.x; k < nt; k += kGpBlock) tile[k] = train[k0 + k];
        __syncthreads();
        if (i < count) acc = inside ? gp_sum64<NU2, false>(g, tile, T, nt, r.x, r.y, r.z, acc)
                                    : gp_sum64<NU2, true>(g, tile, T, nt, r.x, r.y, r.z, acc);
    }
    if (gridDim.y == 1) {
        if (i < count) out[i] = gp_value(g, acc);
        return;
    }
    if (i < count) part[(size_t)blockIdx.y * count + i] = acc;
    if (!gp_last(arrived) || i >= count) return;
    acc = __ldcg(part + i);
    #pragma unroll 4
    for (int s = 1; s < gridDim.y; ++s) acc += __ldcg(part + (size_t)s * count + i);
    out[i] = gp_value(g, acc);
}

__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x) {
    const float s = __fadd_rn(hi, x);
    const float bp = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
    hi = s;
    lo = __fadd_rn(lo, e);
}

// Mixed form: two points a thread, so that two chains of kernel values are in
// flight over one load of the training point.  Bound: the issue rate, about 40
// instructions a kernel value, twelve less where no image is needed (floor
// takes the special-function pipe, which the root and the exponential need).
// 4096 points, 16384 training points: 151 us and 13 us for the chunks' sums
// with one point a thread, images always and nu chosen in the loop; 94 us here
// and 10 us (cold) for k_gp32_sums.
constexpr int kGpThreads32 = kGpBlock / 2;

template <int NU2, bool kWrap>
__device__ __forceinline__ float gp_kernel32(const float4 t, const float (&r)[3], const float (&ps)[3], const float (&si)[3],
                                             const float (&il)[3]) {
    float s0 = t.x - r[0], s1 = t.y - r[1], s2 = t.z - r[2];
    if (kWrap) {
        s0 = fmaf(-ps[0], floorf(fmaf(s0, si[0], 0.5f)), s0);
        s1 = fmaf(-ps[1], floorf(fmaf(s1, si[1], 0.5f)), s1);
        s2 = fmaf(-ps[2], floorf(fmaf(s2, si[2], 0.5f)), s2);
    }
    s0 *= il[0]; s1 *= il[1]; s2 *= il[2];
    return matern32<NU2>(sqrtf(fmaf(s0, s0, fmaf(s1, s1, s2 * s2)))) * t.w;
}

// the FP32 constants, made on the host
struct GpF { float ps[3], si[3], il[3]; };

template <int NU2>
__global__ void __launch_bounds__(kGpThreads32)
k_gp32(GpDev g, GpF f, const float4* __restrict__ train, const float4* __restrict__ points, int count,
       int chunk, float2* __restrict__ part, double* __restrict__ out) {
    __shared__ float4 tile[kGpTile];
    const int kb = blockIdx.y * chunk, ke = min(g.n, kb + chunk);
    int i[2];
    float r[2][3] = {}, hi[2] = {}, lo[2] = {};
    bool inside = true;
    #pragma unroll
    for (int p = 0; p < 2; ++p) {
        i[p] = blockIdx.x * kGpBlock + p * kGpThreads32 + threadIdx.x;
        if (i[p] < count) {
            const float4 x = points[i[p]];
            r[p][0] = x.x; r[p][1] = x.y; r[p][2] = x.z;
            inside = inside && x.w != 0.f;
        }
    }
    inside = __all_sync(0xffffffffu, inside);
    const bool live = i[0] < count, both = __any_sync(0xffffffffu, i[1] < count);
    for (int k0 = kb; k0 < ke; k0 += kGpTile) {
        const int nt = min(kGpTile, ke - k0);
        __syncthreads();
        for (int k = threadIdx.x; k < nt; k += kGpThreads32) tile[k] = train[k0 + k];
        __syncthreads();
        if (!live) continue;
        if (inside && both) {
            #pragma unroll 4
            for (int k = 0; k < nt; ++k) {
                const float4 t = tile[k];
                two_sum_acc(hi[0], lo[0], gp_kernel32<NU2, false>(t, r[0], f.ps, f.si, f.il));
                two_sum_acc(hi[1], lo[1], gp_kernel32<NU2, false>(t, r[1], f.ps, f.si, f.il));
            }
        } else if (inside) {
            #pragma unroll 4
            for (int k = 0; k < nt; ++k)
                two_sum_acc(hi[0], lo[0], gp_kernel32<NU2, false>(tile[k], r[0], f.ps, f.si, f.il));
        } else {
            for (int k = 0; k < nt; ++k) {
                const float4 t = tile[k];
                two_sum_acc(hi[0], lo[0], gp_kernel32<NU2, true>(t, r[0], f.ps, f.si, f.il));
                if (both) two_sum_acc(hi[1], lo[1], gp_kernel32<NU2, true>(t, r[1], f.ps, f.si, f.il));
            }
        }
    }
    const bool split = gridDim.y > 1;
    #pragma unroll
    for (int p = 0; p < 2; ++p) {
        if (i[p] >= count) continue;
        if (split) part[(size_t)blockIdx.y * count + i[p]] = make_float2(hi[p], lo[p]);
        else out[i[p]] = gp_value(g, (double)hi[p] + (double)lo[p]);
    }
}

// The chunks' parts added in FP64, kGpLanes threads a point.  (Four FP64
// instructions a part: the last CTA of a block of points to arrive would take
// 19 us for 256 points and 76 chunks.)
constexpr int kGpLanes = 4;

__global__ void __launch_bounds__(128)
k_gp32_sums(GpDev g, const float2* __restrict__ part, int nsplit, int count, double* __restrict__ out) {
    const int i = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) / kGpLanes), lane = threadIdx.x % kGpLanes;
    double acc = 0.0;
    if (i < count) {
        #pragma unroll 4
        for (int s = lane; s < nsplit; s += kGpLanes) {
            const float2 x = part[(size_t)s * count + i];
            acc += (double)x.x + (double)x.y;
        }
    }
    #pragma unroll
    for (int o = 1; o < kGpLanes; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (i < count && lane == 0) out[i] = gp_value(g, acc);
}

// --------------------------------------------------------------------------
// GPHeBenzenePotential: fold, GP, long-range switch
// --------------------------------------------------------------------------
struct Benzene {
    double r0, gama, x1, x2, x3, x4, x5, x6, x7, x8, x9, x10, x11, x12;
};

__device__ __forceinline__ double rad2deg(double a) { return (a * 180.0) / 3.14159265358979323846; }
__device__ __forceinline__ double deg2rad(double a) { return (a * 3.14159265358979323846) / 180.0; }

// the fold of GPHeBenzenePotential::V (potential.cpp:5621-5656); cut = 1
// marks the hard core rho < 3, z < 2
__global__ void k_benzene_fold(const double* __restrict__ pos, int count, double* __restrict__ fold,
                               unsigned char* __restrict__ cut) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const double pi = 3.14159265358979323846;
    const double x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1];
    double z = pos[3 * (size_t)i + 2];
    double finx = 0.0, finy = 0.0;
    if (z <= 0.0) z = -z;
    double angle = round(rad2deg(atan2(y, x)) * 10000.0) / 10000.0;
    if (angle < 0.0) angle = 180.0 + (180.0 + angle);
    if (angle <= 30.0) {
        finx = x; finy = y;
    } else {
        double rotateangle = fmod(angle, 60.0) - angle;
        if ((angle + rotateangle) > 30.0) {
            rotateangle = deg2rad(rotateangle);
            const double rx = cos(rotateangle) * x - sin(rotateangle) * y;
            const double ry = sin(rotateangle) * x + cos(rotateangle) * y;
            finx = cos(pi / 3.0) * rx + sin(pi / 3.0) * ry;
            finy = sin(pi / 3.0) * rx - cos(pi / 3.0) * ry;
        } else {
            rotateangle = deg2rad(rotateangle);
            finx = cos(rotateangle) * x - sin(rotateangle) * y;
            finy = sin(rotateangle) * x + cos(rotateangle) * y;
        }
    }
    const double rho = sqrt(finx * finx + finy * finy);
    cut[i] = (rho < 3.0 && z < 2.0) ? 1 : 0;
    fold[3 * (size_t)i] = finx; fold[3 * (size_t)i + 1] = finy; fold[3 * (size_t)i + 2] = z;
}

// GPHeBenzenePotential::long_range (include/potential.h:2455-2480)
__device__ double benzene_long_range(const Benzene& b, double x, double y, double z) {
    const double rnorm = sqrt(x * x + y * y + z * z);
    const double ph0 = atan2(y, x);
    const double th0 = acos(z / rnorm);
    const double tt = cos(th0);
    const double fi = ph0;
    const double normm1 = sqrt(5.0) / 5.0;
    const double normm2 = sqrt(13.0) / 13.0;
    const double normm3 = 0.1792151994e-4;
    const double p1 = -b.x1 / pow(rnorm, 6) - b.x2 / pow(rnorm, 8) - b.x3 / pow(rnorm, 10) - b.x4 / pow(rnorm, 12);
    const double p2 = -normm1 * (1.5 * tt * tt - 0.5) *
                      (b.x5 / pow(rnorm, 6) + b.x6 / pow(rnorm, 8) + b.x7 / pow(rnorm, 10) + b.x8 / pow(rnorm, 12));
    const double p3 = -normm2 * (3.0 / 8.0 + 35.0 / 8.0 * pow(tt, 4) - 15.0 / 4.0 * tt * tt);
    const double p4 = (b.x9 / pow(rnorm, 8) + b.x10 / pow(rnorm, 10) + b.x11 / pow(rnorm, 12));
    const double p5 = -normm3 * 10395.0 * pow(1 - tt * tt, 3) * cos(6 * fi) * b.x12 / pow(rnorm, 10);
    return p1 + p2 + p3 * p4 + p5;
}

__global__ void k_benzene_combine(Benzene b, const double* __restrict__ fold,
                                  const unsigned char* __restrict__ cut, const double* __restrict__ gp,
                                  int count, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    if (cut[i]) { out[i] = 10000.0; return; }
    const double finx = fold[3 * (size_t)i], finy = fold[3 * (size_t)i + 1], z = fold[3 * (size_t)i + 2];
    const double rho = sqrt(finx * finx + finy * finy);
    double d2 = 0.0;
    d2 += finx * finx; d2 += finy * finy; d2 += z * z;
    const double rnorm = sqrt(d2);
    const double h_long = 1.0 / (1.0 + exp(-b.gama * (rnorm - b.r0)));
    double value;
    if (rho > 5.0 || z > 6.5)
        value = (1.0 - h_long) * gp[i] + h_long * benzene_long_range(b, finx, finy, z);
    else
        value = gp[i];
    out[i] = value / 0.695;
}

}  // namespace pgb

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
using namespace pgb;

struct pgb_gp {
    pgb_gp_params p{};
    GpDev g{};
    cudaStream_t stream = nullptr;
    double4* d_train64 = nullptr;
    float4* d_train32 = nullptr;
    Staging stage;
    // per-call scratch: positions, values, fold, cut flags (grown on demand)
    void* d_buf = nullptr;
    size_t buf_bytes = 0;
    void* d_part = nullptr;              // the normalised points, the per-chunk partial sums
    size_t part_bytes = 0;
    unsigned* d_arrived = nullptr;       // a counter a block of points, zero between calls
    int arrived_blocks = 0;
    std::string err;
    int fail(int code, const std::string& m) { err = m; return code; }
    int cfail(cudaError_t e, const char* where) {
        err = std::string("CUDA error ") + cudaGetErrorString(e) + " at " + where;
        return e == cudaErrorMemoryAllocation ? PGB_ENOMEM : PGB_ECUDA;
    }
};

namespace {
thread_local std::string g_gperr;

int ensure_buf(pgb_gp* h, size_t bytes) {
    if (bytes <= h->buf_bytes) return PGB_OK;
    if (h->d_buf) { cudaStreamSynchronize(h->stream); cudaFree(h->d_buf); h->d_buf = nullptr; h->buf_bytes = 0; }
    cudaError_t e = cudaMalloc(&h->d_buf, bytes);
    if (e != cudaSuccess) { h->d_buf = nullptr; return h->cfail(e, "cudaMalloc(GP scratch)"); }
    h->buf_bytes = bytes;
    return PGB_OK;
}

// Chunks of training points so that the grid covers the GPU: about eight CTAs
// an SM (they even out to the last one), chunks of at least 32 points (FP64:
// 8), below which staging a chunk and adding its sum cost what it saves.  From
// 608 blocks of points on there is one chunk.
constexpr int kGpLeast32 = 32, kGpLeast64 = 8;

cudaError_t launch_gp(pgb_gp* h, const double* d_pos, int count, double* d_out) {
    if (count <= 0) return cudaSuccess;
    const int bx = (count + kGpBlock - 1) / kGpBlock;
    const int want = bx >= 4 * 152 ? 1 : (8 * 152 + bx - 1) / bx;
    const int least = h->p.precision == PGB_MIXED ? kGpLeast32 : kGpLeast64;
    const int ns = std::max(1, std::min(want, (h->g.n + least - 1) / least));
    const int chunk = (((h->g.n + ns - 1) / ns + 7) / 8) * 8;
    const int nsplit = (h->g.n + chunk - 1) / chunk;
    // the points, then the chunks' sums
    const size_t points = (size_t)count * (h->p.precision == PGB_MIXED ? sizeof(float4) : sizeof(double4));
    const size_t need = points + (nsplit > 1 ? (size_t)nsplit * count * sizeof(double) : 0);
    if (need > h->part_bytes) {
        if (h->d_part) { cudaStreamSynchronize(h->stream); cudaFree(h->d_part); h->d_part = nullptr; h->part_bytes = 0; }
        cudaError_t e = cudaMalloc(&h->d_part, need);
        if (e != cudaSuccess) { h->d_part = nullptr; return e; }
        h->part_bytes = need;
    }
    if (h->p.precision != PGB_MIXED && nsplit > 1 && bx > h->arrived_blocks) {
        if (h->d_arrived) { cudaStreamSynchronize(h->stream); cudaFree(h->d_arrived); h->d_arrived = nullptr; h->arrived_blocks = 0; }
        const int blocks = std::max(bx, 4 * 152);        // more blocks than that take one chunk
        cudaError_t e = cudaMalloc(&h->d_arrived, blocks * sizeof(unsigned));
        if (e != cudaSuccess) { h->d_arrived = nullptr; return e; }
        if ((e = cudaMemsetAsync(h->d_arrived, 0, blocks * sizeof(unsigned), h->stream)) != cudaSuccess) return e;
        h->arrived_blocks = blocks;
    }
    dim3 grid(bx, nsplit);
    const GpDev& g = h->g;
    char* base = static_cast<char*>(h->d_part);
    auto run = [&](auto k32, auto k64) {
        if (h->p.precision == PGB_MIXED) {
            GpF f;
            for (int d = 0; d < 3; ++d) { f.ps[d] = (float)g.pside[d]; f.si[d] = (float)g.sideInv[d]; f.il[d] = (float)g.invell[d]; }
            float4* r = reinterpret_cast<float4*>(base);
            k_gp_points<float4><<<(count + 127) / 128, 128, 0, h->stream>>>(g, d_pos, count, r);
            float2* part = reinterpret_cast<float2*>(base + points);
            k32<<<grid, kGpThreads32, 0, h->stream>>>(g, f, h->d_train32, r, count, chunk, part, d_out);
            if (nsplit > 1) {
                const int each = 128 / kGpLanes;
                k_gp32_sums<<<(count + each - 1) / each, 128, 0, h->stream>>>(g, part, nsplit, count, d_out);
            }
        } else {
            double4* r = reinterpret_cast<double4*>(base);
            k_gp_points<double4><<<(count + 127) / 128, 128, 0, h->stream>>>(g, d_pos, count, r);
            k64<<<grid, kGpBlock, 0, h->stream>>>(g, h->d_train64, r, count, chunk, h->d_arrived,
                                                  reinterpret_cast<double*>(base + points), d_out);
        }
    };
    if (g.nu2 == 1) run(k_gp32<1>, k_gp64<1>);
    else if (g.nu2 == 3) run(k_gp32<3>, k_gp64<3>);
    else run(k_gp32<5>, k_gp64<5>);
    return cudaGetLastError();
}

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }
}  // namespace

extern "C" {

int pgb_gp_create(const pgb_gp_params* p, const double* training, int n, pgb_gp** out) {
    if (!out) return PGB_EINVAL;
    *out = nullptr;
    if (!p || !training || n <= 0) { g_gperr = "gp_create: parameters and training rows required"; return PGB_EINVAL; }
    // MaternKernel::selectKernel (gpkernel.cpp:71-89): nu = 1/2, 3/2 or 5/2
    int nu2 = 0;
    if (std::fabs(p->matern_nu - 0.5) < 1.0e-12) nu2 = 1;
    else if (std::fabs(p->matern_nu - 1.5) < 1.0e-12) nu2 = 3;
    else if (std::fabs(p->matern_nu - 2.5) < 1.0e-12) nu2 = 5;
    if (!nu2) { g_gperr = "gp_create: only nu = 1/2, 3/2 and 5/2 are supported"; return PGB_EINVAL; }
    if (p->precision != PGB_FP64 && p->precision != PGB_MIXED) { g_gperr = "gp_create: precision"; return PGB_EINVAL; }
    for (int d = 0; d < 3; ++d)
        if (!(p->ell[d] > 0.0) || p->norm_scale[d] == 0.0 || !(p->side[d] > 0.0)) {
            g_gperr = "gp_create: ell, norm_scale and side must be non-zero";
            return PGB_EINVAL;
        }
    int dev = 0;
    if (cudaGetDeviceCount(&dev) != cudaSuccess || dev == 0) {
        cudaGetLastError();
        g_gperr = "gp_create: no CUDA device";
        return PGB_ECUDA;
    }
    pgb_gp* h = new pgb_gp();
    h->p = *p;
    GpDev& g = h->g;
    for (int d = 0; d < 3; ++d) {
        g.off[d] = p->norm_offset[d];
        g.scale[d] = p->norm_scale[d];
        g.invell[d] = 1.0 / p->ell[d];
        g.pside[d] = p->periodic[d] ? p->side[d] : 0.0;
        g.sideInv[d] = 1.0 / p->side[d];
    }
    g.standard_mean = p->standard_mean; g.standard_std = p->standard_std;
    g.mu = p->mean; g.sigma2 = p->sigma2; g.nu2 = nu2; g.n = n;
    double most[3] = {0.0, 0.0, 0.0};                    // a NaN stays: no point is inside then
    // the training rows and, behind them, the 64 powers 2^(j/64) of exp_neg64
    std::vector<double4> t64((size_t)n + kExpTable / 4);
    std::vector<float4> t32((size_t)n);
    for (int k = 0; k < n; ++k) {
        const double* r = training + 4 * (size_t)k;
        t64[k] = make_double4(r[0], r[1], r[2], r[3]);
        t32[k] = make_float4((float)r[0], (float)r[1], (float)r[2], (float)r[3]);
        for (int d = 0; d < 3; ++d) {
            const double x = std::fabs(r[d]);
            most[d] = x > most[d] || x != x ? x : most[d];
        }
    }
    for (int j = 0; j < kExpTable; ++j) reinterpret_cast<double*>(t64.data() + n)[j] = std::exp2(j / 64.0);
    for (int d = 0; d < 3; ++d) {
        g.perInv[d] = p->periodic[d] ? g.sideInv[d] : 0.0;
        g.reach[d] = most[d] * g.perInv[d];
    }
    cudaError_t e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
        h->stage.block = static_cast<char*>(pinned_acquire());
        if (!h->stage.block) e = cudaErrorMemoryAllocation;
    }
    if (e == cudaSuccess) e = cudaMalloc(&h->d_train64, t64.size() * sizeof(double4));
    if (e == cudaSuccess) e = cudaMalloc(&h->d_train32, t32.size() * sizeof(float4));
    if (e == cudaSuccess) e = cudaMemcpy(h->d_train64, t64.data(), t64.size() * sizeof(double4), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(h->d_train32, t32.data(), t32.size() * sizeof(float4), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        g_gperr = std::string("gp_create: ") + cudaGetErrorString(e);
        pgb_gp_destroy(h);
        return e == cudaErrorMemoryAllocation ? PGB_ENOMEM : PGB_ECUDA;
    }
    *out = h;
    return PGB_OK;
}

int pgb_gp_destroy(pgb_gp* h) {
    if (!h) return PGB_OK;
    if (h->stream) cudaStreamSynchronize(h->stream);
    cudaFree(h->d_train64); cudaFree(h->d_train32); cudaFree(h->d_buf); cudaFree(h->d_part);
    cudaFree(h->d_arrived);
    pinned_release(h->stage.block);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return PGB_OK;
}

const char* pgb_gp_last_error(const pgb_gp* h) { return h ? h->err.c_str() : g_gperr.c_str(); }
void* pgb_gp_stream(pgb_gp* h) { return h ? (void*)h->stream : nullptr; }

int pgb_gp_eval_device_async(pgb_gp* h, const double* d_pos, double* d_values, int count) {
    if (!h || count < 0 || (count > 0 && (!d_pos || !d_values))) return PGB_EINVAL;
    cudaError_t e = launch_gp(h, d_pos, count, d_values);
    if (e != cudaSuccess) return h->cfail(e, "GP launch");
    return PGB_OK;
}

// A call's positions as the kernels read them and values as they write them:
// both in the handle's host block when they fit there, else nullptr.
static double* gp_direct(pgb_gp* h, const double* pos, size_t pb, size_t vb) {
    char* in = vb <= kResultBytes ? h->stage.take(pb, h->stream) : nullptr;
    if (in) std::memcpy(in, pos, pb);
    return reinterpret_cast<double*>(in);
}

int pgb_gp_eval(pgb_gp* h, const double* pos, double* values, int count) {
    if (!h || count < 0 || (count > 0 && (!pos || !values))) return PGB_EINVAL;
    if (count == 0) return PGB_OK;
    const size_t pb = (size_t)count * 3 * sizeof(double), vb = (size_t)count * sizeof(double);
    if (double* in = gp_direct(h, pos, pb, vb)) {
        cudaError_t e = launch_gp(h, in, count, reinterpret_cast<double*>(h->stage.result()));
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) return h->cfail(e, "GP eval");
        std::memcpy(values, h->stage.result(), vb);
        return PGB_OK;
    }
    int rc = ensure_buf(h, al256(pb) + vb); if (rc) return rc;
    char* base = static_cast<char*>(h->d_buf);
    double* d_pos = reinterpret_cast<double*>(base);
    double* d_val = reinterpret_cast<double*>(base + al256(pb));
    cudaError_t e = cudaMemcpyAsync(d_pos, pos, pb, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = launch_gp(h, d_pos, count, d_val);
    if (e == cudaSuccess) e = cudaMemcpyAsync(values, d_val, vb, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return h->cfail(e, "GP eval");
    return PGB_OK;
}

int pgb_gp_math_check(const double* x, int n, int what, double* out) {
    if (n <= 0 || !x || !out || what < 0 || what > 3) return PGB_EINVAL;
    double t[kExpTable];
    for (int j = 0; j < kExpTable; ++j) t[j] = std::exp2(j / 64.0);
    double* d = nullptr;
    const size_t nb = (size_t)n * sizeof(double);
    cudaError_t e = cudaMalloc(&d, 2 * nb + sizeof(t));
    if (e == cudaSuccess) e = cudaMemcpy(d, x, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + 2 * (size_t)n, t, sizeof(t), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_gp_math<<<(n + 255) / 256, 256>>>(d, n, what, d + 2 * (size_t)n, d + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, nb, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? PGB_OK : PGB_ECUDA;
}

int pgb_gp_benzene_v(pgb_gp* h, const double* pos, double* values, int count) {
    if (!h || count < 0 || (count > 0 && (!pos || !values))) return PGB_EINVAL;
    if (count == 0) return PGB_OK;
    // GPHeBenzenePotential constants (include/potential.h:2433-2448)
    Benzene b{5.765366674e+00, 1.671477473e+01, 2.290626821e+05, 4.069217828e+06, 9.542607077e+07, 0.0,
              -4.775615288e+04, -1.263899296e+07, -2.959330054e+08, 0.0, 9.511488779e+05,
              2.551023972e+08, 0.0, 1.883887454e+08};
    const size_t pb = (size_t)count * 3 * sizeof(double), vb = (size_t)count * sizeof(double);
    const size_t o_fold = al256(pb), o_gp = o_fold + al256(pb), o_val = o_gp + al256(vb),
                 o_cut = o_val + al256(vb);
    int rc = ensure_buf(h, o_cut + (size_t)count); if (rc) return rc;
    char* base = static_cast<char*>(h->d_buf);
    double* d_pos = reinterpret_cast<double*>(base);
    double* d_fold = reinterpret_cast<double*>(base + o_fold);
    double* d_gp = reinterpret_cast<double*>(base + o_gp);
    double* d_val = reinterpret_cast<double*>(base + o_val);
    unsigned char* d_cut = reinterpret_cast<unsigned char*>(base + o_cut);
    const int blocks = (count + 255) / 256;
    double* in = gp_direct(h, pos, pb, vb);
    cudaError_t e = cudaSuccess;
    if (in) { d_pos = in; d_val = reinterpret_cast<double*>(h->stage.result()); }
    else e = cudaMemcpyAsync(d_pos, pos, pb, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) {
        k_benzene_fold<<<blocks, 256, 0, h->stream>>>(d_pos, count, d_fold, d_cut);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = launch_gp(h, d_fold, count, d_gp);
    if (e == cudaSuccess) {
        k_benzene_combine<<<blocks, 256, 0, h->stream>>>(b, d_fold, d_cut, d_gp, count, d_val);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && !in) e = cudaMemcpyAsync(values, d_val, vb, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess && in) std::memcpy(values, d_val, vb);
    if (e != cudaSuccess) return h->cfail(e, "GP benzene");
    return PGB_OK;
}

}  // extern "C"
