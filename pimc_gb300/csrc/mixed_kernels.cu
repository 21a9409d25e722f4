// mixed_kernels.cu -- FP32 pair evaluation with FP64 accumulation.
//
// Pair potentials and gradients are the analytic Aziz form in FP32 (no
// table), read from the float4 position mirror; each thread accumulates its
// pairs with Kahan compensation and the block folds the partial sums in FP64.
#include <algorithm>

#include "pgb_device.cuh"

namespace pgb {

__global__ void k_pos32_from64(PathView v, float4* __restrict__ out) {
    size_t n = (size_t)v.M * v.Ne;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        size_t s = i / v.Ne, p = i % v.Ne;
        const double* X = v.pos + s * 3 * v.Ne;
        out[i] = make_float4((float)X[p], (float)X[v.Ne + p], (float)X[2 * v.Ne + p], 0.f);
    }
}

cudaError_t launch_pos32_from64(const PathView& v, float4* d_pos32, cudaStream_t s) {
    size_t n = (size_t)v.M * v.Ne;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) return cudaSuccess;
    k_pos32_from64<<<blocks, 256, 0, s>>>(v, d_pos32);
    return cudaGetLastError();
}

// The box in FP32, made on the host: in a kernel the six conversions take the
// FP64 pipe 16 clocks each, for every warp.
struct BoxF { float L0, L1, L2, I0, I1, I2; };
static BoxF box_f(const PathView& v) {
    return {(float)v.side[0], (float)v.side[1], (float)v.side[2],
            (float)v.sideInv[0], (float)v.sideInv[1], (float)v.sideInv[2]};
}

// d^2V/dr^2 in FP32 (potential.cpp:1877-1907 with d2F of potential.h:976-983)
__device__ __forceinline__ float aziz_d2v32(float r2, const AzizF& a) {
    float rinv = rsqrtf(r2);
    float x = r2 * rinv * a.rminv;
    float ix = rinv * a.rm;
    float ix2 = ix * ix;
    float ix6 = ix2 * ix2 * ix2;
    float e = __expf(x * fmaf(a.beta, x, -a.alpha));
    float ab = fmaf(-2.0f * a.beta, x, a.alpha);
    float T1 = a.A * fmaf(ab, ab, 2.0f * a.beta) * e;
    float t = fmaxf(fmaf(a.D, ix, -1.0f), 0.0f);
    float F = __expf(-t * t);
    float p0 = ix6 * fmaf(ix2, fmaf(ix2, a.C10, a.C8), a.C6);
    float p1 = ix * ix6 * fmaf(ix2, fmaf(ix2, 10.0f * a.C10, 8.0f * a.C8), 6.0f * a.C6);
    float p2 = ix2 * ix6 * fmaf(ix2, fmaf(ix2, 110.0f * a.C10, 72.0f * a.C8), 42.0f * a.C6);
    float dF = 2.0f * a.D * ix2 * t * F;
    float Dix = a.D * ix;
    float d2F = (x < a.D) ? 2.0f * a.D * ix2 * ix * (2.0f * Dix * Dix * Dix - 4.0f * Dix * Dix - Dix + 2.0f) * F : 0.0f;
    return a.eps_rm * a.rminv * (T1 - p2 * F + 2.0f * p1 * dF - p0 * d2F);
}

constexpr int kBeadBlock32 = 256;

__global__ void __launch_bounds__(kBeadBlock32)
k_bead_actions32(PathView v, AzizF az, const int2* __restrict__ beads, int k, int shift,
                 int mode, double tau, double lambda, double vf0, double vf1, double gf0,
                 double gf1, const double* __restrict__ over, double* __restrict__ out,
                 const float4* __restrict__ fall) {
    extern __shared__ float4 lpos[];
    int* lidx = reinterpret_cast<int*>(lpos + v.Ne);
    __shared__ double red[kBeadBlock32 / 32];
    __shared__ int wcount[kBeadBlock32 / 32];
    __shared__ int s_total;
    const int Ne = v.Ne;
    const int b = blockIdx.x;
    const int s = beads[b].x, p = beads[b].y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (s < 0 || s >= v.M || p < 0 || p >= Ne || !v.on[(size_t)s * Ne + p]) {
        if (tid == 0) out[b] = 0.0;
        return;
    }
    const int eo = s % 2;
    const double vf = eo ? vf1 : vf0, gf = eo ? gf1 : gf0;
    const double t = (double)shift * tau;
    const bool need_v = (mode != PGB_ACTION_CORR);
    const bool need_c = (mode == PGB_ACTION_CORR) ? (gf > kEPS)
                      : (mode == PGB_ACTION_FULL) ? (shift == 1 && gf > kEPS) : false;
    const float L0 = (float)v.side[0], L1 = (float)v.side[1], L2 = (float)v.side[2];
    const float I0 = (float)v.sideInv[0], I1 = (float)v.sideInv[1], I2 = (float)v.sideInv[2];
    const float rc2 = (float)v.rc2;
    const float4* P = v.pos32 + (size_t)s * Ne;
    const float4 r1 = over ? make_float4((float)over[3 * b], (float)over[3 * b + 1],
                                         (float)over[3 * b + 2], 0.f)
                           : P[p];
    const int st1 = bead_state(v, s, p);
    if (tid == 0) s_total = 0;
    __syncthreads();
    KahanF vs;
    for (int base = 0; base < Ne; base += kBeadBlock32) {
        int j = base + tid;
        bool in = false;
        float4 rj = make_float4(0, 0, 0, 0);
        if (j < Ne && j != p && v.on[(size_t)s * Ne + j]) {
            rj = P[j];
            float dx = min_image32(rj.x - r1.x, L0, I0);
            float dy = min_image32(rj.y - r1.y, L1, I1);
            float dz = min_image32(rj.z - r1.z, L2, I2);
            float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (r2 < rc2) {
                in = true;
                if (need_v) vs.add((float)pair_factor(st1, bead_state(v, s, j)) * aziz_v32(r2, az));
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) wcount[w] = __popc(m);
        __syncthreads();
        int off = s_total;
        for (int i = 0; i < w; ++i) off += wcount[i];
        if (in) {
            const int slot_ = off + __popc(m & ((1u << lane) - 1u));
            lpos[slot_] = rj;
            lidx[slot_] = j;
        }
        __syncthreads();
        if (tid == 0) { int tot = 0; for (int i = 0; i < kBeadBlock32 / 32; ++i) tot += wcount[i]; s_total += tot; }
        __syncthreads();
    }
    const int nlist = s_total;
    double Vnn = need_v ? block_sum(vs.value(), red) : 0.0;
    double corr_g = 0.0;
    if (need_c && fall) {
        // Every active same-slice bead is in the list (rc covers the box), so
        // the inner sum of gradVnnSquared, F3(b2) = sum over b3 != p, b2 of
        // gradV(r_b2 - r_b3), does not depend on where p is: it is the slice
        // force on b2 less p's own term at p's current position.  O(n) per bead.
        const float4 rpo = P[p];
        KahanF ts;
        float f1x = 0.f, f1y = 0.f, f1z = 0.f;
        const float4* Fs = fall + (size_t)s * Ne;
        for (int n = tid; n < nlist; n += kBeadBlock32) {
            const float4 r2v = lpos[n];
            const float dx = min_image32(r2v.x - r1.x, L0, I0);
            const float dy = min_image32(r2v.y - r1.y, L1, I1);
            const float dz = min_image32(r2v.z - r1.z, L2, I2);
            const float g = aziz_g32(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), az);
            const float F2x = g * dx, F2y = g * dy, F2z = g * dz;
            f1x -= F2x; f1y -= F2y; f1z -= F2z;
            float Fox = F2x, Foy = F2y, Foz = F2z;
            if (over) {
                const float ox = min_image32(r2v.x - rpo.x, L0, I0);
                const float oy = min_image32(r2v.y - rpo.y, L1, I1);
                const float oz = min_image32(r2v.z - rpo.z, L2, I2);
                const float go = aziz_g32(fmaf(ox, ox, fmaf(oy, oy, oz * oz)), az);
                Fox = go * ox; Foy = go * oy; Foz = go * oz;
            }
            const float4 fa = Fs[lidx[n]];
            const float F3x = fa.x - Fox, F3y = fa.y - Foy, F3z = fa.z - Foz;
            const float d22 = fmaf(F2x, F2x, fmaf(F2y, F2y, F2z * F2z));
            const float d23 = fmaf(F2x, F3x, fmaf(F2y, F3y, F2z * F3z));
            ts.add(fmaf(2.0f, d23, d22));
        }
        double T = block_sum(ts.value(), red);
        double Fx = block_sum((double)f1x, red), Fy = block_sum((double)f1y, red),
               Fz = block_sum((double)f1z, red);
        corr_g = T + (Fx * Fx + Fy * Fy + Fz * Fz);
    } else if (need_c) {
        KahanF ts;
        float f1x = 0.f, f1y = 0.f, f1z = 0.f;
        for (int n = tid; n < nlist; n += kBeadBlock32) {
            float4 r2v = lpos[n];
            float dx = min_image32(r2v.x - r1.x, L0, I0);
            float dy = min_image32(r2v.y - r1.y, L1, I1);
            float dz = min_image32(r2v.z - r1.z, L2, I2);
            float g = aziz_g32(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), az);
            float F2x = g * dx, F2y = g * dy, F2z = g * dz;
            f1x -= F2x; f1y -= F2y; f1z -= F2z;
            float F3x = 0.f, F3y = 0.f, F3z = 0.f;
            for (int m2 = 0; m2 < nlist; ++m2) {
                if (m2 == n) continue;
                float4 r3 = lpos[m2];
                float ex = min_image32(r2v.x - r3.x, L0, I0);
                float ey = min_image32(r2v.y - r3.y, L1, I1);
                float ez = min_image32(r2v.z - r3.z, L2, I2);
                float g3 = aziz_g32(fmaf(ex, ex, fmaf(ey, ey, ez * ez)), az);
                F3x = fmaf(g3, ex, F3x); F3y = fmaf(g3, ey, F3y); F3z = fmaf(g3, ez, F3z);
            }
            float d22 = fmaf(F2x, F2x, fmaf(F2y, F2y, F2z * F2z));
            float d23 = fmaf(F2x, F3x, fmaf(F2y, F3y, F2z * F3z));
            ts.add(fmaf(2.0f, d23, d22));
        }
        double T = block_sum(ts.value(), red);
        double Fx = block_sum((double)f1x, red), Fy = block_sum((double)f1y, red),
               Fz = block_sum((double)f1z, red);
        corr_g = T + (Fx * Fx + Fy * Fy + Fz * Fz);
    }
    if (tid == 0) {
        double bareU = vf * t * Vnn;
        double corU = need_c ? gf * t * t * t * lambda * corr_g : 0.0;
        out[b] = (mode == PGB_ACTION_BARE) ? bareU : (mode == PGB_ACTION_CORR) ? corU : bareU + corU;
    }
}

cudaError_t launch_bead_actions32(const PathView& v, AzizParams a, const int2* d_beads, int k,
                                  int shift, int mode, double tau, double lambda,
                                  const double vf[2], const double gf[2], const double* d_over,
                                  double* d_out, cudaStream_t s, const float4* d_force) {
    if (k <= 0) return cudaSuccess;
    size_t smem = (size_t)v.Ne * (sizeof(float4) + sizeof(int));
    if (smem > 200 * 1024) return cudaErrorInvalidValue;     // one slice's list in shared memory
    {
        const cudaError_t ae = set_smem_limit(k_bead_actions32, 200 * 1024);
        if (ae != cudaSuccess) return ae;
    }
    k_bead_actions32<<<k, kBeadBlock32, smem, s>>>(v, make_aziz_f(a), d_beads, k, shift, mode,
                                                   tau, lambda, vf[0], vf[1], gf[0], gf[1], d_over,
                                                   d_out, d_force);
    return cudaGetLastError();
}

// One warp per bead when every active same-slice bead is in the list (the
// cutoff covers the box): no list compaction, and the GSF correction in O(n)
// from the cached slice forces `fall` (see k_bead_actions32).  With `delta`
// set and trial positions given, the warp evaluates the bead at its trial and
// at its current position and writes U(trial) - U(current): one launch per
// batch of trial moves.  Each warp takes kBeadsPerWarp beads in turn and
// leaves its FP32 (hi, lo) sums in shared memory; the FP64 assembly of the
// actions then runs one bead per lane, so the narrow FP64 pipe sees a full
// warp per instruction instead of one lane.
constexpr int kWarpBeadBlock = 256;
constexpr int kBeadsPerWarp = 4;
constexpr int kBeadsPerBlock = (kWarpBeadBlock / 32) * kBeadsPerWarp;   // 32

__device__ __forceinline__ float pair_factor32(int st1, int st2) {
    if (st1 == 2 && st2 == 2) return 1.0f;
    if (st1 == 0 && st2 == 0) return 0.0f;
    return 0.5f;
}

// What a bead's sums are multiplied by, vf t and gf t^3 lambda for t = shift
// tau, even and odd slices: products made once on the host in the order the
// action takes them (a kernel's one lane would wait 64 clocks for each).
struct Scales32 { double bare[2], cor[2], gf[2]; };

static Scales32 scales32(int shift, double tau, double lambda, const double vf[2], const double gf[2]) {
    const double t = (double)shift * tau;
    Scales32 a;
    for (int o = 0; o < 2; ++o) { a.bare[o] = vf[o] * t; a.cor[o] = gf[o] * t * t * t * lambda; a.gf[o] = gf[o]; }
    return a;
}

// A bead's action from its FP64 sums; the roundings are spelt out so that the
// two kernels that assemble actions give the same bits.
__device__ __forceinline__ double assemble32(int mode, bool need_c, double bare, double cor, double V, double T,
                                             double fx, double fy, double fz) {
    const double bareU = __dmul_rn(bare, V);
    double corU = 0.0;
    if (need_c) {
        const double f2 = __fma_rn(fx, fx, __fma_rn(fy, fy, __dmul_rn(fz, fz)));
        corU = __dmul_rn(cor, __dadd_rn(T, f2));
    }
    return (mode == PGB_ACTION_BARE) ? bareU : (mode == PGB_ACTION_CORR) ? corU : __dadd_rn(bareU, corU);
}

__global__ void __launch_bounds__(kWarpBeadBlock)
k_bead_actions32_full(PathView v, AzizF az, const int2* __restrict__ beads, int k, int shift,
                      int mode, const Scales32 sc, const double* __restrict__ over, const float4* __restrict__ fall,
                      int delta, double* __restrict__ out) {
    // per bead of the block: Vn Vo Tn To Fnx Fny Fnz Fox Foy Foz as (hi, lo)
    __shared__ float2 s_part[kBeadsPerBlock][10];
    __shared__ int s_state[kBeadsPerBlock];      // 0 inactive or out of range, 1 active
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int Ne = v.Ne;
    const bool both = delta && over;             // also the current position
    const float L0 = (float)v.side[0], L1 = (float)v.side[1], L2 = (float)v.side[2];
    const float I0 = (float)v.sideInv[0], I1 = (float)v.sideInv[1], I2 = (float)v.sideInv[2];
    for (int r = 0; r < kBeadsPerWarp; ++r) {
        const int lb = warp * kBeadsPerWarp + r;           // bead within the block
        const int b = blockIdx.x * kBeadsPerBlock + lb;
        if (b >= k) { if (lane == 0) s_state[lb] = 0; continue; }
        const int s = beads[b].x, p = beads[b].y;
        if (s < 0 || s >= v.M || p < 0 || p >= Ne || !v.on[(size_t)s * Ne + p]) {
            if (lane == 0) s_state[lb] = 0;
            continue;
        }
        const int eo = s % 2;
        const double gf = eo ? sc.gf[1] : sc.gf[0];
        const bool need_v = (mode != PGB_ACTION_CORR);
        const bool need_c = (mode == PGB_ACTION_CORR) ? (gf > kEPS)
                          : (mode == PGB_ACTION_FULL) ? (shift == 1 && gf > kEPS) : false;
        const float4* P = v.pos32 + (size_t)s * Ne;
        const float4* Fs = fall + (size_t)s * Ne;
        const float4 rpo = P[p];
        const float4 r1 = over ? make_float4((float)over[3 * b], (float)over[3 * b + 1],
                                             (float)over[3 * b + 2], 0.f) : rpo;
        const int st1 = bead_state(v, s, p);
        KahanF vn, vo, tn, to;
        float fnx = 0.f, fny = 0.f, fnz = 0.f, fox = 0.f, foy = 0.f, foz = 0.f;
        for (int j = lane; j < Ne; j += 32) {
            if (j == p || !v.on[(size_t)s * Ne + j]) continue;
            const float4 rj = P[j];
            const float dx = min_image32(rj.x - r1.x, L0, I0);
            const float dy = min_image32(rj.y - r1.y, L1, I1);
            const float dz = min_image32(rj.z - r1.z, L2, I2);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const float fac = pair_factor32(st1, bead_state(v, s, j));
            float ox = dx, oy = dy, oz = dz, ro2 = r2;
            if (over) {
                ox = min_image32(rj.x - rpo.x, L0, I0);
                oy = min_image32(rj.y - rpo.y, L1, I1);
                oz = min_image32(rj.z - rpo.z, L2, I2);
                ro2 = fmaf(ox, ox, fmaf(oy, oy, oz * oz));
            }
            if (need_v) {
                vn.add(fac * aziz_v32(r2, az));
                if (both) vo.add(fac * aziz_v32(ro2, az));
            }
            if (need_c) {
                const float g = aziz_g32(r2, az);
                const float F2x = g * dx, F2y = g * dy, F2z = g * dz;
                float Fox = F2x, Foy = F2y, Foz = F2z;
                if (over) {
                    const float go = aziz_g32(ro2, az);
                    Fox = go * ox; Foy = go * oy; Foz = go * oz;
                }
                const float4 fa = Fs[j];
                // F3: the slice force on j less the term of p at its current position
                const float F3x = fa.x - Fox, F3y = fa.y - Foy, F3z = fa.z - Foz;
                fnx -= F2x; fny -= F2y; fnz -= F2z;
                tn.add(fmaf(2.0f, fmaf(F2x, F3x, fmaf(F2y, F3y, F2z * F3z)),
                            fmaf(F2x, F2x, fmaf(F2y, F2y, F2z * F2z))));
                if (both) {
                    fox -= Fox; foy -= Foy; foz -= Foz;
                    to.add(fmaf(2.0f, fmaf(Fox, F3x, fmaf(Foy, F3y, Foz * F3z)),
                                fmaf(Fox, Fox, fmaf(Foy, Foy, Foz * Foz))));
                }
            }
        }
        // only the sums the action has: a butterfly is 45 instructions
        float2 parts[10] = {};
        parts[0] = warp_ff(vn);
        if (both) parts[1] = warp_ff(vo);
        if (need_c) {
            parts[2] = warp_ff(tn);
            parts[4] = ff_butterfly(fnx, 0.f); parts[5] = ff_butterfly(fny, 0.f); parts[6] = ff_butterfly(fnz, 0.f);
            if (both) {
                parts[3] = warp_ff(to);
                parts[7] = ff_butterfly(fox, 0.f); parts[8] = ff_butterfly(foy, 0.f); parts[9] = ff_butterfly(foz, 0.f);
            }
        }
        if (lane == 0) {
            #pragma unroll
            for (int q = 0; q < 10; ++q) s_part[lb][q] = parts[q];
            s_state[lb] = 1;
        }
    }
    __syncthreads();
    if (warp == 0) {
        // one bead of the block per lane: the FP64 assembly of its action(s)
        const int b = blockIdx.x * kBeadsPerBlock + lane;
        if (b < k) {
            double res = 0.0;
            if (s_state[lane]) {
                const int s = beads[b].x;
                const int eo = s % 2;
                const double bare = eo ? sc.bare[1] : sc.bare[0], cor = eo ? sc.cor[1] : sc.cor[0];
                const double gf = eo ? sc.gf[1] : sc.gf[0];
                const bool need_v = (mode != PGB_ACTION_CORR);
                const bool need_c = (mode == PGB_ACTION_CORR) ? (gf > kEPS)
                                  : (mode == PGB_ACTION_FULL) ? (shift == 1 && gf > kEPS) : false;
                const float2* q = s_part[lane];
                auto dd = [](float2 x) { return (double)x.x + (double)x.y; };
                auto action = [&](double V, double T, double fx, double fy, double fz) {
                    return assemble32(mode, need_c, bare, cor, V, T, fx, fy, fz);
                };
                res = action(need_v ? dd(q[0]) : 0.0, dd(q[2]), dd(q[4]), dd(q[5]), dd(q[6]));
                if (both)
                    res = __dsub_rn(res, action(need_v ? dd(q[1]) : 0.0, dd(q[3]), dd(q[7]), dd(q[8]), dd(q[9])));
            }
            out[b] = res;
        }
    }
}

cudaError_t launch_bead_actions32_full(const PathView& v, AzizParams a, const int2* d_beads, int k,
                                       int shift, int mode, double tau, double lambda,
                                       const double vf[2], const double gf[2], const double* d_over,
                                       const float4* d_force, int delta, double* d_out,
                                       cudaStream_t s) {
    if (k <= 0) return cudaSuccess;
    k_bead_actions32_full<<<(k + kBeadsPerBlock - 1) / kBeadsPerBlock, kWarpBeadBlock, 0, s>>>(
        v, make_aziz_f(a), d_beads, k, shift, mode, scales32(shift, tau, lambda, vf, gf),
        d_over, d_force, delta, d_out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Many trials of few beads.  A trial's difference needs the bead's current
// action and, for the gradient term, every partner's force less the bead's
// own term: the same for all trials of the bead.  The trials are sorted by
// bead on the device (count, offsets, scatter: the sorted record is the FP32
// position and the trial's index), a warp takes a bead and a run of its
// trials, evaluates its current position once, keeps the partners (and those
// forces) in shared memory and then makes the trials four at a time, so four
// independent chains of pair arithmetic are in flight.  The sums of a group are reduced together by
// recursive halving, in the butterfly's own tree, so every sum has the bits
// k_bead_actions32_full gives it; the FP64 assembly runs one trial a lane.
//
// Bound: the issue rate, 47 instructions a pair (79 with the gradient), and
// instruction fetch: the loops of both parities and the reductions together
// are larger than the instruction caches, so the even slices' beads go first
// and the reductions are not inlined (1.01 -> 0.87 ms at the time).  10^6
// trials, N = 256, M = 250, GSF: 2.75 ms with both positions evaluated for every
// trial, 0.81 ms here.
//
// A run is as long as two average beads' trials and 16 more, so that evenly
// spread trials stay whole.  A second launch makes the trials of a bead
// beyond its first run, which go to the warps by their place: of a run's length
// of consecutive sorted trials at most one starts another run, and it belongs
// to the bead of the first of them.  With all trials of a bead on one warp, 10^6
// trials of one slice's 256 beads took 4.6 ms, of one worldline's 250 beads 7.9
// ms, 10^5 trials of one bead of 64 particles 51 ms; 1.2, 0.95 and 0.18 ms here
// (unsorted 2.7, 2.6 and 0.15).
// ---------------------------------------------------------------------------
constexpr int kTrialWarps = 4;
constexpr int kTrialRun = 32;                    // trials in a run at least, and their step
// Sorting pays from about three trials a bead on (N = 256, gradient: 2 a bead
// 306 against 374 us, 4 a bead 398 against 719; N = 400: 2 a bead 227 against
// 220, 4 a bead 282 against 395) once its small launches, 12 to 15 us, are
// less than the pairs saved (N = 64: 4 a bead, 32 k trials 58 against 54 us, 16
// a bead 92 against 168; N = 16: 8 k trials 34 against 19).
constexpr double kTrialsPerBead = 3.0;
constexpr double kTrialPairs = 2.5e6;            // trials times partners

__device__ __forceinline__ bool bead_active(const PathView& v, int2 b) {
    return b.x >= 0 && b.x < v.M && b.y >= 0 && b.y < v.Ne && v.on[(size_t)b.x * v.Ne + b.y];
}

// each trial's rank among its bead's trials (kept in the first word of its
// output until the scatter)
__global__ void k_trial_count(PathView v, const int2* __restrict__ beads, int k, int* __restrict__ count,
                              double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k) return;
    const int2 b = beads[i];
    if (bead_active(v, b)) *reinterpret_cast<int*>(out + i) = atomicAdd(count + (size_t)b.x * v.Ne + b.y, 1);
}

// a slice's beads get consecutive places; the slices any order
// (cursor[0] ends as the number of trials; cursor[1] tells that a bead has more
// than a run)
__global__ void __launch_bounds__(256)
k_trial_offsets(PathView v, const int* __restrict__ count, int run, int* __restrict__ cursor, int* __restrict__ offset) {
    __shared__ int wsum[8], s_base;
    const int s = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int b0 = 0; b0 < v.Ne; b0 += 256) {
        const int b = b0 + threadIdx.x;
        const int c = b < v.Ne ? count[(size_t)s * v.Ne + b] : 0;
        if (c > run) cursor[1] = 1;
        int x = c;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < 8; ++w) { const int y = wsum[w]; wsum[w] = t; t += y; }
            s_base = t ? atomicAdd(cursor, t) : 0;
        }
        __syncthreads();
        if (b < v.Ne) offset[(size_t)s * v.Ne + b] = s_base + wsum[warp] + x - c;
        __syncthreads();
    }
}

__global__ void k_trial_scatter(PathView v, const int2* __restrict__ beads, const double* __restrict__ pos, int k,
                                const int* __restrict__ offset, float4* __restrict__ sorted, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k) return;
    const int2 b = beads[i];
    if (!bead_active(v, b)) { out[i] = 0.0; return; }
    const int at = offset[(size_t)b.x * v.Ne + b.y] + *reinterpret_cast<const int*>(out + i);
    sorted[at] = make_float4((float)pos[3 * (size_t)i], (float)pos[3 * (size_t)i + 1], (float)pos[3 * (size_t)i + 2],
                             __int_as_float(i));
}

// one step of ff_butterfly's tree
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
    const float sum = a.x + b.x;
    const float bp = sum - a.x;
    const float err = (a.x - (sum - bp)) + (b.x - bp);
    return make_float2(sum, (a.y + b.y) + err);
}
__device__ __forceinline__ float2 ff_xor(float2 a, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}
// R sums over the warp; lane l returns sum l / (32 / R)
template <int R>
__device__ __forceinline__ float2 ff_halve(float2 (&x)[R], int lane) {
    int o = 16;
    #pragma unroll
    for (int h = R / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
        #pragma unroll
        for (int i = 0; i < h; ++i) x[i] = ff_add(up ? x[i + h] : x[i], ff_xor(up ? x[i] : x[i + h], o));
    }
    for (; o > 0; o >>= 1) x[0] = ff_add(x[0], ff_xor(x[0], o));
    return x[0];
}

static __device__ __noinline__ float2 ff_sums4(float2 a, float2 b, float2 c, float2 d, int lane) {
    float2 x[4] = {a, b, c, d};
    return ff_halve<4>(x, lane);
}
static __device__ __noinline__ float2 ff_sums2(float2 a, float2 b, int lane) {
    float2 x[2] = {a, b};
    return ff_halve<2>(x, lane);
}
template <int R>
__device__ __forceinline__ float2 ff_sums(float2 (&x)[R], int lane) {
    if constexpr (R == 4) return ff_sums4(x[0], x[1], x[2], x[3], lane);
    else return ff_sums2(x[0], x[1], lane);
}

// what a warp keeps of up to 32 finished trials: V T F(3) at the trial
// position, then at the current one, as (hi, lo)
struct TrialBuffer {
    float2 part[10][32];
    int id[32], slice[32];
};

// R trials of one bead over the staged partners (P: position and pair factor,
// negative for none; F: the partner's force less the bead's own term)
template <int R, bool kC>
__device__ __forceinline__ void trial_group(const float4* __restrict__ trial, int count, const float4* P, const float4* F,
                                            int Ne, const BoxF& B, const AzizF& az, bool need_v, int lane, int slice,
                                            const float2 (&old)[5], TrialBuffer& buf, int used) {
    float4 r[R];
    #pragma unroll
    for (int i = 0; i < R; ++i) r[i] = trial[min(i, count - 1)];
    KahanF vn[R], tn[R];
    float fx[R], fy[R], fz[R];
    #pragma unroll
    for (int i = 0; i < R; ++i) fx[i] = fy[i] = fz[i] = 0.f;
    for (int j = lane; j < Ne; j += 32) {
        const float4 rj = P[j];
        if (rj.w < 0.f) continue;
        float4 f3 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kC) f3 = F[j];
        #pragma unroll
        for (int i = 0; i < R; ++i) {
            const float dx = min_image32(rj.x - r[i].x, B.L0, B.I0);
            const float dy = min_image32(rj.y - r[i].y, B.L1, B.I1);
            const float dz = min_image32(rj.z - r[i].z, B.L2, B.I2);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (need_v) vn[i].add(rj.w * aziz_v32(r2, az));
            if (kC) {
                const float g = aziz_g32(r2, az);
                const float F2x = g * dx, F2y = g * dy, F2z = g * dz;
                fx[i] -= F2x; fy[i] -= F2y; fz[i] -= F2z;
                tn[i].add(fmaf(2.0f, fmaf(F2x, f3.x, fmaf(F2y, f3.y, F2z * f3.z)),
                               fmaf(F2x, F2x, fmaf(F2y, F2y, F2z * F2z))));
            }
        }
    }
    const int mine = lane / (32 / R), slot = used + mine;
    const bool write = (lane & (32 / R - 1)) == 0 && mine < count;
    float2 x[R], sum[5] = {};
    #pragma unroll
    for (int i = 0; i < R; ++i) x[i] = make_float2(vn[i].s, -vn[i].c);
    sum[0] = ff_sums<R>(x, lane);
    if (kC) {
        #pragma unroll
        for (int i = 0; i < R; ++i) x[i] = make_float2(tn[i].s, -tn[i].c);
        sum[1] = ff_sums<R>(x, lane);
        #pragma unroll
        for (int i = 0; i < R; ++i) x[i] = make_float2(fx[i], 0.f);
        sum[2] = ff_sums<R>(x, lane);
        #pragma unroll
        for (int i = 0; i < R; ++i) x[i] = make_float2(fy[i], 0.f);
        sum[3] = ff_sums<R>(x, lane);
        #pragma unroll
        for (int i = 0; i < R; ++i) x[i] = make_float2(fz[i], 0.f);
        sum[4] = ff_sums<R>(x, lane);
    }
    if (write) {
        #pragma unroll
        for (int q = 0; q < 5; ++q) { buf.part[q][slot] = sum[q]; buf.part[5 + q][slot] = old[q]; }
        buf.id[slot] = __float_as_int(trial[mine].w);
        buf.slice[slot] = slice;
    }
    __syncwarp();
}

// the beads' first runs, or (kRuns) the others
template <bool kRuns>
__global__ void __launch_bounds__(kTrialWarps * 32, 5)
k_trials32(PathView v, AzizF az, BoxF B, const int2* __restrict__ beads, const int* __restrict__ count,
           const int* __restrict__ cursor, const int* __restrict__ offset, const float4* __restrict__ sorted,
           const float4* __restrict__ fall, int run, int shift, int mode, const Scales32 sc, double* __restrict__ out) {
    extern __shared__ float4 sp[];
    __shared__ TrialBuffer buffers[kTrialWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Ne = v.Ne;
    float4 *P = sp + (size_t)warp * 2 * Ne, *F = P + Ne;
    TrialBuffer& buf = buffers[warp];
    const bool need_v = (mode != PGB_ACTION_CORR);
    auto corr = [&](int s) {
        const double gf = s % 2 ? sc.gf[1] : sc.gf[0];
        return (mode == PGB_ACTION_CORR) ? (gf > kEPS) : (mode == PGB_ACTION_FULL) ? (shift == 1 && gf > kEPS) : false;
    };
    const bool even_c = corr(0), odd_c = corr(1);
    int used = 0;
    auto flush = [&]() {
        if (lane < used) {
            const int s = buf.slice[lane];
            const double bare = s % 2 ? sc.bare[1] : sc.bare[0], cor = s % 2 ? sc.cor[1] : sc.cor[0];
            const bool need_c = s % 2 ? odd_c : even_c;
            auto dd = [&](int q) { const float2 x = buf.part[q][lane]; return (double)x.x + (double)x.y; };
            auto action = [&](double V, double T, double fx, double fy, double fz) {
                return assemble32(mode, need_c, bare, cor, V, T, fx, fy, fz);
            };
            double res;
            if (need_c) {
                res = action(need_v ? dd(0) : 0.0, dd(1), dd(2), dd(3), dd(4));
                res = __dsub_rn(res, action(need_v ? dd(5) : 0.0, dd(6), dd(7), dd(8), dd(9)));
            } else {
                res = action(need_v ? dd(0) : 0.0, 0.0, 0.0, 0.0, 0.0);
                res = __dsub_rn(res, action(need_v ? dd(5) : 0.0, 0.0, 0.0, 0.0, 0.0));
            }
            out[buf.id[lane]] = res;
        }
        used = 0;
        __syncwarp();
    };
    if (kRuns && !cursor[1]) return;
    const size_t items = kRuns ? ((size_t)cursor[0] + run - 1) / run : (size_t)v.M * Ne;
    for (size_t b = (size_t)blockIdx.x * kTrialWarps + warp; b < items; b += (size_t)gridDim.x * kTrialWarps) {
        int s, p, n, first;
        if (kRuns) {
            const int place = (int)(b * run);
            const int2 bead = beads[__float_as_int(sorted[place].w)];
            s = bead.x; p = bead.y;
            const size_t at = (size_t)s * Ne + p;
            const int o = offset[at];
            first = o + (place - o + run - 1) / run * run;
            n = min(o + count[at] - first, run);
            if (first == o || n <= 0) continue;
        } else {
            // the even slices' beads, then the odd ones': an SM's warps run the
            // same loops, whose code does not fit the instruction cache together
            const int line = (int)(b / Ne), evens = (v.M + 1) / 2;
            p = (int)(b - (size_t)line * Ne);
            s = line < evens ? 2 * line : 2 * (line - evens) + 1;
            const size_t at = (size_t)s * Ne + p;
            n = min(count[at], run);
            if (n == 0) continue;
            first = offset[at];
        }
        const bool need_c = s % 2 ? odd_c : even_c;
        const float4* trial = sorted + first;
        // the current position, and the partners for the trials
        const float4* R = v.pos32 + (size_t)s * Ne;
        const float4* Fs = fall + (size_t)s * Ne;
        const float4 rpo = R[p];
        const int st1 = bead_state(v, s, p);
        KahanF vo, to;
        float fox = 0.f, foy = 0.f, foz = 0.f;
        for (int j = lane; j < Ne; j += 32) {
            if (j == p || !v.on[(size_t)s * Ne + j]) { P[j] = make_float4(0.f, 0.f, 0.f, -1.f); continue; }
            const float4 rj = R[j];
            const float fac = pair_factor32(st1, bead_state(v, s, j));
            const float ox = min_image32(rj.x - rpo.x, B.L0, B.I0);
            const float oy = min_image32(rj.y - rpo.y, B.L1, B.I1);
            const float oz = min_image32(rj.z - rpo.z, B.L2, B.I2);
            const float ro2 = fmaf(ox, ox, fmaf(oy, oy, oz * oz));
            if (need_v) vo.add(fac * aziz_v32(ro2, az));
            P[j] = make_float4(rj.x, rj.y, rj.z, fac);
            if (need_c) {
                const float go = aziz_g32(ro2, az);
                const float Fox = go * ox, Foy = go * oy, Foz = go * oz;
                const float4 fa = Fs[j];
                // F3: the slice force on j less the term of p at its current position
                const float F3x = fa.x - Fox, F3y = fa.y - Foy, F3z = fa.z - Foz;
                fox -= Fox; foy -= Foy; foz -= Foz;
                to.add(fmaf(2.0f, fmaf(Fox, F3x, fmaf(Foy, F3y, Foz * F3z)),
                            fmaf(Fox, Fox, fmaf(Foy, Foy, Foz * Foz))));
                F[j] = make_float4(F3x, F3y, F3z, 0.f);
            }
        }
        float2 old[5] = {};
        old[0] = warp_ff(vo);
        if (need_c) {
            old[1] = warp_ff(to);
            old[2] = ff_butterfly(fox, 0.f); old[3] = ff_butterfly(foy, 0.f); old[4] = ff_butterfly(foz, 0.f);
        }
        __syncwarp();
        for (int i = 0; i < n;) {
            const int left = n - i, take = left >= 3 ? min(left, 4) : left;
            if (used + take > 32) flush();
            if (take >= 3) {
                if (need_c) trial_group<4, true>(trial + i, take, P, F, Ne, B, az, need_v, lane, s, old, buf, used);
                else trial_group<4, false>(trial + i, take, P, F, Ne, B, az, need_v, lane, s, old, buf, used);
            } else {
                if (need_c) trial_group<2, true>(trial + i, take, P, F, Ne, B, az, need_v, lane, s, old, buf, used);
                else trial_group<2, false>(trial + i, take, P, F, Ne, B, az, need_v, lane, s, old, buf, used);
            }
            used += take;
            i += take;
        }
    }
    flush();
}

bool trials32_sorted(const PathView& v, int k) {
    return (double)k >= kTrialsPerBead * v.M * v.Ne && (double)k * v.Ne >= kTrialPairs &&
           (size_t)v.Ne * 2 * kTrialWarps * sizeof(float4) <= 160 * 1024;
}

cudaError_t launch_trials32(const PathView& v, AzizParams a, const int2* d_beads, int k, int shift, int mode, double tau,
                            double lambda, const double vf[2], const double gf[2], const double* d_pos,
                            const float4* d_force, int* d_count, float4* d_sorted, double* d_out, cudaStream_t s) {
    const size_t nb = (size_t)v.M * v.Ne, smem = (size_t)v.Ne * 2 * kTrialWarps * sizeof(float4);
    int *offset = d_count + nb + 2, *cursor = d_count + nb;
    cudaError_t e = set_smem_limit(k_trials32<false>, 160 * 1024);
    if (e == cudaSuccess) e = set_smem_limit(k_trials32<true>, 160 * 1024);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(d_count, 0, (nb + 2) * sizeof(int), s)) != cudaSuccess) return e;
    const int blocks = (k + 255) / 256;
    k_trial_count<<<blocks, 256, 0, s>>>(v, d_beads, k, d_count, d_out);
    const int run = std::max<int>(kTrialRun, (int)((2.0 * k / nb + 47.0) / 32.0) * 32);
    k_trial_offsets<<<v.M, 256, 0, s>>>(v, d_count, run, cursor, offset);
    k_trial_scatter<<<blocks, 256, 0, s>>>(v, d_beads, d_pos, k, offset, d_sorted, d_out);
    const BoxF B = box_f(v);
    // two beads a warp: the assembly's lanes half full, the CTAs short enough
    // to even out (eight beads a warp 1.05 ms, two 1.01)
    const size_t each = std::max<size_t>(1, std::min<size_t>(2, nb / (152 * 16)));
    const int grid = (int)((nb + kTrialWarps * each - 1) / (kTrialWarps * each));
    const AzizF az = make_aziz_f(a);
    const Scales32 sc = scales32(shift, tau, lambda, vf, gf);
    k_trials32<false><<<grid, kTrialWarps * 32, smem, s>>>(v, az, B, d_beads, d_count, cursor, offset, d_sorted, d_force, run,
                                                           shift, mode, sc, d_out);
    k_trials32<true><<<std::min(152 * 5, (k / run + kTrialWarps) / kTrialWarps), kTrialWarps * 32, smem, s>>>(
        v, az, B, d_beads, d_count, cursor, offset, d_sorted, d_force, run, shift, mode, sc, d_out);
    return cudaGetLastError();
}

// Same-slice forces of every active bead: F[t][b] = sum over active b3 != b
// of gradV(r_b - r_b3), FP32 with Kahan sums per component.  One CTA per
// slice, O(N^2).
constexpr int kForceBlock = 256;

__global__ void __launch_bounds__(kForceBlock)
k_slice_forces32(PathView v, AzizF az, float4* __restrict__ force) {
    extern __shared__ float4 sp[];
    const int s = blockIdx.x, Ne = v.Ne;
    const float L0 = (float)v.side[0], L1 = (float)v.side[1], L2 = (float)v.side[2];
    const float I0 = (float)v.sideInv[0], I1 = (float)v.sideInv[1], I2 = (float)v.sideInv[2];
    for (int j = threadIdx.x; j < Ne; j += blockDim.x) {
        float4 r = v.pos32[(size_t)s * Ne + j];
        r.w = v.on[(size_t)s * Ne + j] ? 1.f : 0.f;
        sp[j] = r;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < Ne; b += blockDim.x) {
        const float4 rb = sp[b];
        KahanF fx, fy, fz;
        if (rb.w != 0.f) {
            for (int b3 = 0; b3 < Ne; ++b3) {
                const float4 r3 = sp[b3];
                if (b3 == b || r3.w == 0.f) continue;
                const float ex = min_image32(rb.x - r3.x, L0, I0);
                const float ey = min_image32(rb.y - r3.y, L1, I1);
                const float ez = min_image32(rb.z - r3.z, L2, I2);
                const float g = aziz_g32(fmaf(ex, ex, fmaf(ey, ey, ez * ez)), az);
                fx.add(g * ex); fy.add(g * ey); fz.add(g * ez);
            }
        }
        force[(size_t)s * Ne + b] = make_float4(fx.s - fx.c, fy.s - fy.c, fz.s - fz.c, 0.f);
    }
}

cudaError_t launch_slice_forces32(const PathView& v, AzizParams a, float4* d_force, cudaStream_t s) {
    size_t smem = (size_t)v.Ne * sizeof(float4);
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    {
        const cudaError_t ae = set_smem_limit(k_slice_forces32, 200 * 1024);
        if (ae != cudaSuccess) return ae;
    }
    k_slice_forces32<<<v.M, kForceBlock, smem, s>>>(v, make_aziz_f(a), d_force);
    return cudaGetLastError();
}

// Mixed-precision per-slice estimator terms; same outputs, layout and levels
// as k_slice_terms64 (vint, g2, r1, r2, d1, d2, kin, xch).
//
// A bead's force and T matrix are FP32 sums over its partners in index order,
// one thread a bead.  Column c < 128 of a slice collects the beads c, c + 128,
// ... in Kahan sums, the potential of the pairs b2 > b1 and the beads' other
// terms; a Kahan sum depends on its order, so this one is kept whatever the
// launch.  64 beads a CTA, so that 250 slices of 256 beads give every
// sub-partition three warps instead of one and a half, with four pairs in
// flight; a column's potential stays with its first bead's thread, the beads'
// other terms go through memory to the last CTA of the slice.
//
// Bound: latency at this occupancy, then the issue rate (about 55 instructions
// a pair, 100 with the T matrix).  Energy and virial of 256 beads, 250 slices,
// GSF: 2 x 138 us with everything computed by 128 threads a slice, 162 us both
// here.
constexpr int kSliceRows32 = 64, kSliceColumns32 = 128;

// adds x to a Kahan sum where `take`, without a branch
__device__ __forceinline__ void kahan_add_if(KahanF& k, float x, bool take) {
    const float y = x - k.c, t = k.s + y, c = (t - k.s) - y;
    k.s = take ? t : k.s;
    k.c = take ? c : k.c;
}
// keeps the rounding of x: it is not merged into the addition it goes to
__device__ __forceinline__ float rounded(float x) { asm("" : "+f"(x)); return x; }

struct SliceRow32 {
    const PathView& v;
    const AzizF& az;
    const BoxF& B;
    const float4* sp;
    int s, n;
    bool worm;
    __device__ __forceinline__ float factor(int st1, int b2) const {
        return worm ? (float)pair_factor(st1, bead_state(v, s, b2)) : 1.0f;
    }
    __device__ __forceinline__ int state(int b1) const { return worm ? bead_state(v, s, b1) : 2; }
    // the potential of bead b1's pairs with the beads behind it
    __device__ __forceinline__ void potential(int b1, KahanF& vint) const {
        const float4 r1 = sp[b1];
        const int st1 = state(b1);
        #pragma unroll 4
        for (int b2 = b1 + 1; b2 < n; ++b2) {
            const float4 r2 = sp[b2];
            const float dx = min_image32(r1.x - r2.x, B.L0, B.I0);
            const float dy = min_image32(r1.y - r2.y, B.L1, B.I1);
            const float dz = min_image32(r1.z - r2.z, B.L2, B.I2);
            const float V = rounded(aziz_v32(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), az));
            vint.add(factor(st1, b2) * V);
        }
    }
    // bead b1's force and T matrix (xx xy xz yy yz zz) over all partners, and
    // for kV the potential of the pairs behind it
    template <bool kT, bool kV>
    __device__ __forceinline__ void forces(int b1, float (&F)[3], float (&T)[6], KahanF& vint) const {
        const float4 r1 = sp[b1];
        const int st1 = state(b1);
        float Fx = 0.f, Fy = 0.f, Fz = 0.f;
        float T00 = 0.f, T01 = 0.f, T02 = 0.f, T11 = 0.f, T12 = 0.f, T22 = 0.f;
        #pragma unroll 4
        for (int b2 = 0; b2 < n; ++b2) {
            // the bead itself: separation 0, force coefficient 0
            const bool self = b2 == b1;
            const float4 r2 = sp[b2];
            const float dx = min_image32(r1.x - r2.x, B.L0, B.I0);
            const float dy = min_image32(r1.y - r2.y, B.L1, B.I1);
            const float dz = min_image32(r1.z - r2.z, B.L2, B.I2);
            const float rr = self ? 1.0f : fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            float V, g;
            aziz_vg32(rr, az, V, g);
            g = self ? 0.0f : g;
            Fx = fmaf(g, dx, Fx); Fy = fmaf(g, dy, Fy); Fz = fmaf(g, dz, Fz);
            if (kV) kahan_add_if(vint, factor(st1, b2) * rounded(V), b2 > b1);
            if (kT) {
                // T-matrix: (d2V/r^2 - |dV|/r^3) r r^T + |dV|/r I
                const float rinv = rsqrtf(rr);
                const float dV = fabsf(g) * rr * rinv;
                const float d2V = aziz_d2v32(rr, az);
                const float c1 = (d2V - dV * rinv) * rinv * rinv;
                const float c0 = dV * rinv;
                T00 = fmaf(c1, dx * dx, T00 + c0); T11 = fmaf(c1, dy * dy, T11 + c0);
                T22 = fmaf(c1, dz * dz, T22 + c0);
                T01 = fmaf(c1, dx * dy, T01); T02 = fmaf(c1, dx * dz, T02); T12 = fmaf(c1, dy * dz, T12);
            }
        }
        F[0] = Fx; F[1] = Fy; F[2] = Fz;
        T[0] = T00; T[1] = T01; T[2] = T02; T[3] = T11; T[4] = T12; T[5] = T22;
    }
};

// 8 values a lane summed over the warp by recursive halving, in warp_sum's own
// tree (9 FP64 adds instead of 40): lane l returns the sum of value l / 4
__device__ __forceinline__ double warp_sum8(double (&x)[8], int lane) {
    #pragma unroll
    for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
        #pragma unroll
        for (int i = 0; i < h; ++i) {
            const double give = up ? x[i] : x[i + h];
            x[i] = (up ? x[i + h] : x[i]) + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
    return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// work: [M][9][Ne] floats, the beads' terms 1..7 and the columns' potential as
// Kahan pairs in 0 and 8
__global__ void __launch_bounds__(kSliceRows32)
k_slice_terms32(PathView v, AzizF az, BoxF B, int window, int even, int odd, unsigned* __restrict__ arrived,
                float* __restrict__ work, double* __restrict__ terms) {
    extern __shared__ float4 sp[];
    __shared__ double sums[8][kSliceColumns32 / 32];
    __shared__ bool last;
    const int s = blockIdx.x, Ne = v.Ne, n = v.nbs[s], nblk = gridDim.y, tid = threadIdx.x;
    const int level = s % 2 ? odd : even, b1 = blockIdx.y * kSliceRows32 + tid;
    if (level > kSliceNone) {
        for (int j = tid; j < n; j += kSliceRows32) sp[j] = v.pos32[(size_t)s * Ne + j];
        __syncthreads();
    }
    const SliceRow32 row{v, az, B, sp, s, n,
                         s == v.worm[0] || s == v.worm[2] || s == v.worm[4] || s == v.worm[6]};
    float* W = work + (size_t)s * 9 * Ne;
    if (b1 < n) {
        const float4 r1 = v.pos32[(size_t)s * Ne + b1];
        const bool column = b1 < kSliceColumns32;
        float val[8] = {};
        KahanF vint;
        if (level == kSliceV && column) row.potential(b1, vint);
        else if (level >= kSliceF) {
            float F[3], T[6];
            if (level == kSliceT) {
                if (blockIdx.y < 2) row.forces<true, true>(b1, F, T, vint);
                else row.forces<true, false>(b1, F, T, vint);
            } else {
                if (blockIdx.y < 2) row.forces<false, true>(b1, F, T, vint);
                else row.forces<false, false>(b1, F, T, vint);
            }
            const float Fx = F[0], Fy = F[1], Fz = F[2];
            val[1] = fmaf(Fx, Fx, fmaf(Fy, Fy, Fz * Fz));
            if (window > 0) {
                val[2] = fmaf(Fx, r1.x, fmaf(Fy, r1.y, Fz * r1.z));
                const float TFx = fmaf(T[0], Fx, fmaf(T[1], Fy, T[2] * Fz));
                const float TFy = fmaf(T[1], Fx, fmaf(T[3], Fy, T[4] * Fz));
                const float TFz = fmaf(T[2], Fx, fmaf(T[4], Fy, T[5] * Fz));
                val[3] = fmaf(TFx, r1.x, fmaf(TFy, r1.y, TFz * r1.z));
                float mx = 0, my = 0, mz = 0, lx = 0, ly = 0, lz = 0, cx = 0, cy = 0, cz = 0;
                int2 cn = make_int2(s, b1), cp = cn;
                float4 pn = r1, pp = r1;
                for (int gm = 0; gm < window; ++gm) {
                    if (gm > 0) {
                        if (cn.x >= 0) cn = v.next[(size_t)cn.x * Ne + cn.y];
                        if (cp.x >= 0) cp = v.prev[(size_t)cp.x * Ne + cp.y];
                    }
                    // an open end stops the walk, and stands for the neighbours behind it
                    const float4 qn = cn.x >= 0 ? v.pos32[(size_t)cn.x * Ne + cn.y] : pn;
                    const float4 qp = cp.x >= 0 ? v.pos32[(size_t)cp.x * Ne + cp.y] : pp;
                    mx += min_image32(qn.x - pn.x, B.L0, B.I0); my += min_image32(qn.y - pn.y, B.L1, B.I1);
                    mz += min_image32(qn.z - pn.z, B.L2, B.I2);
                    lx += min_image32(qp.x - pp.x, B.L0, B.I0); ly += min_image32(qp.y - pp.y, B.L1, B.I1);
                    lz += min_image32(qp.z - pp.z, B.L2, B.I2);
                    cx += (r1.x + mx) + (r1.x + lx); cy += (r1.y + my) + (r1.y + ly);
                    cz += (r1.z + mz) + (r1.z + lz);
                    pn = qn; pp = qp;
                }
                float den = 1.0f / (2.0f * window);
                float dlx = min_image32(r1.x - cx * den, B.L0, B.I0);
                float dly = min_image32(r1.y - cy * den, B.L1, B.I1);
                float dlz = min_image32(r1.z - cz * den, B.L2, B.I2);
                val[4] = fmaf(Fx, dlx, fmaf(Fy, dly, Fz * dlz));
                val[5] = fmaf(TFx, dlx, fmaf(TFy, dly, TFz * dlz));
                float v1x = 0, v1y = 0, v1z = 0;
                int2 c2 = make_int2(s, b1);
                float4 po = r1;
                float v2x = 0, v2y = 0, v2z = 0;
                for (int gm = 1; gm <= window; ++gm) {
                    c2 = v.next[(size_t)c2.x * Ne + c2.y];
                    if (c2.x < 0) break;
                    float4 q = v.pos32[(size_t)c2.x * Ne + c2.y];
                    const float ex = min_image32(q.x - po.x, B.L0, B.I0), ey = min_image32(q.y - po.y, B.L1, B.I1);
                    const float ez = min_image32(q.z - po.z, B.L2, B.I2);
                    v1x += ex; v1y += ey; v1z += ez;
                    if (gm == 1) { v2x = ex; v2y = ey; v2z = ez; }
                    po = q;
                }
                val[7] = fmaf(v1x, v2x, fmaf(v1y, v2y, v1z * v2z));
            }
        }
        int2 nx = v.next[(size_t)s * Ne + b1];
        if (!(nx.x == kXXX && nx.y == kXXX)) {
            float4 q = v.pos32[(size_t)nx.x * Ne + nx.y];
            float ax = min_image32(q.x - r1.x, B.L0, B.I0), ay = min_image32(q.y - r1.y, B.L1, B.I1);
            float az_ = min_image32(q.z - r1.z, B.L2, B.I2);
            val[6] = fmaf(ax, ax, fmaf(ay, ay, az_ * az_));
        }
        if (column && level > kSliceNone)
            for (int b = b1 + kSliceColumns32; b < n; b += kSliceColumns32) row.potential(b, vint);
        #pragma unroll
        for (int q = 1; q < 8; ++q) W[(size_t)q * Ne + b1] = val[q];
        if (column) { W[b1] = vint.s; W[(size_t)8 * Ne + b1] = vint.c; }
        __threadfence();
    }
    __syncthreads();
    if (nblk > 1) {
        if (tid == 0) last = atomicInc(arrived + s, nblk - 1) == nblk - 1;      // back to 0 for the next call
        __syncthreads();
        if (!last) return;
        __threadfence();
    }
    // the columns' sums widened to FP64 and added over the warps' 32 columns,
    // then the four groups of columns in order
    const int lane = tid & 31;
    for (int g = tid >> 5; g < kSliceColumns32 / 32; g += kSliceRows32 / 32) {
        const int c = 32 * g + lane;
        double x[8];
        #pragma unroll
        for (int q = 0; q < 8; ++q) {
            KahanF k;
            if (q == 0) {
                if (c < n) { k.s = __ldcg(W + c); k.c = __ldcg(W + (size_t)8 * Ne + c); }
            } else
                for (int b = c; b < n; b += kSliceColumns32) k.add(__ldcg(W + (size_t)q * Ne + b));
            x[q] = k.value();
        }
        const double t = warp_sum8(x, lane);
        if ((lane & 3) == 0) sums[lane >> 2][g] = t;
    }
    __syncthreads();
    if (tid < 8) terms[(size_t)tid * v.M + s] = sums[tid][0] + sums[tid][1] + sums[tid][2] + sums[tid][3];
}

static int slice_blocks32(int Ne) { return (Ne + kSliceRows32 - 1) / kSliceRows32; }

size_t slice_terms32_work(const PathView& v) { return (size_t)9 * v.M * v.Ne * sizeof(float); }

cudaError_t launch_slice_terms32(const PathView& v, AzizParams a, int window, int even, int odd, unsigned* d_arrived,
                                 void* d_work, double* d_terms, cudaStream_t s) {
    size_t smem = (size_t)v.Ne * sizeof(float4);
    {
        const cudaError_t ae = set_smem_limit(k_slice_terms32, 200 * 1024);
        if (ae != cudaSuccess) return ae;
    }
    k_slice_terms32<<<dim3(v.M, slice_blocks32(v.Ne)), kSliceRows32, smem, s>>>(
        v, make_aziz_f(a), box_f(v), window, even, odd, d_arrived, static_cast<float*>(d_work), d_terms);
    return cudaGetLastError();
}

}  // namespace pgb
