// scatter.cu -- rho_q(t) in FP32 and the CUDA-core S(q) / F(q,tau) kernels.
//
// S(q) and F(q,tau) of the reference (estimator.cpp:3705-3737, 3923-3961 and
// gpu_ssf/gpu_isf, estimator_gpu.cu:67-165, 288-380) are pair sums over beads;
// both equal correlations of the collective density
//     rho_q(t) = sum_j exp(i q . r_j(t)):
//     S(q)     = 1/(N M) sum_t |rho_q(t)|^2
//     F(q,tau) = 1/(N M) sum_t Re[rho_q(t) conj(rho_q(t+tau))]
// which turns O(Q M N^2) (S) and O(Q M^2 N^2) (F) into O(Q M N) + O(Q M^2).
#include <algorithm>

#include "isf_tc.cuh"

namespace pgb {

// One CTA = one slice t x 256 q-vectors; each thread owns one q and streams
// the slice's beads from shared memory (broadcast reads).  q . r / 2pi =
// sum_d n_d u_d with n_d = q_d L_d / 2pi and u_d = r_d / L_d.  Lattice q
// (integer n_d) use the fixed-point phase (rho_partial_lattice: three integer
// multiply-adds, no rounding); others the FP32 turn reduction (rho_partial).
// Either way __sincosf sees |angle| <= pi and the special-function pipe does
// only the sine and cosine.
constexpr int kRhoBlock = 256;

// Once per call, in one launch: the beads of every slice as fractions of the
// box, FP32 turns for general q and 32-bit fixed-point turns for lattice q (the
// FP64 conversion runs once per bead instead of once per (bead, q block)), and
// each wave vector in turns per box side, n_d = q_d L_d / 2 pi: FP32 turns with
// a lattice flag in w, and the integers of lattice vectors (the reference's q
// lists of lattice type) for the exact fixed-point phase.  The first blocks
// take the wave vectors; `beads` is 0 where the masked form makes the bead
// fractions.
__global__ void k_rho_setup(PathView v, const double* __restrict__ q, int nq, int qblocks, size_t beads,
                            float4* __restrict__ uf, int4* __restrict__ ui, float4* __restrict__ qf,
                            int4* __restrict__ qi, int* __restrict__ err) {
    if ((int)blockIdx.x < qblocks) {
        const int iq = blockIdx.x * blockDim.x + threadIdx.x;
        if (err && iq == 0) *err = 0;
        if (iq >= nq) return;
        const double inv2pi = 0.15915494309189533577;
        const double dx = q[3*iq] * v.side[0] * inv2pi, dy = q[3*iq+1] * v.side[1] * inv2pi,
                     dz = q[3*iq+2] * v.side[2] * inv2pi;
        const double rx = rint(dx), ry = rint(dy), rz = rint(dz);
        const bool lattice = fabs(dx - rx) < 1e-6 && fabs(dy - ry) < 1e-6 && fabs(dz - rz) < 1e-6 &&
                             fabs(rx) < 1048576.0 && fabs(ry) < 1048576.0 && fabs(rz) < 1048576.0;
        qf[iq] = make_float4((float)dx, (float)dy, (float)dz, lattice ? 1.f : 0.f);
        qi[iq] = make_int4(lattice ? (int)rx : 0, lattice ? (int)ry : 0, lattice ? (int)rz : 0, 0);
        return;
    }
    const size_t stride = (size_t)(gridDim.x - qblocks) * blockDim.x;
    for (size_t idx = (size_t)(blockIdx.x - qblocks) * blockDim.x + threadIdx.x; idx < beads; idx += stride) {
        const size_t t = idx / v.Ne, j = idx - t * v.Ne;
        const double* X = v.pos + t * 3 * v.Ne;
        const double ux = X[j] * v.sideInv[0], uy = X[v.Ne + j] * v.sideInv[1],
                     uz = X[2 * v.Ne + j] * v.sideInv[2];
        uf[idx] = make_float4((float)ux, (float)uy, (float)uz, 0.f);
        ui[idx] = make_int4(fixed_turns(ux), fixed_turns(uy), fixed_turns(uz), 0);
    }
}

// The same conversion restricted to the beads inside a cylinder about the z
// axis, x^2 + y^2 < maxR^2 (include(), estimator.cpp:4309-4311), packed to
// the front of each slice in bead order so that the sums keep one order.
// One CTA per slice; cnt[t] receives the slice's count.
constexpr int kMaskBlock = 256;

__global__ void __launch_bounds__(kMaskBlock)
k_rho_positions_masked(PathView v, double maxR2, float4* __restrict__ uf, int4* __restrict__ ui,
                       int* __restrict__ cnt) {
    __shared__ int warp_base[kMaskBlock / 32 + 1];
    const int t = blockIdx.x;
    const int n = v.nbs[t];
    const double* X = v.pos + (size_t)t * 3 * v.Ne;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int j0 = 0; j0 < n; j0 += kMaskBlock) {
        const int j = j0 + threadIdx.x;
        bool in = false;
        double x = 0.0, y = 0.0, z = 0.0;
        if (j < n) {
            x = X[j]; y = X[v.Ne + j]; z = X[2 * v.Ne + j];
            in = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)) < maxR2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (lane == 0) warp_base[warp] = __popc(bal);
        __syncthreads();
        if (threadIdx.x == 0) {
            int s = 0;
            for (int w = 0; w < kMaskBlock / 32; ++w) { const int c = warp_base[w]; warp_base[w] = s; s += c; }
            warp_base[kMaskBlock / 32] = s;
        }
        __syncthreads();
        if (in) {
            const size_t o = (size_t)t * v.Ne + base + warp_base[warp] + __popc(bal & ((1u << lane) - 1u));
            const double ux = x * v.sideInv[0], uy = y * v.sideInv[1], uz = z * v.sideInv[2];
            uf[o] = make_float4((float)ux, (float)uy, (float)uz, 0.f);
            ui[o] = make_int4(fixed_turns(ux), fixed_turns(uy), fixed_turns(uz), 0);
        }
        base += warp_base[kMaskBlock / 32];
        __syncthreads();
    }
    if (threadIdx.x == 0) cnt[t] = base;
}

template <bool kSplit>
__global__ void __launch_bounds__(kRhoBlock)
k_rhoq32(PathView v, const float4* __restrict__ uf, const int4* __restrict__ ui,
         const int* __restrict__ cnt, const float4* __restrict__ qf, const int4* __restrict__ qi,
         int nq, float2* __restrict__ rho, IsfOperand split) {
    extern __shared__ float4 su[];
    int4* si = reinterpret_cast<int4*>(su + v.Ne);
    const int t = blockIdx.y;
    const int n = cnt ? cnt[t] : v.nbs[t];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        su[j] = uf[(size_t)t * v.Ne + j];
        si[j] = ui[(size_t)t * v.Ne + j];
    }
    __syncthreads();
    const int iq = blockIdx.x * kRhoBlock + threadIdx.x;
    if (iq >= (kSplit ? split.qpad : nq)) return;
    float2 r = make_float2(0.f, 0.f);
    if (!kSplit || iq < nq) {
        // lattice wave vectors take the exact fixed-point phase, any other q the
        // FP32 turn reduction
        const float4 f = qf[iq];
        if (f.w != 0.f) {
            const int4 k = qi[iq];
            r = rho_partial_lattice(si, n, k.x, k.y, k.z);
        } else {
            r = rho_partial(su, n, f.x, f.y, f.z);
        }
    }
    if (kSplit) {
        // (Re rho | Im rho) of row iq, zero rows beyond nq; the two-byte stores
        // hide behind the sines of the other warps
        const size_t a = tiled_index(iq, t, 2 * v.M, kTM), b = tiled_index(iq, v.M + t, 2 * v.M, kTM);
        split_bf16(r.x, split.hi[a], split.lo[a]);
        split_bf16(r.y, split.hi[b], split.lo[b]);
    } else {
        rho[(size_t)iq * v.M + t] = r;
    }
}

namespace {
struct RhoWork { size_t ui, cnt, qf, qi, total; };
RhoWork rho_work(const PathView& v, int nq) {
    const size_t nb = (size_t)v.M * v.Ne;
    RhoWork w;
    w.ui = nb * sizeof(float4);
    w.qf = w.ui + nb * sizeof(int4);
    w.qi = w.qf + (size_t)nq * sizeof(float4);
    w.cnt = w.qi + (size_t)nq * sizeof(int4);
    w.total = w.cnt + (size_t)v.M * sizeof(int);
    return w;
}
}  // namespace

size_t rhoq32_work_bytes(const PathView& v, int nq) { return rho_work(v, nq).total; }

cudaError_t launch_rhoq32(const PathView& v, const double* d_q, int nq, float2* d_rho,
                          void* d_work, cudaStream_t s, double maxR2, const IsfOperand* split) {
    if (nq <= 0) return cudaSuccess;
    size_t smem = (size_t)v.Ne * (sizeof(float4) + sizeof(int4));
    if (smem > 200 * 1024) return cudaErrorInvalidValue;   // one slice must fit in shared memory
    {
        const cudaError_t ae = split ? set_smem_limit(k_rhoq32<true>, 200 * 1024) : set_smem_limit(k_rhoq32<false>, 200 * 1024);
        if (ae != cudaSuccess) return ae;
    }
    const RhoWork w = rho_work(v, nq);
    char* base = static_cast<char*>(d_work);
    float4* uf = reinterpret_cast<float4*>(base);
    int4* ui = reinterpret_cast<int4*>(base + w.ui);
    float4* qf = reinterpret_cast<float4*>(base + w.qf);
    int4* qi = reinterpret_cast<int4*>(base + w.qi);
    int* cnt = nullptr;
    size_t nb = (size_t)v.M * v.Ne;
    if (maxR2 > 0.0) {
        cnt = reinterpret_cast<int*>(base + w.cnt);
        k_rho_positions_masked<<<v.M, kMaskBlock, 0, s>>>(v, maxR2, uf, ui, cnt);
        nb = 0;
    }
    const int qblocks = (nq + 255) / 256;
    const int blocks = qblocks + (int)std::min<size_t>((nb + 255) / 256, 152 * 16);
    k_rho_setup<<<blocks, 256, 0, s>>>(v, d_q, nq, qblocks, nb, uf, ui, qf, qi, split ? split->err : nullptr);
    const int rows = split ? split->qpad : nq;
    dim3 grid((rows + kRhoBlock - 1) / kRhoBlock, v.M);
    if (split) k_rhoq32<true><<<grid, kRhoBlock, smem, s>>>(v, uf, ui, cnt, qf, qi, nq, nullptr, *split);
    else k_rhoq32<false><<<grid, kRhoBlock, smem, s>>>(v, uf, ui, cnt, qf, qi, nq, d_rho, IsfOperand{});
    return cudaGetLastError();
}

// S(q) = norm sum_t |rho_q(t)|^2: four FP64 instructions a density, the FP64
// pipe the bound, so one warp a wave vector and one reduction a vector instead
// of eight (2048 vectors, M = 512: 26 -> 13 us); but a CTA a vector for fewer
// than kSsfFew, where a warp's own chain is the time.  S(q) in the first form
// and the second, us: M = 1000, 1 vector 19.1 and 15.0, 150 23.1 and 18.1, 300
// 26.2 and 22.2, 608 28.1 and 28.1, 1579 47 and 55; M = 124, 150 17.1 and 15.0,
// 300 17.9 both, 608 20.2 and 22.1.
constexpr int kSsfBlock = 128, kSsfFew = 300;

__global__ void __launch_bounds__(kSsfBlock)
k_ssf_from_rho32(const float2* __restrict__ rho, int nq, int M, double norm, double* __restrict__ out) {
    const int iq = blockIdx.x * (kSsfBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (iq >= nq) return;
    double re = 0.0, im = 0.0;
    #pragma unroll 4
    for (int t = lane; t < M; t += 32) {
        const float2 r = rho[(size_t)iq * M + t];
        const double x = r.x, y = r.y;
        re = __fma_rn(x, x, re);
        im = __fma_rn(y, y, im);
    }
    const double s = warp_sum(re + im);
    if (lane == 0) out[iq] = s * norm;
}

__global__ void __launch_bounds__(256)
k_ssf_from_rho32_few(const float2* __restrict__ rho, int M, double norm, double* __restrict__ out) {
    __shared__ double red[8];
    double acc = 0.0;
    for (int t = threadIdx.x; t < M; t += 256) {
        const float2 r = rho[(size_t)blockIdx.x * M + t];
        const double x = r.x, y = r.y;
        acc = __fma_rn(x, x, __fma_rn(y, y, acc));
    }
    const double s = block_sum(acc, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s * norm;
}

cudaError_t launch_ssf_from_rho32(const float2* d_rho, int nq, int M, double norm,
                                  double* d_out, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    constexpr int each = kSsfBlock / 32;
    if (nq < kSsfFew) k_ssf_from_rho32_few<<<nq, 256, 0, s>>>(d_rho, M, norm, d_out);
    else k_ssf_from_rho32<<<(nq + each - 1) / each, kSsfBlock, 0, s>>>(d_rho, nq, M, norm, d_out);
    return cudaGetLastError();
}

// CUDA-core circular correlation: each thread owns kTauPerThread consecutive
// tau of one wave vector and slides a register window along t, one new shared
// load and one broadcast for kTauPerThread complex multiply-adds; sums of 64
// terms in FP32, those in FP64.  Several vectors share a CTA, so that its
// lanes are full (a vector needs (M/2 + 1)/8 threads); their densities are
// repeated beyond M for the window, with one entry of padding in eight, so
// that the threads' windows, eight entries apart, fall into different banks.
// 1579 vectors, M = 250: 36 us with one vector a CTA, a modulo a step and the
// windows in four banks, 25 us here; 341 vectors, M = 4, whole calls 50 us, 83
// with 128 vectors a CTA copied one after another, 35 here.
constexpr int kTauPerThread = 8;
constexpr int kIsfBlock = 128;

__host__ __device__ __forceinline__ int isf_pad(int i) { return i + (i >> 3); }
// float2 entries a vector takes: M + the last window's end, padded
__host__ __device__ __forceinline__ int isf_row(int M) { return isf_pad(M + M / 2 + 1 + 2 * kTauPerThread) + 1; }

__global__ void __launch_bounds__(kIsfBlock)
k_isf_direct32(const float2* __restrict__ rho, int nq, int M, int each, int per, double norm,
               double* __restrict__ out) {
    extern __shared__ float2 sr[];
    const int nt = M / 2 + 1, row = isf_row(M), ext = M + nt + 2 * kTauPerThread;
    const int q0 = blockIdx.x * each, qn = min(each, nq - q0);
    for (int x = threadIdx.x; x < qn * ext; x += kIsfBlock) {
        const int q = x / ext, t = x - q * ext;
        sr[q * row + isf_pad(t)] = rho[(size_t)(q0 + q) * M + t % M];
    }
    __syncthreads();
    for (int w = threadIdx.x; w < qn * per; w += kIsfBlock) {
        const int q = w / per, tau0 = (w - q * per) * kTauPerThread;
        const float2* S = sr + q * row;
        double acc[kTauPerThread];
        float2 win[kTauPerThread];
        #pragma unroll
        for (int k = 0; k < kTauPerThread; ++k) { acc[k] = 0.0; win[k] = S[isf_pad(tau0 + k)]; }
        for (int t0 = 0; t0 < M; t0 += 64) {
            float c[kTauPerThread];
            #pragma unroll
            for (int k = 0; k < kTauPerThread; ++k) c[k] = 0.f;
            const int tend = min(M, t0 + 64);
            int t = t0;
            for (; t + kTauPerThread <= tend; t += kTauPerThread) {
                // at step u the window's entry of tau0 + k is win[(u + k) % 8]
                const float2* A = S + isf_pad(t);
                const float2* N = S + isf_pad(t + tau0 + kTauPerThread);
                #pragma unroll
                for (int u = 0; u < kTauPerThread; ++u) {
                    const float2 a = A[u];
                    #pragma unroll
                    for (int k = 0; k < kTauPerThread; ++k) {
                        const float2 b = win[(u + k) % kTauPerThread];
                        c[k] = fmaf(a.x, b.x, fmaf(a.y, b.y, c[k]));
                    }
                    win[u] = N[u];
                }
            }
            for (; t < tend; ++t) {                                  // the last M % 8
                const float2 a = S[isf_pad(t)];
                #pragma unroll
                for (int k = 0; k < kTauPerThread; ++k) c[k] = fmaf(a.x, win[k].x, fmaf(a.y, win[k].y, c[k]));
                #pragma unroll
                for (int k = 0; k < kTauPerThread - 1; ++k) win[k] = win[k + 1];
                win[kTauPerThread - 1] = S[isf_pad(t + tau0 + kTauPerThread)];
            }
            #pragma unroll
            for (int k = 0; k < kTauPerThread; ++k) acc[k] += c[k];
        }
        #pragma unroll
        for (int k = 0; k < kTauPerThread; ++k)
            if (tau0 + k < nt) out[(size_t)(q0 + q) * nt + tau0 + k] = acc[k] * norm;
    }
}

// the same from memory, for M whose densities do not fit in shared memory with
// their repetition
__global__ void __launch_bounds__(256)
k_isf_long32(const float2* __restrict__ rho, int M, double norm, double* __restrict__ out) {
    extern __shared__ float2 sr[];
    const int iq = blockIdx.x;
    const int nt = M / 2 + 1;
    for (int t = threadIdx.x; t < M; t += blockDim.x) sr[t] = rho[(size_t)iq * M + t];
    __syncthreads();
    for (int tau = threadIdx.x; tau < nt; tau += blockDim.x) {
        double acc = 0.0;
        for (int t0 = 0; t0 < M; t0 += 64) {
            float c = 0.f;
            const int tend = min(M, t0 + 64);
            for (int t = t0; t < tend; ++t) {
                const float2 a = sr[t], b = sr[t + tau < M ? t + tau : t + tau - M];
                c = fmaf(a.x, b.x, fmaf(a.y, b.y, c));
            }
            acc += c;
        }
        out[(size_t)iq * nt + tau] = acc * norm;
    }
}

cudaError_t launch_isf_direct32(const float2* d_rho, int nq, int M, double norm, double* d_out,
                                cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    const int per = (M / 2 + 1 + kTauPerThread - 1) / kTauPerThread;
    const size_t row = (size_t)isf_row(M) * sizeof(float2);
    if (row <= 200 * 1024) {
        // no more vectors a CTA than leave every SM one
        const int most = std::min(std::max(1, kIsfBlock / per), (nq + 151) / 152);
        const int each = std::max<int>(1, std::min<size_t>(most, 200 * 1024 / row));
        const cudaError_t ae = set_smem_limit(k_isf_direct32, 200 * 1024);
        if (ae != cudaSuccess) return ae;
        k_isf_direct32<<<(nq + each - 1) / each, kIsfBlock, each * row, s>>>(d_rho, nq, M, each, per, norm, d_out);
        return cudaGetLastError();
    }
    const size_t smem = (size_t)M * sizeof(float2);
    if (smem > 200 * 1024) return cudaErrorInvalidValue;    // one q's densities in shared memory
    const cudaError_t ae = set_smem_limit(k_isf_long32, 200 * 1024);
    if (ae != cudaSuccess) return ae;
    k_isf_long32<<<nq, 256, smem, s>>>(d_rho, M, norm, d_out);
    return cudaGetLastError();
}

}  // namespace pgb
