// fp64_kernels.cu -- the FP64 "plain form" kernels.
//
// Compiled with -fmad=false: every multiply and add rounds once, in the order
// it is written, and fused operations are spelt out.  The tables, the direct
// pair form and the path arithmetic keep the reference's order; the fast pair
// form (pair64.cuh) rounds differently in the last bit or two, and totals
// differ through that and through summation order (parallel reductions).
#include <cooperative_groups.h>

#include "pair64.cuh"

namespace cg = cooperative_groups;

namespace pgb {

// ---------------------------------------------------------------------------
// Aziz functions for the tables (src/potential.cpp:1821-1907 and the F, dF,
// d2F helpers of include/potential.h:963-983).
// ---------------------------------------------------------------------------
struct AzizD {
    double rm, A, epsilon, alpha, beta, D, C6, C8, C10;
    __device__ double F(double x) const { return (x < D ? exp(-(D/x - 1.0)*(D/x - 1.0)) : 1.0); }
    __device__ double dF(double x) const {
        double ix = 1.0/x;
        double r = 2.0*D*ix*ix*(D*ix-1.0)*exp(-(D*ix - 1.0)*(D*ix - 1.0));
        return (x < D ? r : 0.0);
    }
    __device__ double d2F(double x) const {
        double ix = 1.0/x;
        double r = 2.0*D*ix*ix*ix*( 2.0*D*D*D*ix*ix*ix - 4.0*D*D*ix*ix
                - D*ix + 2.0) * exp(-(D*ix - 1.0)*(D*ix - 1.0));
        return (x < D ? r : 0.0);
    }
    __device__ double V(double r) const {
        double x = r / rm;
        double Urep = A * exp(-alpha*x + beta*x*x);
        if (x < kEPS) return 0.0;
        else if (x < 0.01) return (epsilon * Urep);
        double ix2 = 1.0 / (x * x);
        double ix6 = ix2 * ix2 * ix2;
        double ix8 = ix6 * ix2;
        double ix10 = ix8 * ix2;
        double Uatt = -( C6*ix6 + C8*ix8 + C10*ix10 ) * F(x);
        return ( epsilon * (Urep + Uatt) );
    }
    __device__ double dVdr(double r) const {
        double x = r / rm;
        double T1 = A * (-alpha + 2.0*beta*x) * exp(-alpha*x + beta*x*x);
        if (x < kEPS) return 0.0;
        else if (x < 0.01) return ( ( epsilon / rm ) * T1 );
        double ix = 1.0 / x;
        double ix2 = ix*ix;
        double ix6 = ix2 * ix2 * ix2;
        double ix7 = ix6 * ix;
        double ix8 = ix6 * ix2;
        double ix9 = ix8 * ix;
        double ix10 = ix8 * ix2;
        double ix11 = ix10 * ix;
        double T2 = ( 6.0*C6*ix7 + 8.0*C8*ix9 + 10.0*C10*ix11 ) * F(x);
        double T3 = -( C6*ix6 + C8*ix8 + C10*ix10 ) * dF(x);
        return ( ( epsilon / rm ) * (T1 + T2 + T3) );
    }
    __device__ double d2Vdr2(double r) const {
        double x = r / rm;
        double abFactor2 = (alpha - 2.0*beta*x)*(alpha-2.0*beta*x);
        double T1 = A * (2*beta + abFactor2) * exp(-alpha*x + beta*x*x);
        if (x < kEPS) return 0.0;
        else if (x < 0.01) return ( ( epsilon / rm ) * T1 );
        double ix = 1.0 / x;
        double ix2 = ix*ix;
        double ix6 = ix2 * ix2 * ix2;
        double ix7 = ix6 * ix;
        double ix8 = ix6 * ix2;
        double ix9 = ix8 * ix;
        double ix10 = ix8 * ix2;
        double ix11 = ix10 * ix;
        double ix12 = ix11 * ix;
        double T2 = - ( 42.0*C6*ix8 + 72.0*C8*ix10 + 110.0*C10*ix12 ) * F(x);
        double T3 = 2.0*( 6.0*C6*ix7 + 8.0*C8*ix9 + 10.0*C10*ix11 ) * dF(x);
        double T4 = - ( C6*ix6 + C8*ix8 + C10*ix10 ) * d2F(x);
        return ( ( epsilon / (rm*rm) ) * (T1 + T2 + T3 + T4) );
    }
};

__global__ void k_build_tables(const double* __restrict__ r, int n, AzizD az,
                               double* tV, double* tdV, double* td2V) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double x = r[i];
        tV[i] = az.V(x);
        tdV[i] = az.dVdr(x);
        td2V[i] = az.d2Vdr2(x);
    }
}

cudaError_t launch_build_tables(const double* d_r, int n, AzizParams a,
                                double* tV, double* tdV, double* td2V, cudaStream_t s) {
    AzizD az{a.rm, a.A, a.epsilon, a.alpha, a.beta, a.D, a.C6, a.C8, a.C10};
    int blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    k_build_tables<<<blocks, 256, 0, s>>>(d_r, n, az, tV, tdV, td2V);
    return cudaGetLastError();
}

// PotentialBase::V(const dVec*, double*, int) and gradV/grad2V, batched.
__global__ void k_potential_batch64(PathView v, const double* __restrict__ sep,
                                    double* out, int n, int what) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double3 d = make_double3(sep[3*i], sep[3*i+1], sep[3*i+2]);
        if (what == 0) out[i] = V64(v, d);
        else if (what == 1) { double3 g = gradV64(v, d); out[3*i] = g.x; out[3*i+1] = g.y; out[3*i+2] = g.z; }
        else out[i] = grad2V64(v, d);
    }
}

cudaError_t launch_potential_batch64(const PathView& v, const double* d_sep,
                                     double* d_out, int n, int what, cudaStream_t s) {
    int blocks = (n + 255) / 256;
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) blocks = 1;
    k_potential_batch64<<<blocks, 256, 0, s>>>(v, d_sep, d_out, n, what);
    return cudaGetLastError();
}

// Sums of Q per-thread values over the CTA: all to shared memory, then one
// warp a quantity, so that the twelve FP64 adds of a quantity run once and on
// all four sub-partitions instead of in every warp.
constexpr int kPairBlock = 256;

template <int Q>
__device__ __forceinline__ void block_sums(const double (&val)[Q], double (*buf)[kPairBlock], double* out) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    #pragma unroll
    for (int q = 0; q < Q; ++q) buf[q][tid] = val[q];
    __syncthreads();
    for (int q = warp; q < Q; q += kPairBlock / 32) {
        double s = buf[q][lane];
        #pragma unroll
        for (int i = 1; i < kPairBlock / 32; ++i) s += buf[q][lane + 32 * i];
        s = warp_sum(s);
        if (lane == 0) out[q] = s;
    }
    __syncthreads();
}

// what a bead's action is made of, and its assembly (action.cpp:487-740)
struct BeadSpec {
    int shift, mode;
    double tau, lambda, vf[2], gf[2];
    __device__ __forceinline__ bool need_v() const { return mode != PGB_ACTION_CORR; }
    __device__ __forceinline__ bool need_c(int s) const {
        return gf[s % 2] > kEPS && (mode == PGB_ACTION_CORR || (mode == PGB_ACTION_FULL && shift == 1));
    }
    __device__ __forceinline__ double action(int s, double V, double T, double fx, double fy, double fz) const {
        const double t = (double)shift * tau;
        const double bareU = vf[s % 2] * t * V;
        const double corU = need_c(s) ? gf[s % 2] * t * t * t * lambda * (T + (fx * fx + fy * fy + fz * fz)) : 0.0;
        return mode == PGB_ACTION_BARE ? bareU : mode == PGB_ACTION_CORR ? corU : bareU + corU;
    }
};

// True when a worm end lies on slice s, so that pair factors differ from 1
__device__ __forceinline__ bool worm_on_slice(const PathView& v, int s) {
    return s == v.worm[0] || s == v.worm[2] || s == v.worm[4] || s == v.worm[6];
}

// ---------------------------------------------------------------------------
// Per-bead potential action, a cluster of CTAs per bead.
//
// Phase 1 builds the LookupTable interaction list of the bead (every active
// bead of the same slice, other than itself, with |r2 - r1|^2 < rc^2;
// lookuptable.cpp:464-516), sums Vnn (action.cpp:1044-1060) and keeps each
// member's F2 = gradV(r2 - r1).  Phase 2 is gradVnnSquared
// (action.cpp:1282-1337), T = sum_n |F2_n|^2 + 2 F2_n . F3_n with
// F3_n = sum over the other members m of gradV(r_n - r_m).  gradV is odd, so
//     sum_n F2_n . F3_n = sum_{n<m} gradV(r_n - r_m) . (F2_n - F2_m):
// each pair of members once.  Pairs go to threads by offset around the list,
// (n, n + o mod size), o <= size / 2, so neighbouring lanes read neighbouring
// members; the cluster's CTAs take turns at them and the first one adds the
// shares through distributed shared memory.
//
// Bound: the FP64 pipe, about 27 instructions a pair, 16 clocks of an SM a
// warp instruction.  31 beads of a 64-particle GSF path (a bisection's range):
// 173 us with one thread a member and every ordered pair in the direct form,
// 15.6 us here; as trials 2 x 173 and 21.6 us.  kBoth evaluates the trial and
// the current position of the bead over one pass of the members' pairs, and
// writes the difference.
// ---------------------------------------------------------------------------
constexpr int kMaxCluster = 8;

// shared memory a list member takes
constexpr int bead_pairs_bytes(bool both) { return (both ? 9 : 6) * (int)sizeof(double) + 3 * (int)sizeof(float); }

template <bool kBoth>
__global__ void __launch_bounds__(kPairBlock)
k_bead_pairs64(PathView v, double invdr, const int2* __restrict__ beads, BeadSpec a, int csize,
               const double* __restrict__ over, double* __restrict__ out) {
    constexpr int Q = kBoth ? 10 : 5;
    extern __shared__ double smem[];
    const int Ne = v.Ne;
    double *lx = smem, *ly = lx + Ne, *lz = ly + Ne;                     // members' positions
    double *fx = lz + Ne, *fy = fx + Ne, *fz = fy + Ne;                  // F2 at the trial (or current) position
    double *gx = fz + Ne, *gy = gx + Ne, *gz = gy + Ne;                  // F2 at the current position (kBoth)
    float* ux = reinterpret_cast<float*>(kBoth ? gz + Ne : gx);          // box fractions
    float *uy = ux + Ne, *uz = uy + Ne;
    __shared__ double buf[Q][kPairBlock];
    __shared__ double sums[Q], cross[2], share[kMaxCluster][2];
    __shared__ int wcount[kPairBlock / 32];
    __shared__ int s_total;

    const int b = blockIdx.x / csize, rank = blockIdx.x - b * csize;
    const int s = beads[b].x, p = beads[b].y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (s < 0 || s >= v.M || p < 0 || p >= Ne || !v.on[(size_t)s * Ne + p]) {
        if (tid == 0 && rank == 0) out[b] = 0.0;
        return;                                  // the whole cluster
    }
    const bool need_v = a.need_v(), need_c = a.need_c(s);
    if (!need_c && rank > 0) return;             // no shares: no cluster barrier below

    const double* X = v.pos + (size_t)s * 3 * Ne;
    const float4* P = v.pos32 + (size_t)s * Ne;
    const float Ix = (float)v.sideInv[0], Iy = (float)v.sideInv[1], Iz = (float)v.sideInv[2];
    // `over` (trial positions) replaces the bead's stored position
    const double x1 = over ? over[3 * b] : X[p];
    const double y1 = over ? over[3 * b + 1] : X[Ne + p];
    const double z1 = over ? over[3 * b + 2] : X[2 * Ne + p];
    const float u1 = box_fraction((float)x1, Ix), u2 = box_fraction((float)y1, Iy), u3 = box_fraction((float)z1, Iz);
    double xo = 0.0, yo = 0.0, zo = 0.0;
    float o1 = 0.f, o2 = 0.f, o3 = 0.f;
    if (kBoth) {
        xo = X[p]; yo = X[Ne + p]; zo = X[2 * Ne + p];
        o1 = box_fraction((float)xo, Ix); o2 = box_fraction((float)yo, Iy); o3 = box_fraction((float)zo, Iz);
    }
    const bool worm = worm_on_slice(v, s);
    const int st1 = worm ? bead_state(v, s, p) : 2;
    if (tid == 0) s_total = 0;
    __syncthreads();

    // Vn Sn Fn(3) [Vo So Fo(3)]
    double val[Q] = {};
    for (int base = 0; base < Ne; base += kPairBlock) {
        const int j = base + tid;
        bool in = false;
        double xj = 0.0, yj = 0.0, zj = 0.0, ax = 0.0, ay = 0.0, az = 0.0, bx = 0.0, by = 0.0, bz = 0.0;
        float vx = 0.f, vy = 0.f, vz = 0.f;
        if (j < Ne && j != p && v.on[(size_t)s * Ne + j]) {
            xj = X[j]; yj = X[Ne + j]; zj = X[2 * Ne + j];
            const float4 f = P[j];
            vx = box_fraction(f.x, Ix); vy = box_fraction(f.y, Iy); vz = box_fraction(f.z, Iz);
            // LookupTable stores sep = getSeparation(bead2, bead1) = r2 - r1
            const Pair64 d = pair64(v, invdr, xj - x1, yj - y1, zj - z1, vx - u1, vy - u2, vz - u3);
            in = d.r2 < v.rc2;
            const double fac = worm ? pair_factor(st1, bead_state(v, s, j)) : 1.0;
            if (in) {
                if (need_v) val[0] += fac * table64(v.tV, d.k);
                if (need_c) {
                    const double g = table64(v.tdV, d.k) * d.y;
                    ax = g * d.dx; ay = g * d.dy; az = g * d.dz;
                    val[1] = __fma_rn(ax, ax, __fma_rn(ay, ay, __fma_rn(az, az, val[1])));
                    val[2] -= ax; val[3] -= ay; val[4] -= az;
                }
            }
            if (kBoth) {                         // whole lists: the same members, unless a position is not finite
                const Pair64 e = pair64(v, invdr, xj - xo, yj - yo, zj - zo, vx - o1, vy - o2, vz - o3);
                if (e.r2 < v.rc2) {
                    in = true;
                    if (need_v) val[Q - 5] += fac * table64(v.tV, e.k);
                    if (need_c) {
                        const double g = table64(v.tdV, e.k) * e.y;
                        bx = g * e.dx; by = g * e.dy; bz = g * e.dz;
                        val[Q - 4] = __fma_rn(bx, bx, __fma_rn(by, by, __fma_rn(bz, bz, val[Q - 4])));
                        val[Q - 3] -= bx; val[Q - 2] -= by; val[Q - 1] -= bz;
                    }
                }
            }
        }
        if (!need_c) continue;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) wcount[w] = __popc(m);
        __syncthreads();
        int off = s_total;
        for (int i = 0; i < w; ++i) off += wcount[i];
        if (in) {
            const int q = off + __popc(m & ((1u << lane) - 1u));
            lx[q] = xj; ly[q] = yj; lz[q] = zj;
            fx[q] = ax; fy[q] = ay; fz[q] = az;
            if (kBoth) { gx[q] = bx; gy[q] = by; gz[q] = bz; }
            ux[q] = vx; uy[q] = vy; uz[q] = vz;
        }
        __syncthreads();
        if (tid == 0) { int tot = 0; for (int i = 0; i < kPairBlock / 32; ++i) tot += wcount[i]; s_total += tot; }
        __syncthreads();
    }
    double tn = 0.0, to = 0.0;
    if (need_c) {
        // the first CTA's shared memory is written below: it has started by then
        if (csize > 1) cg::this_cluster().sync();
        const int n = s_total;
        double c[2] = {0.0, 0.0};
        if (n > 1) {
            const int half = (n - 1) / 2, total = n * half + (n % 2 ? 0 : n / 2);
            const int stride = csize * kPairBlock, so = stride / n, si = stride - so * n;
            int idx = rank * kPairBlock + tid;
            int o = idx / n, i = idx - o * n;
            ++o;
            for (; idx < total; idx += stride) {
                int j = i + o;
                if (j >= n) j -= n;
                const Pair64 d = pair64(v, invdr, lx[i] - lx[j], ly[i] - ly[j], lz[i] - lz[j], ux[i] - ux[j],
                                        uy[i] - uy[j], uz[i] - uz[j]);
                const double g = table64(v.tdV, d.k) * d.y;
                c[0] = __fma_rn(g, __fma_rn(d.dx, fx[i] - fx[j], __fma_rn(d.dy, fy[i] - fy[j], d.dz * (fz[i] - fz[j]))), c[0]);
                if (kBoth)
                    c[1] = __fma_rn(g, __fma_rn(d.dx, gx[i] - gx[j], __fma_rn(d.dy, gy[i] - gy[j], d.dz * (gz[i] - gz[j]))), c[1]);
                i += si; o += so;
                if (i >= n) { i -= n; ++o; }
            }
        }
        if (kBoth) block_sums<2>(c, buf, cross);
        else { const double c1[1] = {c[0]}; block_sums<1>(c1, buf, cross); }
        if (csize > 1) {
            cg::cluster_group cl = cg::this_cluster();
            if (tid < (kBoth ? 2 : 1)) cl.map_shared_rank(&share[0][0], 0)[2 * rank + tid] = cross[tid];
            cl.sync();
            if (rank > 0) return;
            for (int r = 0; r < csize; ++r) { tn += share[r][0]; if (kBoth) to += share[r][1]; }
        } else { tn = cross[0]; if (kBoth) to = cross[1]; }
    }
    block_sums<Q>(val, buf, sums);
    if (tid == 0) {
        double U = a.action(s, sums[0], sums[1] + 2.0 * tn, sums[2], sums[3], sums[4]);
        if (kBoth) U -= a.action(s, sums[Q - 5], sums[Q - 4] + 2.0 * to, sums[Q - 3], sums[Q - 2], sums[Q - 1]);
        out[b] = U;
    }
}

// Same-slice forces F_b = sum over active b3 != b of gradV(r_b - r_b3) of the
// slices whose action has a gradient term, [M][3][Ne].  One CTA per slice and
// block of kForceRows beads, four (eight) threads a bead over the partners.
constexpr int kForceRows = 64;

__global__ void __launch_bounds__(kPairBlock)
k_slice_forces64(PathView v, double invdr, int even, int odd, double* __restrict__ force) {
    extern __shared__ double smem[];
    const int s = blockIdx.x, Ne = v.Ne;
    if (!(s % 2 ? odd : even)) return;
    double *lx = smem, *ly = lx + Ne, *lz = ly + Ne;
    float *ux = reinterpret_cast<float*>(lz + Ne), *uy = ux + Ne, *uz = uy + Ne;
    __shared__ double acc[3][kPairBlock];
    const float Ix = (float)v.sideInv[0], Iy = (float)v.sideInv[1], Iz = (float)v.sideInv[2];
    for (int j = threadIdx.x; j < Ne; j += kPairBlock) {
        const double* X = v.pos + (size_t)s * 3 * Ne;
        const float4 f = v.pos32[(size_t)s * Ne + j];
        lx[j] = X[j]; ly[j] = X[Ne + j]; lz[j] = X[2 * Ne + j];
        ux[j] = box_fraction(f.x, Ix); uy[j] = box_fraction(f.y, Iy); uz[j] = box_fraction(f.z, Iz);
    }
    __syncthreads();
    const int b0 = blockIdx.y * kForceRows, nb = min(kForceRows, Ne - b0);
    const int rows = nb > 32 ? 64 : 32, parts = kPairBlock / rows;
    const int r = threadIdx.x & (rows - 1), part = threadIdx.x / rows, i = b0 + r;
    double Fx = 0.0, Fy = 0.0, Fz = 0.0;
    if (r < nb && v.on[(size_t)s * Ne + i]) {
        for (int j = part; j < Ne; j += parts) {
            if (j == i || !v.on[(size_t)s * Ne + j]) continue;
            const Pair64 d = pair64(v, invdr, lx[i] - lx[j], ly[i] - ly[j], lz[i] - lz[j], ux[i] - ux[j], uy[i] - uy[j],
                                    uz[i] - uz[j]);
            if (!(d.r2 < v.rc2)) continue;       // not finite: in no list
            const double g = table64(v.tdV, d.k) * d.y;
            Fx = __fma_rn(g, d.dx, Fx); Fy = __fma_rn(g, d.dy, Fy); Fz = __fma_rn(g, d.dz, Fz);
        }
    }
    acc[0][threadIdx.x] = Fx; acc[1][threadIdx.x] = Fy; acc[2][threadIdx.x] = Fz;
    __syncthreads();
    if (part < 3 && r < nb) {                    // one part a component
        double t = acc[part][r];
        for (int q = 1; q < parts; ++q) t += acc[part][r + q * rows];
        force[((size_t)s * 3 + part) * Ne + i] = t;
    }
}

// 16 values a lane summed over the warp by recursive halving (16 adds instead
// of 80): lane l returns the sum of value l / 2
__device__ __forceinline__ double warp_sum16(double (&x)[16], int lane) {
    #pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
        #pragma unroll
        for (int i = 0; i < h; ++i) {
            const double give = up ? x[i] : x[i + h];
            x[i] = (up ? x[i + h] : x[i]) + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// Many beads: one warp a bead, O(n) a bead, the inner sums of the gradient
// term from the slice forces, F3_n = F_n - gradV(r_n - r_p) with r_p the
// bead's stored position.  Needs lists that take in the whole slice.  Each
// warp takes kWarpBeads beads in turn; the assembly runs one bead a lane.
constexpr int kWarpBeads = 4;
constexpr int kBlockBeads = kWarpBeads * kPairBlock / 32;

template <bool kBoth>
__global__ void __launch_bounds__(kPairBlock)
k_bead_warp64(PathView v, double invdr, const int2* __restrict__ beads, int k, BeadSpec a,
              const double* __restrict__ over, const double* __restrict__ force, double* __restrict__ out) {
    __shared__ double part[kBlockBeads][11];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Ne = v.Ne;
    const float Ix = (float)v.sideInv[0], Iy = (float)v.sideInv[1], Iz = (float)v.sideInv[2];
    auto active = [&](int2 b) {
        return b.x >= 0 && b.x < v.M && b.y >= 0 && b.y < Ne && v.on[(size_t)b.x * Ne + b.y];
    };
    for (int r = 0; r < kWarpBeads; ++r) {
        const int lb = warp * kWarpBeads + r;
        const long long b = (long long)blockIdx.x * kBlockBeads + lb;
        if (b >= k) break;
        const int s = beads[b].x, p = beads[b].y;
        if (!active(beads[b])) continue;
        const bool need_v = a.need_v(), need_c = a.need_c(s);
        const double* X = v.pos + (size_t)s * 3 * Ne;
        const double* F = force + (size_t)s * 3 * Ne;
        const float4* P = v.pos32 + (size_t)s * Ne;
        const double xo = X[p], yo = X[Ne + p], zo = X[2 * Ne + p];
        const float o1 = box_fraction((float)xo, Ix), o2 = box_fraction((float)yo, Iy), o3 = box_fraction((float)zo, Iz);
        const double x1 = kBoth ? over[3 * b] : xo, y1 = kBoth ? over[3 * b + 1] : yo, z1 = kBoth ? over[3 * b + 2] : zo;
        const float u1 = box_fraction((float)x1, Ix), u2 = box_fraction((float)y1, Iy), u3 = box_fraction((float)z1, Iz);
        const bool worm = worm_on_slice(v, s);
        const int st1 = worm ? bead_state(v, s, p) : 2;
        double x[16] = {};                       // V T F(3) at the stored position, then at the trial one
        for (int j = lane; j < Ne; j += 32) {
            if (j == p || !v.on[(size_t)s * Ne + j]) continue;
            const double xj = X[j], yj = X[Ne + j], zj = X[2 * Ne + j];
            const float4 f = P[j];
            const float vx = box_fraction(f.x, Ix), vy = box_fraction(f.y, Iy), vz = box_fraction(f.z, Iz);
            const double fac = worm ? pair_factor(st1, bead_state(v, s, j)) : 1.0;
            const Pair64 e = pair64(v, invdr, xj - xo, yj - yo, zj - zo, vx - o1, vy - o2, vz - o3);
            Pair64 d = e;
            if (kBoth) d = pair64(v, invdr, xj - x1, yj - y1, zj - z1, vx - u1, vy - u2, vz - u3);
            const bool ine = e.r2 < v.rc2, ind = d.r2 < v.rc2;       // true unless a position is not finite
            if (need_v) {
                if (ine) x[0] += fac * table64(v.tV, e.k);
                if (kBoth && ind) x[5] += fac * table64(v.tV, d.k);
            }
            if (need_c) {
                double ex = 0.0, ey = 0.0, ez = 0.0;
                if (ine) {
                    const double g = table64(v.tdV, e.k) * e.y;
                    ex = g * e.dx; ey = g * e.dy; ez = g * e.dz;
                }
                // |F2|^2 + 2 F2.F3 = F2 . (F2 + 2 F3), F3 without the bead's own term
                const double hx = 2.0 * (F[j] - ex), hy = 2.0 * (F[Ne + j] - ey), hz = 2.0 * (F[2 * Ne + j] - ez);
                x[1] = __fma_rn(ex, ex + hx, __fma_rn(ey, ey + hy, __fma_rn(ez, ez + hz, x[1])));
                x[2] -= ex; x[3] -= ey; x[4] -= ez;
                if (kBoth && ind) {
                    const double g = table64(v.tdV, d.k) * d.y;
                    const double tx = g * d.dx, ty = g * d.dy, tz = g * d.dz;
                    x[6] = __fma_rn(tx, tx + hx, __fma_rn(ty, ty + hy, __fma_rn(tz, tz + hz, x[6])));
                    x[7] -= tx; x[8] -= ty; x[9] -= tz;
                }
            }
        }
        const double t = warp_sum16(x, lane);
        if (!(lane & 1) && lane < 20) part[lb][lane >> 1] = t;
    }
    __syncthreads();
    const long long b = (long long)blockIdx.x * kBlockBeads + lane;
    if (warp == 0 && b < k) {
        double U = 0.0;
        if (active(beads[b])) {
            const int s = beads[b].x;
            const double* q = part[lane];
            U = a.action(s, q[0], q[1], q[2], q[3], q[4]);
            if (kBoth) U = a.action(s, q[5], q[6], q[7], q[8], q[9]) - U;
        }
        out[b] = U;
    }
}

// From here on the warp form is the faster; below, it leaves warps idle.  Whole
// calls, clusters against warps, without a gradient term: 64 beads a slice, 1824
// beads 45 and 46 us, 2432 63 and 54 (128 beads a slice: 50 and 59, 63 and 68,
// 4864 105 and 79).  With one the warp form makes the forces of all slices
// first, M n^2 pairs on few CTAs while M is small, and a cluster n^2 / 2 pairs a
// bead, which fill the SMs from about 10^5 / n beads on.  GSF, whole calls, n
// beads a slice, M slices, clusters and warps in us:
//   n = 16   M = 62: 496 beads 31 and 44; M = 1000: 1000 42 and 56, 3000 79 and 66
//   n = 64   M = 62: 248 55 and 81, 496 89 and 82; M = 124: 372 72 and 81, 496 88
//            and 82; M = 500: 1500 139 and 165, 2000 174 and 166; M = 1000: 2000
//            173 and 166
//   n = 128  M = 124: 248 145 and 182, 372 206 and 182; M = 250: 1000 283 and 291,
//            1500 412 and 291; M = 500: 1000 285 and 292, 1500 411 and 292
//   n = 256  M = 62: 124 269 and 333, 186 503 and 334; M = 250: 250 505 and 549,
//            500 987 and 551
constexpr int kManyBeads = 2048;
static double many_gradient(const PathView& v) {
    const double n = v.Ne, slices = std::max(v.M * std::min(4.0, 640.0 / n), 2.5e4 / n);
    return std::min(std::min(2048.0, slices), std::min(1.24e5 / n, 1.8e7 / (n * n)));
}

template <bool kBoth>
static cudaError_t bead_pairs64(const PathView& v, const int2* d_beads, int k, const BeadSpec& a, bool corr,
                                const double* d_over, double* d_out, cudaStream_t s) {
    const size_t smem = (size_t)v.Ne * bead_pairs_bytes(kBoth);
    const cudaError_t ae = set_smem_limit(k_bead_pairs64<kBoth>, 200 * 1024);
    if (ae != cudaSuccess) return ae;
    int c = 1;
    if (corr)
        while (c < kMaxCluster && 2 * c * k <= 2 * 152) c *= 2;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)k * c);
    cfg.blockDim = dim3(kPairBlock);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = c > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_bead_pairs64<kBoth>, v, 1.0 / v.dr, d_beads, a, c, d_over, d_out);
}

// The same with the list alone in shared memory, every ordered pair of members
// in the direct form: for slices whose list and forces do not fit above.
constexpr int kBeadBlock = 256;

__global__ void __launch_bounds__(kBeadBlock)
k_bead_actions64(PathView v, const int2* __restrict__ beads, int k, int shift, int mode,
                 double tau, double lambda, double vf0, double vf1, double gf0,
                 double gf1, const double* __restrict__ over, double* __restrict__ out) {
    extern __shared__ double smem[];
    const int Ne = v.Ne;
    double* lx = smem;
    double* ly = lx + Ne;
    double* lz = ly + Ne;
    int* lid = reinterpret_cast<int*>(lz + Ne);
    __shared__ double red[kBeadBlock / 32];
    __shared__ int wcount[kBeadBlock / 32];
    __shared__ int s_total;

    const int b = blockIdx.x;
    const int s = beads[b].x, p = beads[b].y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (s < 0 || s >= v.M || p < 0 || p >= Ne || !v.on[(size_t)s * Ne + p]) {
        if (tid == 0) out[b] = 0.0;
        return;
    }
    const int eo = s % 2;
    const double vf = eo ? vf1 : vf0;
    const double gf = eo ? gf1 : gf0;
    const double t = (double)shift * tau;
    const bool need_v = (mode != PGB_ACTION_CORR);
    const bool need_c = (mode == PGB_ACTION_CORR) ? (gf > kEPS)
                      : (mode == PGB_ACTION_FULL) ? (shift == 1 && gf > kEPS) : false;

    const double* X = v.pos + (size_t)s * 3 * Ne;
    // `over` (trial positions) replaces the bead's stored position
    const double x1 = over ? over[3 * b] : X[p];
    const double y1 = over ? over[3 * b + 1] : X[Ne + p];
    const double z1 = over ? over[3 * b + 2] : X[2 * Ne + p];
    const int st1 = bead_state(v, s, p);
    if (tid == 0) s_total = 0;
    __syncthreads();

    double vsum = 0.0;
    for (int base = 0; base < Ne; base += kBeadBlock) {
        int j = base + tid;
        bool in = false;
        double dx = 0, dy = 0, dz = 0;
        if (j < Ne && j != p && v.on[(size_t)s * Ne + j]) {
            // LookupTable stores sep = getSeparation(bead2, bead1) = r2 - r1
            dx = min_image(X[j] - x1, v.side[0], v.sideInv[0]);
            dy = min_image(X[Ne + j] - y1, v.side[1], v.sideInv[1]);
            dz = min_image(X[2 * Ne + j] - z1, v.side[2], v.sideInv[2]);
            double3 d = make_double3(dx, dy, dz);
            if (dot3(d, d) < v.rc2) {
                in = true;
                if (need_v) vsum += pair_factor(st1, bead_state(v, s, j)) * V64(v, d);
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) wcount[w] = __popc(m);
        __syncthreads();
        int off = s_total;
        for (int i = 0; i < w; ++i) off += wcount[i];
        if (in) {
            int pos = off + __popc(m & ((1u << lane) - 1u));
            lx[pos] = X[j]; ly[pos] = X[Ne + j]; lz[pos] = X[2 * Ne + j];
            lid[pos] = j;
        }
        __syncthreads();
        if (tid == 0) { int tot = 0; for (int i = 0; i < kBeadBlock / 32; ++i) tot += wcount[i]; s_total += tot; }
        __syncthreads();
    }
    const int nlist = s_total;
    double Vnn = 0.0;
    if (need_v) Vnn = 0.0 + block_sum(vsum, red);   // totVext (0, free) + totVint

    double corr_g = 0.0;
    if (need_c) {
        double tsum = 0.0, f1x = 0.0, f1y = 0.0, f1z = 0.0;
        for (int n = tid; n < nlist; n += kBeadBlock) {
            double x2 = lx[n], y2 = ly[n], z2 = lz[n];
            double3 d12 = make_double3(min_image(x2 - x1, v.side[0], v.sideInv[0]),
                                       min_image(y2 - y1, v.side[1], v.sideInv[1]),
                                       min_image(z2 - z1, v.side[2], v.sideInv[2]));
            double3 F2 = gradV64(v, d12);
            f1x -= F2.x; f1y -= F2.y; f1z -= F2.z;
            double3 F3 = make_double3(0.0, 0.0, 0.0);
            for (int m2 = 0; m2 < nlist; ++m2) {
                if (m2 == n) continue;
                double3 d23 = make_double3(min_image(x2 - lx[m2], v.side[0], v.sideInv[0]),
                                           min_image(y2 - ly[m2], v.side[1], v.sideInv[1]),
                                           min_image(z2 - lz[m2], v.side[2], v.sideInv[2]));
                double3 g = gradV64(v, d23);
                F3.x += g.x; F3.y += g.y; F3.z += g.z;
            }
            double3 Z = make_double3(0.0, 0.0, 0.0);
            tsum += dot3(F2, F2) + 2.0 * dot3(Z, F2) + 2.0 * dot3(F2, F3);
        }
        double T = block_sum(tsum, red);
        double Fx = block_sum(f1x, red), Fy = block_sum(f1y, red), Fz = block_sum(f1z, red);
        double3 Fint1 = make_double3(Fx, Fy, Fz);
        double3 Z = make_double3(0.0, 0.0, 0.0);
        corr_g = T + (dot3(Z, Z) + 2.0 * dot3(Z, Fint1) + dot3(Fint1, Fint1));
    }
    if (tid == 0) {
        double bareU = vf * t * Vnn;
        double corU = need_c ? gf * t * t * t * lambda * corr_g : 0.0;
        double U;
        if (mode == PGB_ACTION_BARE) U = bareU;
        else if (mode == PGB_ACTION_CORR) U = corU;
        else U = bareU + corU;
        out[b] = U;
    }
}

static bool has_corr(int shift, int mode, const double gf[2]) {
    return (gf[0] > kEPS || gf[1] > kEPS) && (mode == PGB_ACTION_CORR || (mode == PGB_ACTION_FULL && shift == 1));
}

// The warp form: whole lists, many beads, and for a gradient term the forces
// of one slice in shared memory.  Returns false when the call is not for it.
static bool bead_warp64(const PathView& v, const int2* d_beads, int k, const BeadSpec& a, bool corr,
                        const double* d_over, double* d_force, double* d_out, cudaStream_t s, cudaError_t* e) {
    const size_t fsmem = (size_t)v.Ne * (3 * sizeof(double) + 3 * sizeof(float));
    if (k < (corr ? many_gradient(v) : kManyBeads) || (corr && (!d_force || fsmem > 200 * 1024))) return false;
    if (corr) {
        if ((*e = set_smem_limit(k_slice_forces64, 200 * 1024)) != cudaSuccess) return true;
        k_slice_forces64<<<dim3(v.M, (v.Ne + kForceRows - 1) / kForceRows), kPairBlock, fsmem, s>>>(
            v, 1.0 / v.dr, a.gf[0] > kEPS, a.gf[1] > kEPS, d_force);
    }
    const int grid = (k + kBlockBeads - 1) / kBlockBeads;
    if (d_over) k_bead_warp64<true><<<grid, kPairBlock, 0, s>>>(v, 1.0 / v.dr, d_beads, k, a, d_over, d_force, d_out);
    else k_bead_warp64<false><<<grid, kPairBlock, 0, s>>>(v, 1.0 / v.dr, d_beads, k, a, nullptr, d_force, d_out);
    *e = cudaGetLastError();
    return true;
}

cudaError_t launch_bead_actions64(const PathView& v, const int2* d_beads, int k, int shift,
                                  int mode, double tau, double lambda, const double vf[2],
                                  const double gf[2], const double* d_over, double* d_force, bool whole,
                                  double* d_out, cudaStream_t s) {
    if (k <= 0) return cudaSuccess;
    const BeadSpec a{shift, mode, tau, lambda, {vf[0], vf[1]}, {gf[0], gf[1]}};
    const bool corr = has_corr(shift, mode, gf);
    cudaError_t e = cudaSuccess;
    if (whole && !d_over && bead_warp64(v, d_beads, k, a, corr, nullptr, d_force, d_out, s, &e)) return e;
    if ((size_t)v.Ne * bead_pairs_bytes(false) <= 200 * 1024)
        return bead_pairs64<false>(v, d_beads, k, a, corr, d_over, d_out, s);
    const size_t smem = (size_t)v.Ne * (3 * sizeof(double) + sizeof(int));
    if ((e = set_smem_limit(k_bead_actions64, 200 * 1024)) != cudaSuccess) return e;
    k_bead_actions64<<<k, kBeadBlock, smem, s>>>(v, d_beads, k, shift, mode, tau, lambda,
                                                 vf[0], vf[1], gf[0], gf[1], d_over, d_out);
    return cudaGetLastError();
}

bool launch_trial_actions64(const PathView& v, const int2* d_beads, int k, int shift, int mode, double tau,
                            double lambda, const double vf[2], const double gf[2], const double* d_over,
                            double* d_force, double* d_out, cudaStream_t s, cudaError_t* e) {
    *e = cudaSuccess;
    if (k <= 0) return true;
    const BeadSpec a{shift, mode, tau, lambda, {vf[0], vf[1]}, {gf[0], gf[1]}};
    const bool corr = has_corr(shift, mode, gf);
    if (bead_warp64(v, d_beads, k, a, corr, d_over, d_force, d_out, s, e)) return true;
    if ((size_t)v.Ne * bead_pairs_bytes(true) > 200 * 1024) return false;
    *e = bead_pairs64<true>(v, d_beads, k, a, corr, d_over, d_out, s);
    return true;
}

// ---------------------------------------------------------------------------
// Per-slice terms of the estimators:
//   vint: LocalAction::V(slice)            action.cpp:902-947 (i<j, sep r2-r1)
//   g2:   gradVSquared(slice)              action.cpp:1188-1223
//   r1,d1: rDOTgradUterm1/deltadotgradUterm1 sums (action.cpp:1446,1588)
//   r2,d2: T-matrix terms of rDOTgradUterm2/deltadotgradUterm2 (1503,1700)
//   kin:  sum |getVelocity|^2                path.h:189-203
//   xch:  sum (r_{t+W}-r_t).(r_{t+1}-r_t)     estimator.cpp:1138-1152
// Output layout: terms[q * M + t] for q = 0..7 in the order above; terms above
// a slice's level (kSliceNone .. kSliceT) are 0.
//
// Bound: the FP64 pipe, 16 clocks of an SM a warp instruction.  A potential
// alone takes each pair once (about 20 instructions); forces take each ordered
// pair, because the sums belong to one bead: 64 beads a CTA, four (eight)
// threads a bead over its partners, 24 instructions a pair, 39 with the T
// matrix (one coefficient c1 = (V'' - |V'|/r)/r^2 on r r^T and |V'|/r on the
// diagonal, where the direct form divides eighteen times).  The centroid
// window's two chains of links run on two of those threads.  An energy and a
// virial sample of 64 particles, 124 slices, primitive action: 2 x 586 us with
// one thread a bead, everything computed in the direct form; 73 us together
// here (the potential alone, then forces).
// ---------------------------------------------------------------------------
constexpr int kSliceRows = 64;

__device__ __forceinline__ double3 pos64(const PathView& v, int2 b) {
    const double* X = v.pos + (size_t)b.x * 3 * v.Ne;
    return make_double3(X[b.y], X[v.Ne + b.y], X[2 * v.Ne + b.y]);
}
__device__ __forceinline__ float3 fraction64(const PathView& v, int2 b) {
    const float4 f = v.pos32[(size_t)b.x * v.Ne + b.y];
    return make_float3(box_fraction(f.x, (float)v.sideInv[0]), box_fraction(f.y, (float)v.sideInv[1]),
                       box_fraction(f.z, (float)v.sideInv[2]));
}
// getSeparation(a, b) = r_a - r_b in the box (path.h:179-184)
__device__ __forceinline__ double3 link64(const PathView& v, double3 a, float3 ua, double3 b, float3 ub) {
    bool ok = true;
    const double x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    double3 d = make_double3(image64(x, ua.x - ub.x, v.side[0], ok), image64(y, ua.y - ub.y, v.side[1], ok),
                             image64(z, ua.z - ub.z, v.side[2], ok));
    if (!ok)
        d = make_double3(min_image(x, v.side[0], v.sideInv[0]), min_image(y, v.side[1], v.sideInv[1]),
                         min_image(z, v.side[2], v.sideInv[2]));
    return d;
}

// The sum over g < window of the displacement from a bead to its g-th
// neighbour along `link`, the displacement to the window-th one and the first
// step.  An open end stops the walk, and stands for the neighbours behind it.
struct ChainSums { double3 sum, reach, step; };
__device__ __forceinline__ ChainSums chain64(const PathView& v, const int2* __restrict__ link, int s, int p, int window) {
    ChainSums c{};
    int2 at = make_int2(s, p);
    double3 r = pos64(v, at);
    float3 u = fraction64(v, at);
    for (int g = 0; g < window; ++g) {
        c.sum.x += c.reach.x; c.sum.y += c.reach.y; c.sum.z += c.reach.z;
        if (at.x >= 0) at = link[(size_t)at.x * v.Ne + at.y];
        if (at.x < 0) continue;
        const double3 q = pos64(v, at);
        const float3 w = fraction64(v, at);
        const double3 d = link64(v, q, w, r, u);
        c.reach.x += d.x; c.reach.y += d.y; c.reach.z += d.z;
        if (g == 0) c.step = d;
        r = q; u = w;
    }
    return c;
}

// one slice's row block with forces (and the T matrix): adds to the thread's
// vint g2 r1 r2 d1 d2 kin xch
template <bool kT>
__device__ __forceinline__ void slice_rows64(const PathView& v, double invdr, int s, int n, int b0, int window,
                                             const double* lx, const double* ly, const double* lz,
                                             double (*buf)[kPairBlock], double (&val)[8]) {
    constexpr int Q = kT ? 10 : 3;
    const int nb = min(kSliceRows, n - b0);
    if (nb <= 0) return;                                        // uniform over the CTA
    const int rows = nb > 32 ? 64 : 32, parts = kPairBlock / rows, tid = threadIdx.x;
    const int r = tid & (rows - 1), part = tid / rows, i = b0 + r;
    const float4* P = v.pos32 + (size_t)s * v.Ne;
    const float Ix = (float)v.sideInv[0], Iy = (float)v.sideInv[1], Iz = (float)v.sideInv[2];
    const bool worm = worm_on_slice(v, s);
    // F(3), T: xx yy zz xy xz yz and the diagonal's sum
    double acc[10] = {};
    if (r < nb) {
        const double x1 = lx[i], y1 = ly[i], z1 = lz[i];
        const float4 f = P[i];
        const float u1 = box_fraction(f.x, Ix), u2 = box_fraction(f.y, Iy), u3 = box_fraction(f.z, Iz);
        const int st1 = worm ? bead_state(v, s, i) : 2;
        for (int j = part; j < n; j += parts) {
            if (j == i) continue;
            const float4 q = P[j];
            const Pair64 d = pair64(v, invdr, x1 - lx[j], y1 - ly[j], z1 - lz[j], u1 - box_fraction(q.x, Ix),
                                    u2 - box_fraction(q.y, Iy), u3 - box_fraction(q.z, Iz));
            const double dV = table64(v.tdV, d.k), g = dV * d.y;
            acc[0] = __fma_rn(g, d.dx, acc[0]); acc[1] = __fma_rn(g, d.dy, acc[1]); acc[2] = __fma_rn(g, d.dz, acc[2]);
            if (j > i) val[0] += (worm ? pair_factor(st1, bead_state(v, s, j)) : 1.0) * table64(v.tV, d.k);
            if (kT) {
                const double c0 = fabs(g), c1 = (table64(v.td2V, d.k) - c0) * (d.y * d.y);
                const double tx = c1 * d.dx, ty = c1 * d.dy, tz = c1 * d.dz;
                acc[3] = __fma_rn(tx, d.dx, acc[3] + c0); acc[4] = __fma_rn(ty, d.dy, acc[4] + c0);
                acc[5] = __fma_rn(tz, d.dz, acc[5] + c0);
                acc[6] = __fma_rn(tx, d.dy, acc[6]); acc[7] = __fma_rn(tx, d.dz, acc[7]); acc[8] = __fma_rn(ty, d.dz, acc[8]);
            }
        }
    }
    // the bead's neighbours along its worldline: forward on its first thread,
    // backward on its second
    ChainSums c{};
    if (r < nb && part < 2 && window > 0) c = chain64(v, part ? v.prev : v.next, s, i, window);
    __syncthreads();
    #pragma unroll
    for (int q = 0; q < Q; ++q) buf[q][tid] = acc[q];
    if (part == 1) { buf[Q][r] = c.sum.x; buf[Q][64 + r] = c.sum.y; buf[Q][128 + r] = c.sum.z; }
    __syncthreads();
    for (int q = part; q < Q; q += parts) {                     // every part adds some of the quantities
        double t = buf[q][r];
        for (int k = 1; k < parts; ++k) t += buf[q][r + k * rows];
        buf[q][r] = t;
    }
    __syncthreads();
    if (r >= nb || part) return;
    const double Fx = buf[0][r], Fy = buf[1][r], Fz = buf[2][r];
    const double x1 = lx[i], y1 = ly[i], z1 = lz[i];
    val[1] = __fma_rn(Fx, Fx, __fma_rn(Fy, Fy, Fz * Fz));
    if (window <= 0) return;
    val[2] = __fma_rn(Fx, x1, __fma_rn(Fy, y1, Fz * z1));
    // centroid deviation delta = r - com, com the mean of the window's two
    // walks (action.cpp:1625-1645)
    const double den = -1.0 / (2.0 * window);
    const double ex = min_image((c.sum.x + buf[Q][r]) * den, v.side[0], v.sideInv[0]);
    const double ey = min_image((c.sum.y + buf[Q][64 + r]) * den, v.side[1], v.sideInv[1]);
    const double ez = min_image((c.sum.z + buf[Q][128 + r]) * den, v.side[2], v.sideInv[2]);
    val[4] = __fma_rn(Fx, ex, __fma_rn(Fy, ey, Fz * ez));
    val[7] = __fma_rn(c.reach.x, c.step.x, __fma_rn(c.reach.y, c.step.y, c.reach.z * c.step.z));
    if (kT) {
        const double a = buf[6][r], b = buf[7][r], e = buf[8][r];
        const double TFx = __fma_rn(buf[3][r], Fx, __fma_rn(a, Fy, b * Fz));
        const double TFy = __fma_rn(a, Fx, __fma_rn(buf[4][r], Fy, e * Fz));
        const double TFz = __fma_rn(b, Fx, __fma_rn(e, Fy, buf[5][r] * Fz));
        val[3] = __fma_rn(TFx, x1, __fma_rn(TFy, y1, TFz * z1));
        val[5] = __fma_rn(TFx, ex, __fma_rn(TFy, ey, TFz * ez));
    }
}

// blocks of a slice: row blocks of kSliceRows beads; with several, each leaves
// its eight sums in `part` and the last to arrive adds them in block order
__global__ void __launch_bounds__(kPairBlock)
k_slice_terms64(PathView v, double invdr, int window, int even, int odd, unsigned* __restrict__ arrived,
                double* __restrict__ part, double* __restrict__ terms) {
    extern __shared__ double sm[];
    __shared__ double buf[11][kPairBlock];
    __shared__ double sums[8];
    __shared__ bool last;
    const int s = blockIdx.x, Ne = v.Ne, n = v.nbs[s], tid = threadIdx.x, nblk = gridDim.y;
    const int level = s % 2 ? odd : even, b0 = blockIdx.y * kSliceRows;
    double *lx = sm, *ly = lx + Ne, *lz = ly + Ne;
    if (level > kSliceNone) {
        const double* X = v.pos + (size_t)s * 3 * Ne;
        for (int j = tid; j < n; j += kPairBlock) { lx[j] = X[j]; ly[j] = X[Ne + j]; lz[j] = X[2 * Ne + j]; }
        __syncthreads();
    }
    double val[8] = {};
    if (level == kSliceT) slice_rows64<true>(v, invdr, s, n, b0, window, lx, ly, lz, buf, val);
    else if (level == kSliceF) slice_rows64<false>(v, invdr, s, n, b0, window, lx, ly, lz, buf, val);
    else if (level == kSliceV && n > 1) {
        // each pair once, by offset around the slice (as in k_bead_pairs64)
        const float4* P = v.pos32 + (size_t)s * Ne;
        const float Ix = (float)v.sideInv[0], Iy = (float)v.sideInv[1], Iz = (float)v.sideInv[2];
        const bool worm = worm_on_slice(v, s);
        const int half = (n - 1) / 2, total = n * half + (n % 2 ? 0 : n / 2);
        const int stride = nblk * kPairBlock, so = stride / n, si = stride - so * n;
        int idx = blockIdx.y * kPairBlock + tid;
        int o = idx / n, i = idx - o * n;
        ++o;
        for (; idx < total; idx += stride) {
            int j = i + o;
            if (j >= n) j -= n;
            const float4 a = P[i], b = P[j];
            const Pair64 d = pair64(v, invdr, lx[i] - lx[j], ly[i] - ly[j], lz[i] - lz[j],
                                    box_fraction(a.x, Ix) - box_fraction(b.x, Ix), box_fraction(a.y, Iy) - box_fraction(b.y, Iy),
                                    box_fraction(a.z, Iz) - box_fraction(b.z, Iz));
            val[0] += (worm ? pair_factor(bead_state(v, s, i), bead_state(v, s, j)) : 1.0) * table64(v.tV, d.k);
            i += si; o += so;
            if (i >= n) { i -= n; ++o; }
        }
    }
    if (tid < kSliceRows && b0 + tid < n) {
        const int2 at = make_int2(s, b0 + tid), nx = v.next[(size_t)s * Ne + at.y];
        if (nx.x >= 0) {
            const double3 d = link64(v, pos64(v, nx), fraction64(v, nx), pos64(v, at), fraction64(v, at));
            val[6] = __fma_rn(d.x, d.x, __fma_rn(d.y, d.y, d.z * d.z));
        }
    }
    block_sums<8>(val, buf, sums);
    if (nblk == 1) {
        if (tid < 8) terms[(size_t)tid * v.M + s] = sums[tid];
        return;
    }
    if (tid < 8) { part[((size_t)s * nblk + blockIdx.y) * 8 + tid] = sums[tid]; __threadfence(); }
    __syncthreads();
    if (tid == 0) last = atomicInc(arrived + s, nblk - 1) == nblk - 1;      // back to 0 for the next call
    __syncthreads();
    if (!last || tid >= 8) return;
    __threadfence();
    double t = 0.0;
    for (int k = 0; k < nblk; ++k) t += __ldcg(part + ((size_t)s * nblk + k) * 8 + tid);
    terms[(size_t)tid * v.M + s] = t;
}

static int slice_blocks(int Ne) { return (Ne + kSliceRows - 1) / kSliceRows; }

size_t slice_terms64_work(const PathView& v) { return (size_t)8 * v.M * slice_blocks(v.Ne) * sizeof(double); }

cudaError_t launch_slice_terms64(const PathView& v, int window, int even, int odd, unsigned* d_arrived,
                                 void* d_work, double* d_terms, cudaStream_t s) {
    const size_t smem = (size_t)v.Ne * 3 * sizeof(double);
    const cudaError_t ae = set_smem_limit(k_slice_terms64, 200 * 1024);
    if (ae != cudaSuccess) return ae;
    k_slice_terms64<<<dim3(v.M, slice_blocks(v.Ne)), kPairBlock, smem, s>>>(
        v, 1.0 / v.dr, window, even, odd, d_arrived, static_cast<double*>(d_work), d_terms);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// rho_q(t) = sum_j exp(i q . r_j(t)) in FP64 (raw positions, as gpu_isf uses
// raw bead coordinates).
//
// A lattice vector q = 2 pi n / L (every vector of the reference's lattice
// lists) needs no sine per bead: exp(i q . r) is the product of the
// exp(i q_d r_d), and a CTA keeps these of its slice's beads in shared memory
// for every |q_d| that its vectors have, at the place |n_d|.  (Each is a sine
// and a cosine of its own.  Made by products from exp(2 pi i r_d / L_d) they
// were cheaper, but the roundings of 1 / L and of q_d itself then shift all
// phases alike, which F(q,tau) does not average out.)  One thread sums one
// vector over the beads: eight FP64 multiply-adds a bead where the phase and
// its sines take 26, and the FP64 pipe (16 clocks of an SM a warp instruction)
// is the bound.  A list that enumerates a grid symmetric about 0 has -q at the
// mirrored place; its density is the complex conjugate and is written, not
// summed.  Other vectors (shells), and lattice vectors that are too few for
// their table, take the sines.
//
// A cluster of CTAs shares a slice's beads, each with all the vectors and a
// table of its own beads, and adds the parts through distributed shared
// memory: slices are too few and too long to even out over the SMs (250 on
// 152: two on some, one on others), and a table built by every CTA that takes
// some of the vectors is built twice.
//
// S(q) calls, a warp a vector and slice with sincos, and here: 64 beads, 124
// slices, 400 lattice vectors 232 and 83 us, 400 others 232 and 220; 160 beads,
// 250 slices, 200: 525 and 228, 525 and 513; 17 beads, 1000 slices, 96: 255 and
// 62, 255 and 117.  Error of the densities relative to extended precision,
// sincos and here: 40 beads, 62 slices 1.1e-15 and 6.8e-16, 64 beads, |q| < 2
// 4.2e-16 and 3.6e-16, 160 beads 1.6e-15 and 1.0e-15, shells of 100 beads 4.8e-16
// and 4.1e-16; of F(q,tau) 3.7e-16 and 2.7e-16, 2.2e-16 and 2.5e-16, 4.1e-16 and
// 3.1e-16, 2.3e-16 and 1.8e-16.
// ---------------------------------------------------------------------------
constexpr int kRhoThreads = 512;                 // vectors a CTA at most
constexpr int kRhoLeast = 128;                   // threads at least: few vectors share the beads out
constexpr int kRhoPowers = 64;                   // largest |n_d| of the table form
constexpr int kRhoSmem = 48 * 1024;              // four CTAs an SM
constexpr int kRhoCluster = 8;
constexpr int kRhoBeads = 3;                     // a CTA has at least
// Fewer vectors than kRhoFew, or fewer slices than kRhoShort and CTAs (a slice
// and set of vectors each) than three times that, take a warp a vector and
// slice: a CTA a slice and cluster rank leaves the GPU empty there.
// S(q) in this form and the other, us: 65 beads, 250 slices, 1 vector 17 and 34,
// 16 40 and 40, 24 48 and 50, 32 62 and 55; 64 beads, 124 slices, 16 19 and 22,
// 24 25 and 25, 32 30 and 29.  S(q) and F(q,tau) of 24 beads, 16 slices, 400
// vectors 60 and 74 (lattice), 60 and 209 (others); of 5 beads, 20 slices, 4000
// lattice vectors 267 and 97.
constexpr int kRhoFew = 24, kRhoShort = 32;
// FP64 instructions that a table saves a vector and bead, and that it takes an entry
constexpr int kRhoSaved = 18, kRhoEntry = 24;

// 2 pi / L and L / 2 pi
struct Lattice { double step[3], turn[3]; };

// n_d when q_d is 2 pi n_d / L_d to rounding, else kRhoPowers + 1
__device__ __forceinline__ int lattice_index(double q, double step, double turn) {
    const double n = rint(q * turn);
    const bool ok = fabs(n) <= (double)kRhoPowers && fabs(q - n * step) <= 1.0e-15 * fabs(q);
    return ok ? (int)n : kRhoPowers + 1;
}

// exp(i q_d r_d) from the table, the conjugate for n < 0
__device__ __forceinline__ double2 power_of(const double2* E, int n) {
    double2 e = E[n < 0 ? -n : n];
    e.y = __hiloint2double(__double2hiint(e.y) ^ (n & 0x80000000), __double2loint(e.y));
    return e;
}

// (cos x, sin x): x less the nearest quarter turn in two parts (Cody and
// Waite's reduction), Taylor's series of the rest (|r| <= pi/4: the terms left
// out are below 5e-17 of the sine, 2e-18 of the cosine), the quarter turns by
// swap and signs.  21 FP64 instructions; sincos() takes about thirty.
static __device__ __noinline__ double2 far_sines(double x) {
    double sn, cs;
    sincos(x, &sn, &cs);
    return make_double2(cs, sn);
}
__device__ __forceinline__ double2 sines64(double x) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x4197D784) return far_sines(x);     // 1e8 and up, NaN
    const double magic = 6755399441055744.0;                         // 1.5 2^52
    const double t = __fma_rn(x, 0.63661977236758134308, magic), f = t - magic;      // 2 / pi
    const int k = __double2loint(t);
    // pi / 2 rounded, and what is left of it
    const double r = __fma_rn(f, -6.12323399573676588614e-17, __fma_rn(f, -1.57079632679489661923, x)), y = r * r;
    double s = -1.0 / 1307674368000.0, c = 1.0 / 20922789888000.0;   // 1 / 15!, 1 / 16!
    s = __fma_rn(s, y, 1.0 / 6227020800.0); c = __fma_rn(c, y, -1.0 / 87178291200.0);
    s = __fma_rn(s, y, -1.0 / 39916800.0); c = __fma_rn(c, y, 1.0 / 479001600.0);
    s = __fma_rn(s, y, 1.0 / 362880.0); c = __fma_rn(c, y, -1.0 / 3628800.0);
    s = __fma_rn(s, y, -1.0 / 5040.0); c = __fma_rn(c, y, 1.0 / 40320.0);
    s = __fma_rn(s, y, 1.0 / 120.0); c = __fma_rn(c, y, -1.0 / 720.0);
    s = __fma_rn(s, y, -1.0 / 6.0); c = __fma_rn(c, y, 1.0 / 24.0);
    s = __fma_rn(r * y, s, r); c = __fma_rn(c, y, -0.5);
    c = __fma_rn(c, y, 1.0);
    const double a = k & 1 ? s : c, b = k & 1 ? c : s;
    return make_double2(__hiloint2double(__double2hiint(a) ^ ((k + 1) & 2) << 30, __double2loint(a)),
                        __hiloint2double(__double2hiint(b) ^ (k & 2) << 30, __double2loint(b)));
}

// Few vectors: one warp per (q, t), a sine and a cosine a bead.
__global__ void __launch_bounds__(256)
k_rhoq64_few(PathView v, const double* __restrict__ q, int nq, double maxR2, double* __restrict__ rho) {
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= (long long)nq * v.M) return;
    const int iq = (int)(gw / v.M), t = (int)(gw - (long long)iq * v.M), n = v.nbs[t];
    const double qx = q[3 * iq], qy = q[3 * iq + 1], qz = q[3 * iq + 2];
    const double* X = v.pos + (size_t)t * 3 * v.Ne;
    double re = 0.0, im = 0.0;
    for (int j = lane; j < n; j += 32) {
        // cylinder restriction: only beads with x^2 + y^2 < maxR^2
        if (maxR2 > 0.0 && !(X[j] * X[j] + X[v.Ne + j] * X[v.Ne + j] < maxR2)) continue;
        double ph = 0.0;
        ph += qx * X[j]; ph += qy * X[v.Ne + j]; ph += qz * X[2 * v.Ne + j];
        double sn, cs;
        sincos(ph, &sn, &cs);
        re += cs; im += sn;
    }
    re = warp_sum(re); im = warp_sum(im);
    if (lane == 0) reinterpret_cast<double2*>(rho)[gw] = make_double2(re, im);
}

// Thread slot + wide * part, part < parts, has vector slot of the CTA's vectors
// and every parts-th of its beads.
__global__ void __launch_bounds__(kRhoThreads)
k_rhoq64(PathView v, const double* __restrict__ q, int nq, Lattice lat, double maxR2, int wide, int parts, int csize,
         double* __restrict__ rho) {
    extern __shared__ double2 E[];               // [bead][dimension][power]
    __shared__ int s_max;
    __shared__ unsigned long long comp[3][kRhoPowers + 1];   // the |q_d| that a table entry stands for
    const int t = blockIdx.x / csize, rank = blockIdx.x - t * csize, tid = threadIdx.x, T = blockDim.x;
    const int part = tid / wide, n = v.nbs[t];
    const int b0 = (int)((long long)n * rank / csize), b1 = (int)((long long)n * (rank + 1) / csize);
    const int i = blockIdx.y * wide + tid - part * wide, j = nq - 1 - i;
    const double* X = v.pos + (size_t)t * 3 * v.Ne;
    bool live = part < parts && i < nq, mirrored = live;
    int k[3] = {0, 0, 0};
    if (tid == 0) s_max = 0;
    for (int x = tid; x < 3 * (kRhoPowers + 1); x += T) comp[0][x] = ~0ull;
    __syncthreads();
    double a[3] = {0.0, 0.0, 0.0};
    if (live) {
        #pragma unroll
        for (int d = 0; d < 3; ++d) {
            a[d] = q[3 * i + d];
            mirrored = mirrored && a[d] == -q[3 * j + d];
        }
        live = i <= j || !mirrored;              // the other half of a mirrored pair writes both
        #pragma unroll
        for (int d = 0; d < 3; ++d)
            if (live) k[d] = lattice_index(a[d], lat.step[d], lat.turn[d]);
    }
    const int most = max(abs(k[0]), max(abs(k[1]), abs(k[2])));
    bool powers = live && most <= kRhoPowers;
    // components of one index that differ in the last places: the smallest has the entry
    auto bits = [&](int d) { return (unsigned long long)__double_as_longlong(fabs(a[d])); };
    if (powers)
        for (int d = 0; d < 3; ++d) atomicMin(&comp[d][abs(k[d])], bits(d));
    __syncthreads();
    if (powers)
        for (int d = 0; d < 3; ++d) powers = powers && comp[d][abs(k[d])] == bits(d);
    const int nv = __syncthreads_count(powers && part == 0);
    const int warp_most = __reduce_max_sync(0xffffffffu, powers ? most + 1 : 0);
    if ((tid & 31) == 0 && warp_most) atomicMax(&s_max, warp_most);
    __syncthreads();
    double2 S = make_double2(0.0, 0.0);
    int np = s_max;                              // entries 0 .. np - 1; 0: no lattice vector here
    if (nv * kRhoSaved < 3 * kRhoEntry * (np - 1)) { powers = false; np = 0; }
    if (np > 0) {
        const int chunk = max(parts, kRhoSmem / (3 * np * (int)sizeof(double2)));
        for (int j0 = b0; j0 < b1; j0 += chunk) {
            const int nj = min(chunk, b1 - j0);
            __syncthreads();
            for (int x = tid; x < 3 * nj * np; x += T) {
                const int h = x / (3 * nj), dp = x - h * (3 * nj), d = dp / nj, p = dp - d * nj;
                double2 e = make_double2(1.0, 0.0);
                const unsigned long long m = comp[d][h];
                if (h > 0) e = sines64(m == ~0ull ? 0.0 : __longlong_as_double((long long)m) * X[d * v.Ne + j0 + p]);
                // cylinder restriction: beads outside x^2 + y^2 < maxR^2 count 0
                if (d == 0 && maxR2 > 0.0) {
                    const double rx = X[j0 + p], ry = X[v.Ne + j0 + p];
                    if (!(rx * rx + ry * ry < maxR2)) e = make_double2(0.0, 0.0);
                }
                E[(size_t)(3 * p + d) * np + h] = e;
            }
            __syncthreads();
            if (powers)
                for (int p = part; p < nj; p += parts) {
                    const double2* e = E + (size_t)3 * p * np;
                    const double2 x = power_of(e, k[0]), y = power_of(e + np, k[1]), z = power_of(e + 2 * np, k[2]);
                    const double cr = __fma_rn(y.x, z.x, -(y.y * z.y)), ci = __fma_rn(y.x, z.y, y.y * z.x);
                    S.x = __fma_rn(x.x, cr, __fma_rn(-x.y, ci, S.x));
                    S.y = __fma_rn(x.x, ci, __fma_rn(x.y, cr, S.y));
                }
        }
    }
    if (live && !powers) {
        const double qx = q[3 * i], qy = q[3 * i + 1], qz = q[3 * i + 2];
        for (int p = b0 + part; p < b1; p += parts) {
            if (maxR2 > 0.0 && !(X[p] * X[p] + X[v.Ne + p] * X[v.Ne + p] < maxR2)) continue;
            const double2 e = sines64(__fma_rn(qx, X[p], __fma_rn(qy, X[v.Ne + p], qz * X[2 * v.Ne + p])));
            S.x += e.x; S.y += e.y;
        }
    }
    double2* R = reinterpret_cast<double2*>(rho);
    auto write = [&](double2 A) {
        R[(size_t)i * v.M + t] = A;
        if (mirrored && i < j) R[(size_t)j * v.M + t] = make_double2(A.x, -A.y);
    };
    if (parts * csize == 1) {
        if (live) write(S);
        return;
    }
    // the parts, then the CTAs, added in order; the CTAs take turns at the vectors
    __syncthreads();
    E[tid] = S;
    if (csize > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (live && part == 0 && (tid / 32) % csize == rank) {
        S = make_double2(0.0, 0.0);
        for (int r = 0; r < csize; ++r) {
            const double2* Er = csize > 1 ? cg::this_cluster().map_shared_rank(E, r) : E;
            for (int h = 0; h < parts; ++h) {
                const double2 a = Er[tid + h * wide];
                S.x += a.x; S.y += a.y;
            }
        }
        write(S);
    }
    if (csize > 1) cg::this_cluster().sync();    // no CTA leaves while another reads its part
}

cudaError_t launch_rhoq64(const PathView& v, const double* d_q, int nq, double* d_rho,
                          cudaStream_t s, double maxR2) {
    if (nq < 1) return cudaSuccess;
    const int sets = (nq + kRhoThreads - 1) / kRhoThreads;
    if (nq < kRhoFew || (v.M < kRhoShort && v.M * sets < 3 * kRhoShort)) {
        k_rhoq64_few<<<(int)(((long long)nq * v.M + 7) / 8), 256, 0, s>>>(v, d_q, nq, maxR2, d_rho);
        return cudaGetLastError();
    }
    const cudaError_t ae = set_smem_limit(k_rhoq64, kRhoSmem);
    if (ae != cudaSuccess) return ae;
    const int each = (nq + sets - 1) / sets;
    const int wide = each, parts = std::max(1, kRhoLeast / wide);
    // rounds of the SMs, in units of a whole slice: a cluster costs two
    // barriers and a table each, so it has to gain (124 slices of 64 beads, one
    // round either way: 357 us a sample with one CTA a slice, 367 with two,
    // 390 with four; 250 of 128: 464 with two, 439 with four)
    auto rounds = [&](int c) { return (double)(((long long)v.M * sets * c + 151) / 152) / c; };
    int c = 1;
    // (a cluster of eight pays for short paths and many vectors: 160 beads, 80
    // slices, 400 vectors off the lattice 1.37 of the sines' time with four, 1.18
    // with eight, 17 lattice vectors 0.71 and 1.01)
    const int most = v.M < 84 && nq >= 128 ? kRhoCluster : 4;
    for (int d = 2; d <= most && d * kRhoBeads <= v.Ne; d *= 2)
        if (rounds(d) < 0.95 * rounds(c)) c = d;
    Lattice lat;
    const double kTwoPi = 6.283185307179586476925;
    for (int d = 0; d < 3; ++d) { lat.step[d] = kTwoPi / v.side[d]; lat.turn[d] = v.side[d] / kTwoPi; }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)v.M * c, (unsigned)sets);
    cfg.blockDim = dim3((wide * parts + 31) / 32 * 32);
    cfg.dynamicSmemBytes = kRhoSmem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = c > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_rhoq64, v, d_q, nq, lat, maxR2, wide, parts, c, d_rho);
}

// F(q,tau) = norm * sum_t Re(rho_t conj(rho_{t+tau})), tau in [0, M/2].  One
// CTA a wave vector and kIsfThreads tau, the vector's densities in shared
// memory with the first half repeated behind them (no wrap in the loop), one
// thread a tau: two FP64 multiply-adds a term, even and odd slices in sums of
// their own, the FP64 pipe the bound.  300 vectors, M = 250: 79 us with one
// thread an output from L1, 35 us here; one vector, M = 1000, whole calls: 340 us,
// 378 with all tau in one CTA, 109 here.
constexpr int kIsfThreads = 128;

__global__ void __launch_bounds__(kIsfThreads)
k_isf_direct64(const double* __restrict__ rho, int M, double norm, double* __restrict__ out) {
    extern __shared__ double2 E[];
    const int nt = M / 2 + 1;
    const double2* r = reinterpret_cast<const double2*>(rho) + (size_t)blockIdx.x * M;
    for (int t = threadIdx.x; t < M + nt; t += kIsfThreads) E[t] = r[t < M ? t : t - M];
    __syncthreads();
    const int tau = blockIdx.y * kIsfThreads + threadIdx.x;
    if (tau >= nt) return;
    double sum[2] = {0.0, 0.0};
    int t = 0;
    #pragma unroll 2
    for (; t + 1 < M; t += 2) {
        #pragma unroll
        for (int u = 0; u < 2; ++u) {
            const double2 a = E[t + u], b = E[t + u + tau];
            sum[u] = __fma_rn(a.x, b.x, __fma_rn(a.y, b.y, sum[u]));
        }
    }
    if (t < M) sum[0] = __fma_rn(E[t].x, E[t + tau].x, __fma_rn(E[t].y, E[t + tau].y, sum[0]));
    out[(size_t)blockIdx.x * nt + tau] = (sum[0] + sum[1]) * norm;
}

// the same straight from memory, for slices whose densities do not fit
__global__ void k_isf_long64(const double* __restrict__ rho, int nq, int M, double norm,
                             double* __restrict__ out) {
    int nt = M / 2 + 1;
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)nq * nt) return;
    int iq = (int)(i / nt), tau = (int)(i % nt);
    const double* r = rho + (size_t)iq * M * 2;
    double acc = 0.0;
    for (int t = 0; t < M; ++t) {
        int t2 = t + tau; if (t2 >= M) t2 -= M;
        acc += r[2*t] * r[2*t2] + r[2*t+1] * r[2*t2+1];
    }
    out[i] = acc * norm;
}

cudaError_t launch_isf_direct64(const double* d_rho, int nq, int M, double norm,
                                double* d_out, cudaStream_t s) {
    if (nq < 1) return cudaSuccess;
    const size_t smem = (size_t)(M + M / 2 + 1) * sizeof(double2);
    if (smem <= 200 * 1024) {
        const cudaError_t ae = set_smem_limit(k_isf_direct64, 200 * 1024);
        if (ae != cudaSuccess) return ae;
        const dim3 grid(nq, (M / 2 + kIsfThreads) / kIsfThreads);        // M / 2 + 1 tau
        k_isf_direct64<<<grid, kIsfThreads, smem, s>>>(d_rho, M, norm, d_out);
        return cudaGetLastError();
    }
    long long n = (long long)nq * (M / 2 + 1);
    k_isf_long64<<<(int)((n + 255) / 256), 256, 0, s>>>(d_rho, nq, M, norm, d_out);
    return cudaGetLastError();
}

__global__ void k_ssf_from_rho64(const double* __restrict__ rho, int nq, int M, double norm,
                                 double* __restrict__ out) {
    int iq = blockIdx.x;
    __shared__ double red[8];
    double acc = 0.0;
    for (int t = threadIdx.x; t < M; t += blockDim.x) {
        double a = rho[((size_t)iq * M + t) * 2], b = rho[((size_t)iq * M + t) * 2 + 1];
        acc += a * a + b * b;
    }
    double s = block_sum(acc, red);
    if (threadIdx.x == 0) out[iq] = s * norm;
}

cudaError_t launch_ssf_from_rho64(const double* d_rho, int nq, int M, double norm,
                                  double* d_out, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    k_ssf_from_rho64<<<nq, 256, 0, s>>>(d_rho, nq, M, norm, d_out);
    return cudaGetLastError();
}

}  // namespace pgb
