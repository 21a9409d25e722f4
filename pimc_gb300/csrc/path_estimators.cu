// path_estimators.cu -- the path-wide estimators adjacent to the hot path:
// pair correlation g(r), winding-number superfluid fraction and permutation
// cycles (estimator.cpp:2000-2074, 2735-2781, 3181-3246).  FP64, compiled
// with -fmad=false so that every separation, and therefore every histogram
// bin, is the one the reference computes.
#include <algorithm>

#include "pgb_device.cuh"

namespace pgb {

constexpr int kPcfBins = 50;                 // NPCFSEP, include/common.h:85
constexpr int kEstBlock = 256;

// The last CTA of a grid to arrive; the others' global writes are visible to
// it.  The counter returns to 0 for the next call.
__device__ __forceinline__ bool last_to_arrive(unsigned* counter, unsigned blocks) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(counter, blocks - 1) == blocks - 1;
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Separation histogram of the pairs b1 < b2 of slices [t0, t1) with
// ActionBase::updateSepHist's binning (action.cpp:216-224):
// nR = int(|r_b2 - r_b1| / dSep).  One CTA per slice.  The slice is staged
// in shared memory as FP32; each pair's bin is first found in FP32 and, only
// when the FP32 quotient lies within an edge's width of a bin's end, recomputed from the
// FP64 positions exactly as the reference does, so every count is the
// reference's.  Error of the FP32 quotient x = |r| / dSep, dSep = sqrt(3) L / 100:
// a position (|r_d| <= L/2) rounds by at most 2^-25 L, the difference of two
// and its image by twice that each, so |r| is off by at most sqrt(3) 3 2^-24 L,
// 1.8e-5 of a bin; the sum of squares, the reciprocal root and 1/dSep add
// 2e-5 at 50 bins, the step of the quotient 8e-6: together less than half of
// the edge, kSepEdge steps.  In a box that is no cube the first part grows with
// the longer sides over the third, which the bins are made of, and the edge
// with it; a slice with a bead beyond a side's length from the origin takes the
// FP64 form throughout.  The FP64 recomputation
// runs for 2e-4 of the pairs in a cube; its sixty dependent FP64 instructions take a
// warp about 5 us (the FP64 pipe takes 64 clocks of a sub-partition for a warp
// instruction), so these pairs are listed and done together at the end, one a
// thread.  A shared-memory atomic takes about a clock a lane even without
// conflicts (30 us a call), so every lane of every warp counts in its own
// column with plain loads and stores.  What is left is the issue rate, about
// 45 instructions a pair, and sixteen warps a CTA against their latency.
// 256 beads, 250 slices: 43 us with eight warps, an atomic histogram each and
// floor, compare and IEEE root in floating point (64 instructions), 27 us
// here.
constexpr int kSepBits = 16;                 // 127 bins of 2^16 steps fill the mantissa
constexpr int kSepEdge = 7;                  // 1.07e-4 of a bin, in a cube
constexpr int kSepBlock = 512;               // 256 where a slice leaves no room for sixteen histograms
constexpr int kSepNear = 512;

// FP32 constants made on the host: a division or conversion in FP64 by every
// warp of every CTA takes longer than the pairs of a small slice
struct SepF { float side[3], inv[3], step, far; int edge; };

__device__ __forceinline__ int sep_bin64(const PathView& v, int t, int b1, int b2, double dSep) {
    const double3 d = sep64(v, t, b2, b1);
    return (int)(sqrt(d.x * d.x + d.y * d.y + d.z * d.z) / dSep);
}

__global__ void __launch_bounds__(kSepBlock)
k_sep_hist(PathView v, SepF f, int t0, double dSep, unsigned* __restrict__ arrived,
           unsigned long long* __restrict__ hist, unsigned long long* __restrict__ out) {
    extern __shared__ float4 sp[];                       // [n] slice positions, FP32
    __shared__ int2 near_pair[kSepNear];
    __shared__ int s_near;
    if (threadIdx.x == 0) s_near = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, threads = blockDim.x, warps = threads >> 5;
    unsigned* counts = reinterpret_cast<unsigned*>(sp + v.Ne);      // [warp][bin][lane]
    unsigned* own = counts + warp * (32 * kPcfBins) + lane;
    for (int b = threadIdx.x; b < warps * 32 * kPcfBins; b += threads) counts[b] = 0u;
    const int t = t0 + blockIdx.x;
    const int n = v.nbs[t];
    bool out_of_box = false;
    for (int j = threadIdx.x; j < n; j += threads) {
        const float4 r = v.pos32[(size_t)t * v.Ne + j];
        sp[j] = r;
        out_of_box |= fabsf(r.x) > f.side[0] || fabsf(r.y) > f.side[1] || fabsf(r.z) > f.side[2];
    }
    const int edge = __syncthreads_or(out_of_box) ? 1 << (kSepBits - 1) : f.edge;
    const float Lx = f.side[0], Ly = f.side[1], Lz = f.side[2], Lix = f.inv[0], Liy = f.inv[1], Liz = f.inv[2];
    const float step = f.step, far = f.far;
    for (int b1 = warp; b1 < n - 1; b1 += warps) {
        const float4 r1 = sp[b1];
        for (int b2 = b1 + 1 + lane; b2 < n; b2 += 32) {
            const float4 r2 = sp[b2];
            float dx = r2.x - r1.x, dy = r2.y - r1.y, dz = r2.z - r1.z;
            dx = fmaf(-Lx, rint_add(dx * Lix), dx);
            dy = fmaf(-Ly, rint_add(dy * Liy), dy);
            dz = fmaf(-Lz, rint_add(dz * Liz), dz);
            const float rr = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            float ri;
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ri) : "f"(fmaxf(rr, 1.0e-30f)));
            // x with kSepBits fraction bits in the mantissa of 2^23 + x 2^kSepBits
            const int i = __float_as_int(fmaf(fminf(rr * ri, far), step, 8388608.0f));
            if (((i + edge) & ((1 << kSepBits) - 1)) < 2 * edge) {
                const int at = atomicAdd(&s_near, 1);
                if (at < kSepNear) { near_pair[at] = make_int2(b1, b2); continue; }
                const int nR = sep_bin64(v, t, b1, b2, dSep);
                if (nR >= 0 && nR < kPcfBins) ++own[32 * nR];
                continue;
            }
            const int nR = (i >> kSepBits) & 127;
            if (nR < kPcfBins) ++own[32 * nR];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < min(s_near, kSepNear); k += threads) {
        const int nR = sep_bin64(v, t, near_pair[k].x, near_pair[k].y, dSep);
        if (nR >= 0 && nR < kPcfBins) ++own[32 * nR];
    }
    __syncthreads();
    for (int b = warp; b < kPcfBins; b += warps) {
        unsigned int c = 0;
        for (int w = 0; w < warps; ++w) c += counts[(w * kPcfBins + b) * 32 + lane];
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(&hist[b], (unsigned long long)c);
    }
    // the last slice hands the counts over and leaves zeros for the next call
    if (last_to_arrive(arrived, gridDim.x) && threadIdx.x < kPcfBins) out[threadIdx.x] = atomicExch(&hist[threadIdx.x], 0ull);
}

cudaError_t launch_sep_hist(const PathView& v, int slice, unsigned* d_arrived, unsigned long long* d_hist,
                            unsigned long long* out, cudaStream_t s) {
    const double dSep = 0.5 * sqrt(3.0) * v.side[2] / (1.0 * kPcfBins);   // action.cpp:192
    const int t0 = slice >= 0 ? slice : 0, nt = slice >= 0 ? 1 : v.M;
    const size_t pos = (size_t)v.Ne * sizeof(float4), column = kPcfBins * sizeof(unsigned);
    // small slices, more than two CTAs an SM: clearing and adding sixteen
    // histograms is the time (17 beads, 1000 slices: 34 us a call, 31 with eight)
    const bool small = v.Ne <= 32 && nt > 2 * 152;
    const int threads = !small && pos + kSepBlock * column <= 200 * 1024 ? kSepBlock : 256;
    const size_t smem = pos + threads * column;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;   // one slice in shared memory
    {
        const cudaError_t ae = set_smem_limit(k_sep_hist, 200 * 1024);
        if (ae != cudaSuccess) return ae;
    }
    SepF f;
    for (int d = 0; d < 3; ++d) { f.side[d] = (float)v.side[d]; f.inv[d] = (float)v.sideInv[d]; }
    f.step = (float)((1 << kSepBits) / dSep);
    f.far = (float)(127.0 * dSep);
    // 1.18 steps of 2^-16 a unit of |L| / (sqrt(3) L_z), and 1.83; more than twice that
    const double longer = sqrt((v.side[0] * v.side[0] + v.side[1] * v.side[1] + v.side[2] * v.side[2]) / 3.0) / v.side[2];
    f.edge = std::max(kSepEdge, (int)std::min<double>(1 << (kSepBits - 1), ceil(2.72 * longer + 4.2)));
    k_sep_hist<<<nt, threads, smem, s>>>(v, f, t0, dSep, d_arrived, d_hist, out);
    return cudaGetLastError();
}

// Winding and area sums of SuperfluidFractionEstimator::accumulate
// (estimator.cpp:2008-2036): W = sum of getVelocity over the active beads
// (path.h:189-203), Az and I from each bead and its next one.  Partial sums
// per CTA in a fixed order; the last CTA adds the partials, a warp a sum, in
// a fixed order, so the result does not depend on scheduling.  A launch of its
// own for that, one thread a sum, took as long as the partials (12 us of 21).
__global__ void __launch_bounds__(kEstBlock)
k_winding(PathView v, unsigned* __restrict__ arrived, double* __restrict__ part, double* __restrict__ out5) {
    __shared__ double red[5][kEstBlock / 32];
    double w[5] = {};
    const size_t nb = (size_t)v.M * v.Ne;
    const unsigned Ne = v.Ne;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (size_t idx = blockIdx.x * kEstBlock + threadIdx.x; idx < nb; idx += gridDim.x * kEstBlock) {
        const unsigned t = (idx >> 32) ? (unsigned)(idx / Ne) : (unsigned)idx / Ne;
        const unsigned p = (unsigned)(idx - (size_t)t * Ne);
        if (p >= (unsigned)v.nbs[t]) continue;
        const int2 nx = v.next[idx];
        if (nx.x < 0) continue;                              // getVelocity = 0, no area term
        const double* X = v.pos + (size_t)t * 3 * Ne;
        const double* Y = v.pos + (size_t)nx.x * 3 * Ne;
        const double p1x = X[p], p1y = X[Ne + p], p1z = X[2 * Ne + p];
        const double p2x = Y[nx.y], p2y = Y[Ne + nx.y], p2z = Y[2 * Ne + nx.y];
        w[0] += min_image(p2x - p1x, v.side[0], v.sideInv[0]);
        w[1] += min_image(p2y - p1y, v.side[1], v.sideInv[1]);
        w[2] += min_image(p2z - p1z, v.side[2], v.sideInv[2]);
        w[3] += p1x * p2y - p2x * p1y;
        w[4] += p1x * p2x + p1y * p2y;
    }
    #pragma unroll
    for (int k = 0; k < 5; ++k) {
        const double x = warp_sum(w[k]);
        if (lane == 0) red[k][warp] = x;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double x = 0.0;
        for (int k = 0; k < kEstBlock / 32; ++k) x += red[threadIdx.x][k];
        part[(size_t)blockIdx.x * 5 + threadIdx.x] = x;
    }
    if (!last_to_arrive(arrived, gridDim.x) || warp >= 5) return;
    double x = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) x += __ldcg(part + (size_t)b * 5 + warp);
    x = warp_sum(x);
    if (lane == 0) out5[warp] = x;
}

constexpr int kWindBlocks = 152;

size_t winding_work_bytes() { return (size_t)kWindBlocks * 5 * sizeof(double); }

cudaError_t launch_winding(const PathView& v, unsigned* d_arrived, double* d_work, double* d_out5, cudaStream_t s) {
    const size_t nb = (size_t)v.M * v.Ne;
    const int blocks = (int)std::min<size_t>(kWindBlocks, (nb + kEstBlock - 1) / kEstBlock);
    k_winding<<<blocks, kEstBlock, 0, s>>>(v, d_arrived, d_work, d_out5);
    return cudaGetLastError();
}

// Cycle lengths of PermutationCycleEstimator::accumulate
// (estimator.cpp:2735-2781): a slice-0 bead's worldline through the next links
// back to slice 0.  The reference counts a cycle at its first slice-0 bead in
// index order, i.e. at the smallest one; 0 is written for the others and -1
// where the worldline does not close.
//
// A walk is a chain of dependent loads, M a particle of the cycle (74 us at
// 124 slices, 154 us at 250, cycles of three).  Links go to the next slice, so
// a segment of kSegment slices is a map from its first slice's beads to those
// of the segment behind it: every segment and bead walks at once, the last
// CTA composes the maps into slice 0's permutation in shared memory and
// follows its cycles there: 14 and 18 us.  A link to any other slice raises `odd`
// and the last CTA walks every bead link by link.
constexpr int kSegment = 16;

__global__ void __launch_bounds__(kEstBlock)
k_cycles(PathView v, int nseg, unsigned* __restrict__ arrived, int* __restrict__ odd, int* __restrict__ map,
         int* __restrict__ len_out) {
    extern __shared__ int perm[];
    const int Ne = v.Ne, tid = threadIdx.x;
    const int seg = blockIdx.x % nseg, p0 = (blockIdx.x / nseg) * kEstBlock + tid;
    if (p0 < Ne) {
        int p = p0, t = seg * kSegment;
        const int end = min(v.M, t + kSegment);
        for (; t < end && p >= 0; ++t) {
            const int2 b = v.next[(size_t)t * Ne + p];
            if (b.x >= 0 && b.x != (t + 1 == v.M ? 0 : t + 1)) { *odd = 1; p = -1; }
            else p = b.x < 0 ? -1 : b.y;
        }
        map[(size_t)seg * Ne + p0] = p;
    }
    if (!last_to_arrive(arrived, gridDim.x)) return;
    const int nw = v.nbs[0];
    const bool skips = __ldcg(odd) != 0;
    __syncthreads();
    if (skips) {
        if (tid == 0) *odd = 0;                              // zero for the next call
        for (int n = tid; n < nw; n += kEstBlock) {
            const long long limit = (long long)v.M * Ne;
            int2 b = make_int2(0, n);
            long long wl = 0;
            bool smallest = true, closed = false;
            do {
                ++wl;
                if (b.x == 0 && b.y < n) smallest = false;
                b = v.next[(size_t)b.x * Ne + b.y];
                if (b.x < 0) break;                          // open worldline
                if (b.x == 0 && b.y == n) { closed = true; break; }
            } while (wl <= limit);
            len_out[n] = (closed && smallest) ? (int)wl : (closed ? 0 : -1);
        }
        return;
    }
    for (int n = tid; n < nw; n += kEstBlock) {
        int p = n;
        for (int k = 0; k < nseg && p >= 0; ++k) p = __ldcg(map + (size_t)k * Ne + p);
        perm[n] = p < nw ? p : -1;
    }
    __syncthreads();
    for (int n = tid; n < nw; n += kEstBlock) {
        int p = n, steps = 0;
        bool smallest = true;
        do {
            ++steps;
            if (p < n) smallest = false;
            p = perm[p];
        } while (p >= 0 && p != n && steps <= nw);
        len_out[n] = p != n ? -1 : smallest ? steps * v.M : 0;
    }
}

static int cycle_segments(const PathView& v) { return (v.M + kSegment - 1) / kSegment; }

size_t cycles_work_ints(const PathView& v) { return (size_t)cycle_segments(v) * v.Ne; }

cudaError_t launch_cycles(const PathView& v, int nw, unsigned* d_arrived, int* d_odd, int* d_work, int* len,
                          cudaStream_t s) {
    if (nw <= 0) return cudaSuccess;
    const int nseg = cycle_segments(v);
    k_cycles<<<nseg * ((v.Ne + kEstBlock - 1) / kEstBlock), kEstBlock, nw * sizeof(int), s>>>(v, nseg, d_arrived, d_odd,
                                                                                            d_work, len);
    return cudaGetLastError();
}

// Beads of slice 0 inside the cylinder x^2 + y^2 < maxR2: num1DParticles
// (estimator.cpp:4318-4327), one CTA, a fixed-order count.
__global__ void k_count_inside(PathView v, double maxR2, int* __restrict__ out) {
    __shared__ int red[kEstBlock];
    int c = 0;
    const int n = v.nbs[0];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double x = v.pos[j], y = v.pos[v.Ne + j];
        c += (x * x + y * y < maxR2) ? 1 : 0;
    }
    red[threadIdx.x] = c;
    __syncthreads();
    for (int o = kEstBlock / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = red[0];
}

cudaError_t launch_count_inside(const PathView& v, double maxR2, int* d_out, cudaStream_t s) {
    k_count_inside<<<1, kEstBlock, 0, s>>>(v, maxR2, d_out);
    return cudaGetLastError();
}

}  // namespace pgb
