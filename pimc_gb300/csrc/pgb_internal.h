// pgb_internal.h -- shared host/device definitions of the GB300 hot-path
// library.  Host code only sees plain pointers; kernels take a PathView.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "pimc_gb300.h"

namespace pgb {

constexpr double kEPS = 1.0e-7;   // include/common.h:89 (EPS)
constexpr int kXXX = -1;          // include/common.h:93 (XXX)

// Aziz HFD-HE2 parameters (src/potential.cpp:1749-1788)
struct AzizParams {
    double rm, A, epsilon, alpha, beta, D, C6, C8, C10;
};
AzizParams aziz_params(int year);
// message returned by pgb_last_error(NULL) on this host thread
void set_global_error(const std::string& msg);
// Raise func's dynamic shared-memory limit to bytes on the current device.
// The attribute belongs to the device's context, so it is set once per
// (kernel, device) pair, under a process-wide lock, and its return code is
// passed back; a failure is not recorded, so the next call tries again.
cudaError_t set_smem_limit(const void* func, int bytes);
template <class F>
cudaError_t set_smem_limit(F* func, int bytes) { return set_smem_limit(reinterpret_cast<const void*>(func), bytes); }
// Prefer a shared-memory carveout of `percent` (0..100) of the SM's unified
// L1/shared storage for func on the current device, once per (kernel, device)
cudaError_t set_carveout(const void* func, int percent);
template <class F>
cudaError_t set_carveout(F* func, int percent) { return set_carveout(reinterpret_cast<const void*>(func), percent); }

// Host memory that kernels read and write directly: a call's small inputs and
// results go through it without copies of their own (a copy each way takes a
// launch-to-result round trip from 9.7 to 16.7 us on a GB300, whose C2C link
// serves such accesses at memory speed).  A block of kStageBytes holds a ring
// for inputs and room for one call's results.  Blocks are pinned once and kept
// for the next handle, at most kPinnedKept of them: pinning one takes 100 us.
constexpr size_t kRingBytes = 256 * 1024, kResultBytes = 256 * 1024, kStageBytes = kRingBytes + kResultBytes;
constexpr int kPinnedKept = 8;
void* pinned_acquire();          // a block, or nullptr
void pinned_release(void* block);

struct Staging {
    char* block = nullptr;
    size_t at = 0;
    char* result() const { return block + kRingBytes; }
    // Room for `bytes` of input until the stream is waited for; nullptr when it
    // is too large (copy instead).  Waits for the stream where the ring wraps.
    char* take(size_t bytes, cudaStream_t s) {
        bytes = (bytes + 255) & ~(size_t)255;
        if (!block || bytes > kRingBytes / 2) return nullptr;
        if (at + bytes > kRingBytes) {
            if (cudaStreamSynchronize(s) != cudaSuccess) return nullptr;   // the caller's next call reports it
            at = 0;
        }
        char* p = block + at;
        at += bytes;
        return p;
    }
};

// Read-only view of one path handed to kernels by value.
struct PathView {
    int M, Ne;
    double side[3], sideInv[3];
    double rc2;
    // FP64 positions, slice-major SoA: x at pos[(s*3+0)*Ne + p]
    const double* pos;
    const float4* pos32;        // FP32 mirror [M][Ne] (w unused)
    const int2* next;           // [M][Ne] (slice, ptcl)
    const int2* prev;
    const uint8_t* on;          // [M][Ne]
    const int* nbs;             // numBeadsAtSlice [M]
    int worm[8];                // head, tail, special1, special2
    // FP64 direct-lookup tables
    const double* tV;
    const double* tdV;
    const double* td2V;
    double dr;
    int tableLength;
};

struct Ctx {
    pgb_params p{};
    AzizParams az{};
    cudaStream_t stream = nullptr;
    std::string err;
    int M = 0, Ne = 0;
    // tables
    double dr = 0, tailV = 0, maxSep = 0;
    int tableLength = 0;
    double *d_tV = nullptr, *d_tdV = nullptr, *d_td2V = nullptr;
    // path
    double* d_pos = nullptr;      // SoA [M][3][Ne]
    float4* d_pos32 = nullptr;
    int2 *d_next = nullptr, *d_prev = nullptr;
    uint8_t* d_on = nullptr;
    int* d_nbs = nullptr;
    std::vector<int> h_nbs;
    std::vector<int32_t> h_next, h_prev;   // host copies for range walks
    std::vector<uint8_t> h_on;
    int worm[8] = {-1,-1,-1,-1,-1,-1,-1,-1};
    int numBeadsOn = 0;
    bool loaded = false;
    Staging stage;
    unsigned long long* d_hist = nullptr;   // g(r) counts and the cycles' flag, zero between calls
    // scratch (grown on demand)
    void* d_scratch = nullptr; size_t scratch_bytes = 0;
    void* d_tc_tables = nullptr;   // split-BF16 DFT and cosine matrices of this M (built once)
    float4* d_force32 = nullptr;   // per-bead same-slice forces of the current configuration
    bool force_valid = false;      // cleared by every position change
    int* d_trial_count = nullptr;  // counters and places of trials sorted by bead (mixed form)
    unsigned* d_arrived = nullptr; // M arrival counters of kernels whose last CTA adds up (zero between calls)
    double* d_force64 = nullptr;   // scratch of the FP64 many-bead form: slice forces [M][3][Ne]
    void* h_pinned = nullptr; size_t pinned_bytes = 0;
    // plain-form worm state: the LookupTable's per-slice lists of a single
    // grid box (their order decides swap pivots) and the Worm scalars
    std::vector<std::vector<int>> lk_hash;
    std::vector<int> lk_label;
    bool lk_valid = false;
    bool w_diag = true;
    int w_gap = -1, w_length = 0;
    double w_sep[3] = {0.0, 0.0, 0.0};
    // plain-form generator state (MT19937)
    std::vector<uint32_t> mt_state;
    int mt_left = 0, mt_pos = 0;
    bool mt_seeded = false;

    PathView view() const;
    int fail(int code, const std::string& msg) { err = msg; return code; }
    int cuda_fail(cudaError_t e, const char* where);
    int ensure_scratch(size_t bytes);
    int ensure_pinned(size_t bytes);
};

// Write the listed beads (linear index s*Ne + p) from the host mirrors
// (h_next, h_prev, h_on; positions from pos_aos [M][Ne][3]) and numBeadsAtSlice
// to the device, before any later work on the stream.
int upload_beads(Ctx& c, const int* lin, int k, const double* pos_aos);
// pgb_update_beads without its wait: new positions of the listed beads before
// any later work on the stream, the host arrays reusable at once
int queue_update_beads(Ctx& c, const int32_t* beads, const double* pos, int k);

#define PGB_CUDA(ctx, call)                                              \
    do {                                                                 \
        cudaError_t e__ = (call);                                        \
        if (e__ != cudaSuccess) return (ctx)->cuda_fail(e__, #call);     \
    } while (0)

// ---- kernel launchers (implemented in the .cu files) ----
// fp64_kernels.cu (compiled with -fmad=false: IEEE mul/add, no fusion)
cudaError_t launch_build_tables(const double* d_r, int n, AzizParams az,
                                double* tV, double* tdV, double* td2V,
                                cudaStream_t s);
cudaError_t launch_potential_batch64(const PathView& v, const double* d_sep,
                                     double* d_out, int n, int what,
                                     cudaStream_t s);
// `whole`: the cutoff takes in every separation, so a bead's list is its whole
// slice; d_force: room for the FP64 slice forces [M][3][Ne], needed by the
// many-bead form of an action with a gradient term
cudaError_t launch_bead_actions64(const PathView& v, const int2* d_beads, int k,
                                  int shift, int mode, double tau, double lambda,
                                  const double vf[2], const double gf[2],
                                  const double* d_over, double* d_force, bool whole,
                                  double* d_out, cudaStream_t s);
// U(d_over) - U(current) of every bead in one launch, for whole lists; false
// when a slice is too large for it
bool launch_trial_actions64(const PathView& v, const int2* d_beads, int k, int shift, int mode,
                            double tau, double lambda, const double vf[2], const double gf[2],
                            const double* d_over, double* d_force, double* d_out, cudaStream_t s,
                            cudaError_t* e);
// What a slice's terms are asked for: nothing of its pairs, their potential,
// with forces (g2, r1, d1), with the T matrix (r2, d2)
enum { kSliceNone = -1, kSliceV = 0, kSliceF = 1, kSliceT = 2 };
// d_terms: the result [8][M]; d_work: slice_terms64_work(v) bytes; d_arrived: M
// counters, zero between calls; window <= 0: no r1, r2, d1, d2, xch
size_t slice_terms64_work(const PathView& v);
cudaError_t launch_slice_terms64(const PathView& v, int window, int even, int odd, unsigned* d_arrived,
                                 void* d_work, double* d_terms, cudaStream_t s);
// maxR2 > 0: only beads with x^2 + y^2 < maxR2 (cylinder estimators)
cudaError_t launch_rhoq64(const PathView& v, const double* d_q, int nq,
                          double* d_rho /* [q][M][2] */, cudaStream_t s, double maxR2 = 0.0);
cudaError_t launch_isf_direct64(const double* d_rho, int nq, int M, double norm,
                                double* d_out, cudaStream_t s);
// mixed_kernels.cu (FP32 pairs, FP64 accumulation)
cudaError_t launch_bead_actions32(const PathView& v, AzizParams az,
                                  const int2* d_beads, int k, int shift, int mode,
                                  double tau, double lambda, const double vf[2],
                                  const double gf[2], const double* d_over, double* d_out,
                                  cudaStream_t s, const float4* d_force = nullptr);
// one warp per bead, every active same-slice bead in the list; delta = 1 with
// d_over writes U(trial) - U(current)
cudaError_t launch_bead_actions32_full(const PathView& v, AzizParams az, const int2* d_beads, int k,
                                       int shift, int mode, double tau, double lambda,
                                       const double vf[2], const double gf[2], const double* d_over,
                                       const float4* d_force, int delta, double* d_out,
                                       cudaStream_t s);
// trials sorted by bead, for whole lists and enough trials a bead
// (trials32_sorted): d_count 2 M Ne + 2 ints, d_sorted k records
bool trials32_sorted(const PathView& v, int k);
cudaError_t launch_trials32(const PathView& v, AzizParams a, const int2* d_beads, int k, int shift, int mode, double tau,
                            double lambda, const double vf[2], const double gf[2], const double* d_pos,
                            const float4* d_force, int* d_count, float4* d_sorted, double* d_out, cudaStream_t s);
// F[t][b] = sum over active b3 != b of gradV(r_b - r_b3) on slice t, FP32 [M][Ne]
cudaError_t launch_slice_forces32(const PathView& v, AzizParams az, float4* d_force, cudaStream_t s);
// as launch_slice_terms64, with slice_terms32_work(v) bytes
size_t slice_terms32_work(const PathView& v);
cudaError_t launch_slice_terms32(const PathView& v, AzizParams az, int window, int even, int odd, unsigned* d_arrived,
                                 void* d_work, double* d_terms, cudaStream_t s);
cudaError_t launch_pos32_from64(const PathView& v, float4* d_pos32,
                                cudaStream_t s);
// scatter.cu
// d_work: rhoq32_work_bytes(v, nq) of scratch, 16-byte aligned, for the slices
// as box fractions and the wave vectors in turns.  With `split` the densities
// go there, as the tensor-core F(q,tau)'s split operand, and not to d_rho.
struct IsfOperand;
size_t rhoq32_work_bytes(const PathView& v, int nq);
cudaError_t launch_rhoq32(const PathView& v, const double* d_q, int nq, float2* d_rho /* [q][M] */,
                          void* d_work, cudaStream_t s, double maxR2 = 0.0, const IsfOperand* split = nullptr);
cudaError_t launch_ssf_from_rho32(const float2* d_rho, int nq, int M,
                                  double norm, double* d_out, cudaStream_t s);
cudaError_t launch_ssf_from_rho64(const double* d_rho, int nq, int M,
                                  double norm, double* d_out, cudaStream_t s);
cudaError_t launch_isf_direct32(const float2* d_rho, int nq, int M, double norm,
                                double* d_out, cudaStream_t s);
// path_estimators.cu (g(r), winding, permutation cycles; FP64, -fmad=false)
// d_hist: 50 counts, zero between calls; the result goes to out
cudaError_t launch_sep_hist(const PathView& v, int slice, unsigned* d_arrived, unsigned long long* d_hist,
                            unsigned long long* out, cudaStream_t s);
size_t winding_work_bytes();
// d_arrived: one counter, zero between calls
cudaError_t launch_winding(const PathView& v, unsigned* d_arrived, double* d_work, double* d_out5, cudaStream_t s);
// d_odd: a flag, zero between calls; d_work: cycles_work_ints ints; len: the nw
// cycle lengths
size_t cycles_work_ints(const PathView& v);
cudaError_t launch_cycles(const PathView& v, int nw, unsigned* d_arrived, int* d_odd, int* d_work, int* len,
                          cudaStream_t s);
// slice-0 beads with x^2 + y^2 < maxR2 (one int)
cudaError_t launch_count_inside(const PathView& v, double maxR2, int* d_out, cudaStream_t s);
// isf_tc.cu (tcgen05 split-BF16 DFT correlation)
size_t isf_tc_scratch_bytes(int nq, int M);
size_t isf_tc_table_bytes(int M);
cudaError_t isf_tc_build_tables(int M, void* d_tables, cudaStream_t s);
// the A operand of the first GEMM: Re rho | Im rho, [qpad][2M] split and
// tile-ordered, and the pipeline's error word, both set by launch_rhoq32
struct IsfOperand { __nv_bfloat16 *hi, *lo; int qpad; int* err; };
IsfOperand isf_tc_operand(int nq, int M, void* d_scratch);
cudaError_t launch_isf_tc(int nq, int M, double norm, double* d_out, void* d_scratch, const void* d_tables,
                          cudaStream_t s);
bool isf_tc_supported(int M);
// the pipeline's error word (int, 0 or 1) at this offset of the scratch
size_t isf_tc_error_offset(int nq, int M);
// test switch: the first GEMM of later calls stalls before its last chunk
void isf_tc_set_stall_test(int on);

}  // namespace pgb

struct pgb_ctx { pgb::Ctx c; };
