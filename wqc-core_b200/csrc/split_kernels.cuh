// Kernel entry points of the two-site split pipeline and the site kernels.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"

namespace wqc {

enum { kStageY0 = 0, kStageZ = 1, kStageY = 2, kStageB = 3 };
// Jacobi / finalize modes: the range finder's B^H; theta of a split that takes
// the exact path from the start; theta of a range-finder split that fell back.
enum { kJacobiRsvd = 0, kJacobiExact = 1, kJacobiFallback = 2 };
// The cluster Jacobi (jacobi_ring.cu) stores a column as `kr` groups of 32
// rows, one row of each group per lane, and is compiled for these counts: the
// columns of W in the plain form, W's rows and under them V's (each from a
// whole group on) in the precision form's first phase.  0: no instance.
constexpr int jacobi_ring_kr(bool fp32, int M, int vrows) {
    const int need = (M + 31) / 32 + (vrows + 31) / 32;
    if (fp32) return need <= 2 ? 2 : need <= 4 ? 4 : need <= 8 ? 8 : need <= 16 ? 16 : need <= 24 ? 24 : 0;
    return need <= 4 ? (need < 1 ? 1 : need) : need <= 6 ? 6 : need <= 8 ? 8 : need <= 12 ? 12 : 0;
}
// Warps of its largest CTA, one per column of a block: what 64 Ki registers
// hold of two columns' rows per lane and about 70 registers besides.
constexpr int jacobi_ring_warps(int kr, int elem) { return 2 * kr * elem / 4 + 70 <= 128 ? 16 : 12; }
// QR before the Jacobi (jacobi_qr.cu): instances by row groups, columns a CTA
// holds at a time, and the tasks it takes -- from 16 columns (one SVD of 8 columns took 43 us
// without and 56 with it, of 16 columns 125 and 101, of 32 385 and 220) to the
// rows an instance holds.
constexpr int kJacobiQrMin = 16, kJacobiQrMax = 512, kJacobiQrPerCta = 16;
constexpr int jacobi_qr_kr(int M) {
    const int need = (M + 31) / 32;
    return need <= 2 ? (need < 1 ? 1 : need) : need <= 4 ? 4 : need <= 6 ? 6 : need <= 8 ? 8 : need <= 12 ? 12 : 16;
}
inline bool jacobi_qr_takes(int M, int N) { return N >= kJacobiQrMin && M <= kJacobiQrMax; }
cudaError_t jacobi_qr_attributes();  // of every instance, once per process
cudaError_t launch_jacobi_qr(int kr, int C, int tasks, cudaStream_t stream, const SplitJob* jobs, SplitState* st,
                             const SlotBuffers* slots, const int* idx, int mode, int* status);
constexpr int kJacobiRingMaxCluster = 16;
// Entry of a launch's task list: the job in the wave and log2 of the number
// of CTAs it runs on.
constexpr int kJacobiEntryShift = 24;
__host__ __device__ inline int jacobi_entry(int job, int log2_c) { return job | (log2_c << kJacobiEntryShift); }
__host__ __device__ inline int jacobi_entry_job(int e) { return e & ((1 << kJacobiEntryShift) - 1); }
__host__ __device__ inline int jacobi_entry_cluster(int e) { return 1 << (e >> kJacobiEntryShift); }
constexpr int kJacobiStagedThreads = 512;

__global__ void prepare_kernel(const SplitJob* jobs, SplitState* st, int njobs, DeviceMps mps);
__global__ void merge_gate_kernel(const SplitJob* jobs, SplitState* st, const SlotBuffers* slots,
                                  DeviceMps mps);
__global__ void omega_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots);
__global__ void rsvd_gemm_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots, int stage);
__global__ void householder_qr_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots);
constexpr int kQrClusterThreads = 256;
constexpr int kQrRowsPerThread = 8;  // rows of one reflector each thread holds: Y of at most 2048 rows
// The cluster Householder QR (columns in shared memory, or with global_cols
// in the slot's Y and Q buffers), reached through these host functions.
const void* qr_cluster(bool global_cols);
cudaError_t launch_qr_cluster(bool global_cols, const cudaLaunchConfig_t& cfg, const SplitJob* jobs,
                              const SplitState* st, const SlotBuffers* slots);
// Shared memory of the cluster QR for an m x n Y on a cluster of C CTAs.
inline size_t qr_cluster_smem_bytes(int m, int n, int C, bool global_cols = false) {
    const int cpc = (n + C - 1) / C;
    return ((global_cols ? size_t(0) : size_t(2) * cpc * m) + size_t(3) * m + cpc) * sizeof(double2);
}
// Phases of a Jacobi SVD: the plain one; the precision form's first phase
// (complex64 columns carrying W = X V and the accumulated V, written out as
// FP64 for the finish); and its finishing phase (FP64 sweeps that start from
// X V, formed in FP64 by precond_gemm_kernel).
enum { kPhasePlain = 0, kPhaseFp32V = 1, kPhaseFinish = 2 };
// The cluster Jacobi: every instance (for the kernel attributes) and a launch
// of the one for kr row groups, on clusters of the largest size in the list.
std::vector<const void*> jacobi_ring_kernels();
cudaError_t launch_jacobi(bool fp32, int kr, const cudaLaunchConfig_t& cfg, const SplitJob* jobs, SplitState* st,
                          const SlotBuffers* slots, const int* idx, int mode, int phase, int max_sweeps, int* status,
                          unsigned long long* counters);
// The staged variant for working matrices beyond a cluster's shared memory:
// columns in the slot's `gs` workspace, blocks of b columns (b even).
const void* jacobi_staged(bool fp32);
cudaError_t launch_jacobi_staged(bool fp32, const cudaLaunchConfig_t& cfg, const SplitJob* jobs, SplitState* st,
                                 const SlotBuffers* slots, const int* idx, int mode, int phase, int max_sweeps, int b,
                                 int* status, unsigned long long* counters);
// The precision form's FP64 products between its two Jacobi phases, for the
// jobs active in `mode`, in stage order: G = V^H V and V <- V (3 I - G) / 2
// twice (Newton-Schulz: V^H V - I goes from ~1e-6 after the complex64
// rotations to ~1e-12, then to FP64 rounding), then X V into the slot's W
// buffer, X dust-zeroed as the first phase loaded it.
enum { kPrecondGram1 = 0, kPrecondStep1, kPrecondGram2, kPrecondStep2, kPrecondXV, kPrecondStages };
constexpr int kPrecondTile = 32;  // of waves that fill the device (kSmall: kTile)
template <bool kSmall>
__global__ void precond_gemm_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots, int mode,
                                    int stage);
// Shape of the staged Jacobi for an M x N working matrix on a cluster of C
// CTAs: the block width b <= 16 whose two blocks fit `smem_limit` and whose
// sweep is shortest, counted in dependent rotation rounds: (2K-1) steps of
// ceil(K / C) block pairs per CTA, b rounds each, K = ceil(N / 2b) pairs.
// 0 if none fits.  Also returns the shared memory of that choice.
inline int jacobi_staged_b(int M, int N, size_t elem, size_t smem_limit, size_t* smem, int C = 16) {
    int best = 0;
    long best_rounds = 0;
    size_t best_bytes = 0;
    for (int b = 2; b <= 16; ++b) {
        const int K = (N + 2 * b - 1) / (2 * b);
        const size_t len = size_t(M);
        const size_t bytes = size_t(2) * b * len * elem;
        if (bytes > smem_limit) continue;
        const long rounds = long(2 * K - 1) * ((K + C - 1) / C) * b;
        if (!best || rounds < best_rounds) {
            best = b;
            best_rounds = rounds;
            best_bytes = bytes;
        }
    }
    if (best && smem) *smem = best_bytes;
    return best;
}
// Elements (double2) of the `gs` workspace for two-site matrices up to R x R.
inline size_t jacobi_staged_elems(int R) { return size_t(R + 32) * size_t(R); }
// Probe-vector factorisation check of every active Jacobi task (grid: jobs x 2).
constexpr int kProbeThreads = 1024;
__global__ void svd_probe_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots, int mode,
                                 int fp32, int* status);
// noise_rel: singular values below noise_rel * (largest) count as zero (0 in
// the plain form; the precision form's FP32 rounding level).
__global__ void finalize_kernel(const SplitJob* jobs, SplitState* st, const SlotBuffers* slots, int mode,
                                int chi_max, double noise_rel, wqc_split_info* records, int* status);
enum { kRecoverBW = 0, kRecoverQT = 1, kRecoverExact = 2 };
__global__ void recover_gemm_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots,
                                    DeviceMps mps, int stage);
__global__ void cut_kernel(const SplitJob* jobs, SplitState* st, const SlotBuffers* slots, DeviceMps mps, int tiles,
                           int tiles_n, int chi_max, double noise_rel, wqc_split_info* records, int* status);
__global__ void absorb_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots,
                              DeviceMps mps);

// Site kernels (site_kernels.cu).
struct OneQubitOp {
    int site;
    int first;  // first gate in the 2x2 array
    int count;  // gates applied in order
};
__global__ void apply_1q_kernel(const OneQubitOp* ops, const double2* mats, DeviceMps mps);
__global__ void amplitude_zero_kernel(DeviceMps mps, const int* seg, double2* out);
__global__ void reset_sites_kernel(DeviceMps mps);
__global__ void site_envs_kernel(DeviceMps mps, double2* envL, double2* envR, int lfrom, int lto, int rfrom, int rto,
                                 const int* targets, int count, double2* out);
__global__ void dense_step_kernel(const double2* cur, const double2* site, int l, int r, long prefix, int prune,
                                  double2* nxt);
__global__ void pauli_expectation_kernel(DeviceMps mps, const char* labels, int nterms, double2* scratch,
                                         int env_cap, double2* out);
__global__ void overlap_half_kernel(const double2* env, int kl, int bl, const double2* ket, int kr, double2* tmp);
__global__ void overlap_next_kernel(const double2* tmp, int bl, int kr, const double2* bra, int br, double2* next);
// Environments (env_kernels.cu).  The identity chains of `nseg` runs of
// `width` sites (firsts[seg] ..), each with its buffers seg_stride entries
// apart: T (2 cap^2 a site), L (two of cap^2), R (cap^2 a site; R_q contracts
// the sites right of q) and H (2 cap^2).  `left` false: the right chain only;
// then R may lie at offsets of its own, r_at[q], a site's no larger than its
// bonds.
struct EnvChains {
    double2* base;
    size_t seg_stride, t_off, l_off, r_off, h_off;
    const unsigned long long* r_at;
    const int* firsts;
    int nseg, width, cap;
    bool left;
};
// Pauli terms: labels (term t's character width-1-q acts on site q), the first
// site that is not the identity and the number of sites from it to the last
// such one; `work`: 4 cap^2 entries per segment and term of a launch.
struct EnvTerms {
    const char* labels;
    const int* start;
    const int* span;
    double2* work;
};
// Both return the number of kernels launched; `bond` bounds every bond.
int launch_env_chains(const DeviceMps& mps, const EnvChains& ch, bool right, int bond, cudaStream_t stream);
int launch_env_terms(const DeviceMps& mps, const EnvChains& ch, const EnvTerms& tm, int t0, int count, int nterms,
                     int longest, int bond, double2* out, cudaStream_t stream);
template <bool kPacked>
__global__ void sample_shots_kernel(DeviceMps mps, const double2* envs, const unsigned long long* env_at,
                                    const int* bitpos, unsigned long long seed, int shots, unsigned long long* out);

// Adjoint kernels (adjoint_kernels.cu).
struct Adj1q {
    double2 u[4];   // the gate, row-major
    double2 du[4];  // d u / d angle (rotations)
    int has_du;
    int slot;       // gradient slot of this gate instance
    double2* bar;   // cotangent of its site
    const double2* before;  // the site before the gate, from the tape
    const int* dims;        // its bonds
};
// One recomputed operation on the tape, and where the parts of a two-site one
// lie from its base: both sites before it, then theta, W, sigma, perm and the
// split's state after it.  A one-qubit gate has its site and its bonds.
struct AdjTape {
    char* base;
    int site;
};
struct AdjTapeLayout {
    size_t site_b, theta_off, w_off, sigma_off, perm_off, state_off;
};
// One split of the reverse sweep: the tape's copies of its forward inputs
// and outputs, the cotangent sites it updates, and the workspace matrices
// (column-major, leading dimension R = 2 chi_max).
struct AdjSplit {
    const SplitState* st;
    const double2* theta;   // rows x cols, row-major
    const double2* w;       // Jacobi W, M x N column-major
    const double* sigma;    // N
    const int* perm;        // N: sorted position -> column
    const double2* site_l;  // site p before the split: [dl][2][k]
    const double2* site_r;  // site p+1 before the split: [k][2][dr]
    double2* bar_l;         // cotangent of site p
    double2* bar_r;         // cotangent of site p+1
    double2 u[16];          // effective 4x4 of the gate on theta
    double2 *U, *V, *Ub, *Vb, *M, *Nm, *Z, *T1, *tb, *tb0;
    double *inv, *sq;
    int R;
};
enum { kAdjStageOther = 0, kAdjStageM, kAdjStageN, kAdjStageT1, kAdjStageTb, kAdjStageTb2, kAdjStageBarL,
       kAdjStageBarR };
__global__ void adj_pauli_envs_kernel(DeviceMps mps, const char* labels, int cap, int dirs, int dir, int step, int phase,
                                      double2* envs, double2* tmp_all);
__global__ void adj_pauli_holes_kernel(DeviceMps mps, const char* labels, int t0, int cap, int phase,
                                       const double2* envs, double2* tmp_all, double2* holes);
__global__ void adj_pauli_values_kernel(const double2* envs, int n, int cap, int nterms, double2* vals);
__global__ void adj_pauli_accumulate_kernel(DeviceMps mps, double2* const* bars, const double2* holes,
                                            const double* coef_re, int t0, int count, int cap, int first);
__global__ void adj_one_qubit_kernel(const Adj1q* gates, double* grad);
__global__ void adj_tape_before_kernel(DeviceMps mps, const AdjTape* ops, AdjTapeLayout L, int two);
__global__ void adj_tape_after_kernel(const SplitState* states, const SlotBuffers* slots, const AdjTape* ops,
                                      AdjTapeLayout L);
__global__ void adj_split_prep_kernel(const AdjSplit* splits);
__global__ void adj_split_gemm_kernel(const AdjSplit* splits, int stage);
__global__ void adj_split_assemble_kernel(const AdjSplit* splits);
__global__ void adj_split_gate_kernel(const AdjSplit* splits);

// Shared memory of a CTA of the cluster Jacobi: two blocks of b columns.
inline size_t jacobi_ring_smem(int b, int kr, size_t elem) { return size_t(2) * b * 32 * kr * elem; }

}  // namespace wqc
