// Two-site split pipeline: merge + 4x4 gate, range finder (reference rule),
// one-sided Jacobi SVD in a thread-block cluster, cut, and sqrt(S) absorption.
//
// Reference path: src/tn/mps.rs:377-429 (two-site apply), 484-514 (merge),
// 833-866 (4x4 on theta), 937-981 (split dispatch), 983-1053 (range finder),
// 1124-1171 (truncated split), src/tn/svd_guard.rs:25-76 (truncation rule,
// ambiguity test), 91-139 (dust zeroing before the SVD).
//
// Every kernel takes the wave's job array and reads the job's bond dimensions
// from device memory, so a whole circuit can be enqueued without the host
// waiting on the device.
#include <cooperative_groups.h>

#include "common.cuh"
#include "jacobi_device.cuh"
#include "split_kernels.cuh"
#include "tile_gemm.cuh"

namespace cg = cooperative_groups;

namespace wqc {

// ---------------------------------------------------------------------------
// prepare: bond dims and the exact / range-finder decision (mps.rs:937-954).
// ---------------------------------------------------------------------------
__device__ __forceinline__ SplitState split_state(const SplitJob& J, const DeviceMps& mps) {
    SplitState s{};
    s.dl = mps.dl[J.p];
    s.dr = mps.dr[J.p + 1];
    s.k = min(mps.dr[J.p], mps.dl[J.p + 1]);
    s.rows = 2 * s.dl;
    s.cols = 2 * s.dr;
    s.ell = min(min(J.chi_max + kRsvdOversample, s.rows), s.cols);
    const unsigned long long f = (unsigned long long)s.rows * s.cols * s.ell;
    const unsigned long long side = kRsvdMinSide;
    const bool worth = f >= side * side * side;
    s.use_rsvd = (!J.reject && !J.exact_only && s.ell > 0 && s.ell < min(s.rows, s.cols) && worth) ? 1 : 0;
    s.need_exact = s.use_rsvd ? 0 : 1;
    s.path = s.use_rsvd ? WQC_SPLIT_RSVD : WQC_SPLIT_EXACT;
    s.pre_exact = J.pre & 1;
    s.pre_rsvd = (J.pre >> 1) & 1;
    // W of X = theta (rows >= cols) holds left vectors, of theta^H right ones;
    // a Jacobi on R^H gives the other side.
    s.w_rows_of_src = (s.rows < s.cols) != (s.pre_exact != 0) ? 1 : 0;
    return s;
}

// The state of a job as the wave's later kernels read it; a cancelled job is
// skipped by all of them.
__device__ __forceinline__ void publish_state(const SplitJob* jobs, SplitState* st, int j, const DeviceMps& mps) {
    SplitState s{};
    if (*mps.cancel) {
        s.skip = 1;
        if (j == 0) atomicOr(mps.status, kStatusCancelled);
    } else {
        s = split_state(jobs[j], mps);
    }
    st[j] = s;
}

__global__ void prepare_kernel(const SplitJob* jobs, SplitState* st, int njobs, DeviceMps mps) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < njobs) publish_state(jobs, st, j, mps);
}

// ---------------------------------------------------------------------------
// merge + gate: theta'[(a,s'),(t',b)] = sum_{s,t} U[s't',st] sum_g L[a,s,g] R[g,t,b]
// One thread owns one (a, b) pair and its 2x2 physical block.  L and R tiles
// are staged in shared memory.
// ---------------------------------------------------------------------------
constexpr int kMergeTA = 16, kMergeTB = 16, kMergeTK = 16;

__global__ void __launch_bounds__(256) merge_gate_kernel(const SplitJob* jobs, SplitState* st,
                                                         const SlotBuffers* slots, DeviceMps mps) {
    const int j = blockIdx.z;
    const SplitJob& J = jobs[j];
    // Every CTA derives the job's state from the bonds, and one stores it: no
    // kernel of its own before the merge.  The others merge even if that one
    // finds the job cancelled; nothing reads their theta then.
    const SplitState S = split_state(J, mps);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) publish_state(jobs, st, j, mps);
    const int a0 = blockIdx.y * kMergeTA, b0 = blockIdx.x * kMergeTB;
    if (a0 >= S.dl || b0 >= S.dr) return;
    const double2* L = mps.site[J.p];      // [dl][2][k']  with k' = dr of site p
    const double2* R = mps.site[J.p + 1];  // [k''][2][dr] with k'' = dl of site p+1
    const int ldl = mps.dr[J.p];           // row stride of L's (a,s) rows
    const int k = S.k;
    const int dr = S.dr;
    __shared__ double2 Ls[2 * kMergeTA][kMergeTK + 1];
    __shared__ double2 Rs[kMergeTK][2 * kMergeTB + 1];
    __shared__ double2 U[16];
    const int tid = threadIdx.x;
    if (tid < 16) U[tid] = J.u[tid];
    const int ta = tid / kMergeTB, tb = tid % kMergeTB;
    const int a = a0 + ta, b = b0 + tb;
    double2 acc[4] = {cmake(0, 0), cmake(0, 0), cmake(0, 0), cmake(0, 0)};  // [s][t]
    for (int g0 = 0; g0 < k; g0 += kMergeTK) {
        // L tile: rows (a0..a0+TA) x s, cols g
        for (int e = tid; e < 2 * kMergeTA * kMergeTK; e += 256) {
            const int r = e / kMergeTK, c = e % kMergeTK;
            const int aa = a0 + r / 2, ss = r % 2, gg = g0 + c;
            Ls[r][c] = (aa < S.dl && gg < k) ? L[(size_t(aa) * 2 + ss) * ldl + gg] : cmake(0, 0);
        }
        for (int e = tid; e < kMergeTK * 2 * kMergeTB; e += 256) {
            const int r = e / (2 * kMergeTB), c = e % (2 * kMergeTB);
            const int gg = g0 + r, tt = c / kMergeTB, bb = b0 + c % kMergeTB;
            Rs[r][c] = (gg < k && bb < dr) ? R[(size_t(gg) * 2 + tt) * dr + bb] : cmake(0, 0);
        }
        __syncthreads();
#pragma unroll 4
        for (int c = 0; c < kMergeTK; ++c) {
            const double2 l0 = Ls[2 * ta][c], l1 = Ls[2 * ta + 1][c];
            const double2 r0 = Rs[c][tb], r1 = Rs[c][kMergeTB + tb];
            cfma(acc[0], l0, r0);
            cfma(acc[1], l0, r1);
            cfma(acc[2], l1, r0);
            cfma(acc[3], l1, r1);
        }
        __syncthreads();
    }
    if (a >= S.dl || b >= dr) return;
    double2* th = slots[J.slot].theta;
    const int cols = S.cols;
    for (int so = 0; so < 2; ++so)
        for (int to = 0; to < 2; ++to) {
            double2 v = cmake(0, 0);
            for (int q = 0; q < 4; ++q) cfma(v, U[(so * 2 + to) * 4 + q], acc[q]);
            th[size_t(a * 2 + so) * cols + to * dr + b] = v;
        }
}

// ---------------------------------------------------------------------------
// Rademacher test matrix (mps.rs:1103-1122), generated in parallel: element i
// is the LCG state after i+1 steps from (salt | 1), reached by composing the
// affine map x -> a x + c with itself (exact 64-bit wrapping arithmetic).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long lcg_jump(unsigned long long x, unsigned long long n) {
    unsigned long long A = 1ull, Cc = 0ull;            // accumulated map
    unsigned long long a = 6364136223846793005ull, c = 1ull;  // current power
    while (n) {
        if (n & 1ull) {
            A = A * a;
            Cc = Cc * a + c;
        }
        c = c * (a + 1ull);
        a = a * a;
        n >>= 1;
    }
    return A * x + Cc;
}

__global__ void omega_kernel(const SplitJob* jobs, const SplitState* st, const SlotBuffers* slots) {
    const int j = blockIdx.y;
    const SplitState S = st[j];
    if (!S.use_rsvd) return;
    const long total = long(S.cols) * S.ell;
    const unsigned long long salt =
        ((unsigned long long)S.rows * 0x9E37ull + (unsigned long long)S.cols) * 0x9E37ull + (unsigned long long)S.ell;
    const double scale = 1.0 / sqrt(double(S.cols));
    double2* om = slots[jobs[j].slot].omega;
    for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
        const unsigned long long s = lcg_jump(salt | 1ull, (unsigned long long)i + 1ull);
        om[i] = cmake((s & 0x100ull) == 0 ? scale : -scale, (s & 0x200ull) == 0 ? scale : -scale);
    }
}

// ---------------------------------------------------------------------------
// Batched complex FP64 GEMMs of the range finder, dimensions from the job's state.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(kTileThreads) rsvd_gemm_kernel(const SplitJob* jobs, const SplitState* st,
                                                                 const SlotBuffers* slots, int stage) {
    const int j = blockIdx.z;
    const SplitState S = st[j];
    if (!S.use_rsvd) return;
    const SlotBuffers B = slots[jobs[j].slot];
    const int rows = S.rows, cols = S.cols, ell = S.ell;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int m = stage == kStageZ ? cols : stage == kStageB ? ell : rows, n = stage == kStageB ? cols : ell;
    if (m0 >= m || n0 >= n) return;
    __shared__ TileSmem sm;
    auto theta = [&](int i, int k) { return B.theta[size_t(i) * cols + k]; };
    switch (stage) {
        case kStageY0:  // Y0 = theta * Omega   (rows x ell)
            tile_gemm(sm, m0, n0, m, n, cols, true, false, theta,
                      [&](int k, int c) { return B.omega[size_t(k) * ell + c]; },
                      [&](int i, int c, double2 v) { B.y0[size_t(i) * ell + c] = v; });
            break;
        case kStageZ:  // Z = theta^H * Y0    (cols x ell)
            tile_gemm(sm, m0, n0, m, n, rows, false, false,
                      [&](int i, int k) { return cconj(B.theta[size_t(k) * cols + i]); },
                      [&](int k, int c) { return B.y0[size_t(k) * ell + c]; },
                      [&](int i, int c, double2 v) { B.zr[size_t(i) * ell + c] = v; });
            break;
        case kStageY:  // Y = theta * Z, stored column-major for the QR
            tile_gemm(sm, m0, n0, m, n, cols, true, false, theta,
                      [&](int k, int c) { return B.zr[size_t(k) * ell + c]; },
                      [&](int i, int c, double2 v) { B.y[size_t(c) * rows + i] = v; });
            break;
        default:  // kStageB: B = Q^H * theta  (ell x cols), Q column-major rows x ell
            tile_gemm(sm, m0, n0, m, n, rows, true, false,
                      [&](int i, int k) { return cconj(B.q[size_t(i) * rows + k]); }, theta,
                      [&](int i, int c, double2 v) { B.b[size_t(i) * cols + c] = v; });
            break;
    }
}

// ---------------------------------------------------------------------------
// Householder QR of Y (rows x ell, column-major) and the thin Q, one CTA per
// job (LAPACK zgeqr2 + zung2r conventions; thin Q is unique up to column
// phases, which the range finder's results do not depend on).
// ---------------------------------------------------------------------------
constexpr int kQrThreads = 512;

__device__ double block_sum(double v, double* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double t = 0;
    const int nw = blockDim.x >> 5;
    for (int w = 0; w < nw; ++w) t += red[w];  // every thread sums in the same order
    __syncthreads();
    return t;
}

__global__ void __launch_bounds__(kQrThreads) householder_qr_kernel(const SplitJob* jobs, const SplitState* st,
                                                                    const SlotBuffers* slots) {
    const int j = blockIdx.x;
    const SplitState S = st[j];
    if (!S.use_rsvd) return;
    const SlotBuffers B = slots[jobs[j].slot];
    const int m = S.rows, n = S.ell;
    double2* y = B.y;
    double2* q = B.q;
    double2* tau = B.tau;
    __shared__ double red[kQrThreads / 32];
    __shared__ double2 v[512];
    __shared__ double2 s_tau;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = kQrThreads / 32;
    for (int c = 0; c < n; ++c) {
        double2* col = y + size_t(c) * m;
        double part = 0;
        for (int i = c + 1 + tid; i < m; i += kQrThreads) part += cnorm2(col[i]);
        const double xnorm2 = block_sum(part, red);
        const double2 alpha = col[c];
        double2 t = cmake(0, 0);
        double2 sc = cmake(0, 0);
        double beta = alpha.x;
        const bool trivial = (xnorm2 == 0.0 && alpha.y == 0.0);
        if (!trivial) {
            beta = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
            if (alpha.x >= 0) beta = -beta;
            t = cmake((beta - alpha.x) / beta, -alpha.y / beta);
            // sc = 1 / (alpha - beta)
            const double2 d = cmake(alpha.x - beta, alpha.y);
            const double dn = d.x * d.x + d.y * d.y;
            sc = cmake(d.x / dn, -d.y / dn);
        }
        __syncthreads();  // everyone has read col[c]
        for (int i = c + 1 + tid; i < m; i += kQrThreads) {
            const double2 x = trivial ? col[i] : cmul(col[i], sc);
            col[i] = x;
            v[i] = x;
        }
        if (tid == 0) {
            col[c] = cmake(beta, 0.0);
            v[c] = cmake(1.0, 0.0);
            tau[c] = t;
            s_tau = t;
        }
        __syncthreads();
        if (!trivial) {
            const double2 tc = cconj(s_tau);  // apply H^H
            for (int kk = c + 1 + wid; kk < n; kk += nw) {
                double2* ck = y + size_t(kk) * m;
                double2 w = cmake(0, 0);
                for (int i = c + lane; i < m; i += 32) cfma_conj(w, v[i], ck[i]);
                for (int o = 16; o > 0; o >>= 1) {
                    w.x += __shfl_xor_sync(0xffffffffu, w.x, o);
                    w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
                }
                w = cmul(tc, w);
                for (int i = c + lane; i < m; i += 32) ck[i] = csub(ck[i], cmul(v[i], w));
            }
        }
        __syncthreads();
    }
    // Thin Q = H_0 ... H_{n-1} [I; 0], accumulated backward.
    for (int e = tid; e < m * n; e += kQrThreads) {
        const int r = e % m, c = e / m;
        q[e] = cmake(r == c ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    for (int c = n - 1; c >= 0; --c) {
        const double2* col = y + size_t(c) * m;
        for (int i = c + 1 + tid; i < m; i += kQrThreads) v[i] = col[i];
        if (tid == 0) {
            v[c] = cmake(1.0, 0.0);
            s_tau = tau[c];
        }
        __syncthreads();
        const double2 tc = s_tau;
        if (tc.x != 0.0 || tc.y != 0.0) {
            for (int kk = c + wid; kk < n; kk += nw) {
                double2* ck = q + size_t(kk) * m;
                double2 w = cmake(0, 0);
                for (int i = c + lane; i < m; i += 32) cfma_conj(w, v[i], ck[i]);
                for (int o = 16; o > 0; o >>= 1) {
                    w.x += __shfl_xor_sync(0xffffffffu, w.x, o);
                    w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
                }
                w = cmul(tc, w);
                for (int i = c + lane; i < m; i += 32) ck[i] = csub(ck[i], cmul(v[i], w));
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// The same Householder QR and thin Q on a thread-block cluster: CTA r holds
// columns [r*cpc, (r+1)*cpc) of Y and of Q in shared memory.  At step c the
// owner of column c forms the reflector, publishes v_c and tau_c in a
// double-buffered slot of its shared memory and updates its own trailing
// columns; after one cluster barrier the CTAs to its right copy v_c through
// distributed shared memory and update theirs.  Q is then accumulated
// backward with every reflector read from its owner.  Same arithmetic as the
// single-CTA kernel above.  With kGlobalCols the columns stay in the slot's
// Y and Q buffers (L2-resident) instead of shared memory, for shapes whose
// columns do not fit (Y of 512 x 272 at chi 256); only the reflector
// broadcast and the local reflector copy live in shared memory.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void reflect_columns(double2* cols, int ldc, int count, const double2* v, double2 t,
                                                int c, int m, int lane, int wid, int nw) {
    for (int kk = wid; kk < count; kk += nw) {
        double2* ck = cols + size_t(kk) * ldc;
        double2 w = cmake(0, 0);
        for (int i = c + lane; i < m; i += 32) cfma_conj(w, v[i], ck[i]);
        for (int o = 16; o > 0; o >>= 1) {
            w.x += __shfl_xor_sync(0xffffffffu, w.x, o);
            w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
        }
        w = cmul(t, w);
        for (int i = c + lane; i < m; i += 32) ck[i] = csub(ck[i], cmul(v[i], w));
    }
}

// Split cluster barrier: arrive (releasing this thread's writes) and wait
// (acquiring the others') as two steps, so a CTA can work between them.
__device__ __forceinline__ void cluster_arrive_release() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_acquire() {
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <bool kGlobalCols>
__global__ void __launch_bounds__(kQrClusterThreads, 1) qr_cluster_kernel(const SplitJob* jobs, const SplitState* st,
                                                                           const SlotBuffers* slots) {
    cg::cluster_group cluster = cg::this_cluster();
    const int C = int(cluster.num_blocks());
    const int rank = int(cluster.block_rank());
    const int j = blockIdx.x / C;
    const SplitState S = st[j];
    if (!S.use_rsvd) return;  // uniform over the cluster
    const SlotBuffers B = slots[jobs[j].slot];
    const int m = S.rows, n = S.ell;
    const int cpc = (n + C - 1) / C;
    const int c0 = min(n, rank * cpc), c1 = min(n, c0 + cpc), nloc = c1 - c0;
    extern __shared__ __align__(16) double2 qsm[];
    double2* Ys = kGlobalCols ? B.y + size_t(c0) * m : qsm;                      // cpc columns of m
    double2* Qs = kGlobalCols ? B.q + size_t(c0) * m : qsm + size_t(cpc) * m;    // cpc columns of m
    double2* bcast = kGlobalCols ? qsm : qsm + size_t(2) * cpc * m;              // 2 slots of m
    double2* vloc = bcast + size_t(2) * m;                                        // m
    double2* taus = vloc + m;                                                     // cpc local tau values
    __shared__ double red[kQrClusterThreads / 32];
    __shared__ double2 s_tau[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = kQrClusterThreads / 32;
    if (!kGlobalCols)
        for (int e = tid; e < nloc * m; e += kQrClusterThreads) Ys[e] = B.y[size_t(c0) * m + e];
    __syncthreads();
    for (int c = 0; c < n; ++c) {
        const int owner = c / cpc;
        const int slot = c & 1;
        if (rank == owner) {
            double2* col = Ys + size_t(c - c0) * m;
            double part = 0;
            for (int i = c + 1 + tid; i < m; i += kQrClusterThreads) part += cnorm2(col[i]);
            const double xnorm2 = block_sum(part, red);
            const double2 alpha = col[c];
            double2 t = cmake(0, 0), sc = cmake(0, 0);
            double beta = alpha.x;
            const bool trivial = (xnorm2 == 0.0 && alpha.y == 0.0);
            if (!trivial) {
                beta = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
                if (alpha.x >= 0) beta = -beta;
                t = cmake((beta - alpha.x) / beta, -alpha.y / beta);
                const double2 d = cmake(alpha.x - beta, alpha.y);
                const double dn = d.x * d.x + d.y * d.y;
                sc = cmake(d.x / dn, -d.y / dn);
            }
            __syncthreads();
            double2* bv = bcast + size_t(slot) * m;
            for (int i = c + 1 + tid; i < m; i += kQrClusterThreads) {
                const double2 x = trivial ? col[i] : cmul(col[i], sc);
                col[i] = x;
                bv[i] = x;
            }
            if (tid == 0) {
                col[c] = cmake(beta, 0.0);
                bv[c] = cmake(1.0, 0.0);
                taus[c - c0] = t;
                s_tau[slot] = t;
            }
            __syncthreads();
            // v_c and tau_c are published: release them to the cluster, then
            // update this CTA's trailing columns while the others copy v_c.
            cluster_arrive_release();
            if (!trivial)
                reflect_columns(Ys + size_t(c - c0 + 1) * m, m, c1 - c - 1, bv, cconj(t), c, m, lane, wid, nw);
            // The wait below orders nothing written after the arrive: the
            // next column's norm must not start before every warp's update.
            __syncthreads();
            cluster_wait_acquire();
        } else {
            cluster_arrive_release();
            cluster_wait_acquire();
            if (rank > owner && nloc > 0) {
                const double2* rv = cluster.map_shared_rank(bcast, owner) + size_t(slot) * m;
                for (int i = c + tid; i < m; i += kQrClusterThreads) vloc[i] = rv[i];
                const double2 t = *cluster.map_shared_rank(&s_tau[slot], owner);
                __syncthreads();
                if (t.x != 0.0 || t.y != 0.0) reflect_columns(Ys, m, nloc, vloc, cconj(t), c, m, lane, wid, nw);
                __syncthreads();
            }
        }
    }
    if (kGlobalCols) __threadfence();
    cluster.sync();  // every reflector is final
    for (int e = tid; e < nloc * m; e += kQrClusterThreads) {
        const int r = e % m, cc = c0 + e / m;
        Qs[e] = cmake(r == cc ? 1.0 : 0.0, 0.0);
    }
    // Backward accumulation, Q = H_0 ... H_{n-1} E.  Reflector c-1 is read
    // from its owner into registers before reflector c is applied, and
    // stored into the other half of a double buffer (vloc / bcast) after,
    // so the distributed-shared-memory latency overlaps the update.
    double2 pv[kQrRowsPerThread];
    double2 ptau = cmake(0, 0);
    auto pull = [&](int c) {
        const int owner = c / cpc;
        const double2* rcol = kGlobalCols ? B.y + size_t(c) * m
                                          : cluster.map_shared_rank(Ys, owner) + size_t(c - owner * cpc) * m;
#pragma unroll
        for (int k = 0; k < kQrRowsPerThread; ++k) {
            const int i = c + 1 + tid + k * kQrClusterThreads;
            if (i < m) pv[k] = kGlobalCols ? __ldcg(rcol + i) : rcol[i];
        }
        if (tid == 0) ptau = *(cluster.map_shared_rank(taus, owner) + (c - owner * cpc));
    };
    auto place = [&](int c, double2* dst, int sl) {
#pragma unroll
        for (int k = 0; k < kQrRowsPerThread; ++k) {
            const int i = c + 1 + tid + k * kQrClusterThreads;
            if (i < m) dst[i] = pv[k];
        }
        if (tid == 0) {
            dst[c] = cmake(1.0, 0.0);
            s_tau[sl] = ptau;
        }
    };
    int cur = 0;
    if (nloc > 0) {
        pull(c1 - 1);
        place(c1 - 1, vloc, 0);
    }
    __syncthreads();
    for (int c = nloc > 0 ? c1 - 1 : -1; c >= 0; --c) {
        if (c > 0) pull(c - 1);
        const double2 t = s_tau[cur];
        const int first = max(c, c0);
        if ((t.x != 0.0 || t.y != 0.0) && first < c1)
            reflect_columns(Qs + size_t(first - c0) * m, m, c1 - first, cur ? bcast : vloc, t, c, m, lane, wid,
                            nw);
        if (c > 0) place(c - 1, cur ? vloc : bcast, cur ^ 1);
        __syncthreads();
        cur ^= 1;
    }
    if (!kGlobalCols) {
        for (int e = tid; e < nloc * m; e += kQrClusterThreads) B.q[size_t(c0) * m + e] = Qs[e];
        for (int e = tid; e < nloc * m; e += kQrClusterThreads) B.y[size_t(c0) * m + e] = Ys[e];
    }
    if (tid < nloc) B.tau[c0 + tid] = taus[tid];
    cluster.sync();  // no CTA leaves while another may still read its shared memory
}

template <typename T>
__device__ __forceinline__ void jacobi_rotate(T* __restrict__ xp, T* __restrict__ xq, int M, int len, double tol2,
                                              double noise_floor, bool want_ratio, int lane, JacobiSweep& sw) {
    using R = typename JacobiReal<T>::R;
    // Two rows per lane per iteration into two accumulator sets: the loads
    // of the second row overlap the first's FMAs and the dependent chains
    // are half as long (the columns are distinct, hence __restrict__).
    R a_ = 0, b_ = 0, gr_ = 0, gi_ = 0, a1 = 0, b1 = 0, gr1 = 0, gi1 = 0;
    int r0 = lane;
    for (; r0 + 32 < M; r0 += 64) {
        const T u = xp[r0], v = xq[r0], u1 = xp[r0 + 32], v1 = xq[r0 + 32];
        a_ = fma(u.x, u.x, fma(u.y, u.y, a_));
        b_ = fma(v.x, v.x, fma(v.y, v.y, b_));
        gr_ = fma(u.x, v.x, fma(u.y, v.y, gr_));
        gi_ = fma(u.x, v.y, fma(-u.y, v.x, gi_));
        a1 = fma(u1.x, u1.x, fma(u1.y, u1.y, a1));
        b1 = fma(v1.x, v1.x, fma(v1.y, v1.y, b1));
        gr1 = fma(u1.x, v1.x, fma(u1.y, v1.y, gr1));
        gi1 = fma(u1.x, v1.y, fma(-u1.y, v1.x, gi1));
    }
    if (r0 < M) {
        const T u = xp[r0], v = xq[r0];
        a_ = fma(u.x, u.x, fma(u.y, u.y, a_));
        b_ = fma(v.x, v.x, fma(v.y, v.y, b_));
        gr_ = fma(u.x, v.x, fma(u.y, v.y, gr_));
        gi_ = fma(u.x, v.y, fma(-u.y, v.x, gi_));
    }
    a_ += a1;
    b_ += b1;
    gr_ += gr1;
    gi_ += gi1;
    warp_sum4(a_, b_, gr_, gi_, lane);
    double c64, wr64, wi64;
    if (!jacobi_params(a_, b_, gr_, gi_, tol2, noise_floor, want_ratio, sw, c64, wr64, wi64)) return;
    const R wr = R(wr64), wi = R(wi64), cr = R(c64);
    auto rot = [&](const T u, const T v, T& p, T& q) {
        p.x = fma(cr, u.x, -fma(wr, v.x, wi * v.y));
        p.y = fma(cr, u.y, -fma(wr, v.y, -wi * v.x));
        q.x = fma(wr, u.x, fma(-wi, u.y, cr * v.x));
        q.y = fma(wr, u.y, fma(wi, u.x, cr * v.y));
    };
    // Four rows per lane per iteration: all loads issue before the stores.
    int r = lane;
    for (; r + 96 < len; r += 128) {
        T u[4], v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            u[k] = xp[r + 32 * k];
            v[k] = xq[r + 32 * k];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            T p, q;
            rot(u[k], v[k], p, q);
            xp[r + 32 * k] = p;
            xq[r + 32 * k] = q;
        }
    }
    for (; r < len; r += 32) {
        T p, q;
        rot(xp[r], xq[r], p, q);
        xp[r] = p;
        xq[r] = q;
    }
}

// ---------------------------------------------------------------------------
// The same Jacobi SVD for working matrices too large for a cluster's shared
// memory (theta up to 512 x 512 at chi 256: W takes 4 MB in FP64, a 16-CTA
// cluster holds 3.6 MB with two working blocks per CTA).  The padded W
// columns live in the slot's global workspace `gs`, which stays in L2.
// The N' = 2Kb columns form 2K blocks of b; a sweep runs 2K-1 steps of the
// circle method over the blocks (position 0 fixed, block at position p at
// step s: circle_at(p, s, 2K)), and at each step CTA r takes the block pairs
// r, r+C, ... < K: it loads both blocks into shared memory, rotates the b*b
// cross pairs (and, at a sweep's first step, the pairs inside each block),
// and stores them back.  One cluster barrier separates the steps: every
// block is held by one pair per step, so a block's store and its next load
// are ordered by that barrier.  Rotation rule, tolerances, stop test and
// outputs are those of jacobi_ring_kernel.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kJacobiStagedThreads) jacobi_staged_kernel(const SplitJob* jobs, SplitState* st,
                                                                         const SlotBuffers* slots, const int* idx,
                                                                         int mode, int phase, int max_sweeps, int b,
                                                                         int* status, unsigned long long* counters) {
    constexpr bool kF64 = sizeof(T) == sizeof(double2);
    cg::cluster_group cluster = cg::this_cluster();
    const int C = int(cluster.num_blocks());
    const int rank = int(cluster.block_rank());
    const int j = jacobi_entry_job(idx[blockIdx.x / C]);
    const SplitState S = st[j];
    if (!jacobi_active(S, mode)) return;  // uniform over the cluster
    const SplitJob& J = jobs[j];
    const SlotBuffers Bf = slots[J.slot];
    JacobiMatrix X = jacobi_matrix(J, S, Bf, mode);
    const bool pre = jacobi_preconditioned(S, mode);
    if (phase == kPhaseFinish) {  // from X V, in the slot's W buffer
        X.p = Bf.w;
        X.ld = X.M;
        X.by_rows = 0;
        X.by_cols = 1;
    }
    const bool dusted = pre || phase == kPhaseFinish;  // entries already dust-zeroed
    const int M = X.M, N = X.N;
    const int K = (N + 2 * b - 1) / (2 * b);
    const int nblk = 2 * K;
    const int Np = nblk * b;
    const int vrows = phase == kPhaseFp32V ? N : 0;  // as in jacobi_ring_kernel
    const int len = M + vrows;
    const size_t blk = size_t(b) * len;
    T* G = reinterpret_cast<T*>(Bf.gs);
    if (G == nullptr) {  // a state sized without the workspace (uniform over the cluster)
        if (threadIdx.x == 0 && rank == 0) atomicOr(status, kStatusBadShape);
        return;
    }

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sA = reinterpret_cast<T*>(smem_raw);
    T* sB = sA + blk;
    __shared__ JacobiCtl ctl;
    __shared__ double red[kJacobiStagedThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nthreads = blockDim.x;
    const int nwarps = nthreads / 32;
    // Frobenius norm: CTA r reads columns r, r+C, ...
    double part = 0;
    for (int col = rank; col < N; col += C)
        for (int i = tid; i < M; i += nthreads) part += cnorm2(X.at(i, col));
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) red[wid] = part;
    __syncthreads();
    if (tid == 0) {
        double t = 0;
        for (int w = 0; w < nwarps; ++w) t += red[w];
        ctl.fro_part = t;
    }
    cluster.sync();
    double fro2 = 0;
    for (int r = 0; r < C; ++r) fro2 += cluster.map_shared_rank(&ctl, r)->fro_part;
    const double dust = sqrt(fro2) * kDustRel;
    const double dust2 = dust * dust;
    // W (dust-zeroed, zero padding columns) into the workspace.
    double chk_in = 0, chk_out = 0;
    for (int col = rank; col < Np; col += C) {
        T* x = G + size_t(col) * len;
        for (int i = tid; i < M; i += nthreads) {
            double2 v = col < N ? X.at(i, col) : cmake(0, 0);
            if (!dusted && cnorm2(v) < dust2) v = cmake(0, 0);
            chk_in += cnorm2(v);
            x[i] = to_store<T>(v);
        }
        for (int i = tid; i < vrows; i += nthreads) x[M + i] = to_store<T>(cmake(col == i ? 1.0 : 0.0, 0.0));
    }
    __threadfence();
    cluster.sync();
    const double tol2 = kF64 ? kJacobiTol2 : kJacobiTol2Fp32;
    const double noise_floor = (kF64 ? 1e-30 : 1e-12) * fro2;  // squared column norm: 1e-15 (1e-6) of ||W||_F
    int sweep = 0;
    bool converged = false;
    int ctl_rot_last = 0;
    unsigned long long ctl_relmax_bits_last = 0ull;
    for (; sweep < max_sweeps; ++sweep) {
        if (tid == 0) {
            ctl.rot = 0;
            ctl.ecos = ctl.esin = -8192;
            ctl.relmax_bits = 0ull;
        }
        __syncthreads();
        JacobiSweep my;
        const bool want_ratio = sweep == max_sweeps - 1;
        for (int step = 0; step < nblk - 1; ++step) {
            for (int ps = rank; ps < K; ps += C) {
                const int ida = circle_at(ps, step, nblk), idb = circle_at(nblk - 1 - ps, step, nblk);
                const T* ga = G + size_t(ida) * blk;
                const T* gb = G + size_t(idb) * blk;
                for (size_t e = tid; e < blk; e += nthreads) {
                    sA[e] = __ldcg(ga + e);
                    sB[e] = __ldcg(gb + e);
                }
                __syncthreads();
                if (step == 0) {  // pairs inside each block, once per sweep
                    // Circle method on bb = b rounded up to even positions; for
                    // an odd b the extra position is a dummy and its pair is
                    // skipped (uniformly per warp).
                    const int bb = b + (b & 1);
                    for (int s2 = 0; s2 < bb - 1; ++s2) {
                        for (int pq = wid; pq < bb; pq += nwarps) {
                            const bool top = pq < bb / 2;
                            const int i = top ? pq : pq - bb / 2;
                            T* base = top ? sA : sB;
                            const int e1 = circle_at(i, s2, bb), e2 = circle_at(bb - 1 - i, s2, bb);
                            if (e1 < b && e2 < b)
                                jacobi_rotate(base + size_t(e1) * len, base + size_t(e2) * len, M, len, tol2,
                                              noise_floor, want_ratio, lane, my);
                        }
                        __syncthreads();
                    }
                }
                for (int k = 0; k < b; ++k) {
                    for (int i = wid; i < b; i += nwarps) {
                        const int e2 = (i + k) % b;
                        jacobi_rotate(sA + size_t(i) * len, sB + size_t(e2) * len, M, len, tol2,
                                      noise_floor, want_ratio, lane, my);
                    }
                    __syncthreads();
                }
                T* wa = G + size_t(ida) * blk;
                T* wb = G + size_t(idb) * blk;
                for (size_t e = tid; e < blk; e += nthreads) {
                    wa[e] = sA[e];
                    wb[e] = sB[e];
                }
                __syncthreads();  // the next pair's loads overwrite sA, sB
            }
            __threadfence();
            cluster.sync();
        }
        jacobi_report(ctl, my, lane);
        __syncthreads();
        int total = 0, ecos = -8192, esin = -8192;
        unsigned long long relmax_bits = 0;
        cluster.sync();
        for (int r = 0; r < C; ++r) {
            const JacobiCtl* rc = cluster.map_shared_rank(&ctl, r);
            total += rc->rot;
            ecos = max(ecos, rc->ecos);
            esin = max(esin, rc->esin);
            relmax_bits = max(relmax_bits, rc->relmax_bits);
        }
        cluster.sync();
        ctl_rot_last = total;
        ctl_relmax_bits_last = relmax_bits;
        if (jacobi_done(kF64, total, ecos, esin)) {
            converged = true;
            break;
        }
    }
    if (tid == 0 && rank == 0) {
        if (!converged) {
            atomicOr(status, kStatusJacobiNoConvergence);
            // The first such split, its last sweep's rotation count and largest
            // squared |gamma| / sqrt(alpha beta), for the error message.
            if (atomicCAS(status + 1, 0, J.seq + 1) == 0) {
                const unsigned long long bits = ctl_relmax_bits_last;
                status[2] = ctl_rot_last;
                status[3] = int(bits >> 32);
                status[4] = int(bits & 0xffffffffull);
            }
        }
        if (phase != kPhaseFp32V) atomicAdd(counters + 0, 1ull);
        atomicAdd(counters + (phase == kPhaseFp32V ? 2 : 1), (unsigned long long)(converged ? sweep + 1 : sweep));
    }
    if (phase == kPhaseFp32V) {  // V (FP64) and ||X||_F^2 for the finishing phase
        for (int col = rank + C * wid; col < N; col += C * nwarps)
            for (int r = lane; r < N; r += 32) Bf.z[size_t(col) * N + r] = to_f64(__ldcg(G + size_t(col) * len + M + r));
        if (rank == 0 && tid == 0) st[j].fro2 = fro2;
        cluster.sync();
        return;
    }
    // Write back W and the column norms; CTA r takes columns r, r+C, ...,
    // one warp per column.
    for (int col = rank + C * wid; col < N; col += C * nwarps) {
        const T* x = G + size_t(col) * len;
        double s2 = 0;
        for (int r = lane; r < M; r += 32) {
            const double2 v = to_f64(__ldcg(x + r));
            s2 = fma(v.x, v.x, fma(v.y, v.y, s2));
            Bf.w[size_t(col) * M + r] = v;
        }
        for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        if (lane == 0) {
            Bf.sigma[col] = jacobi_sigma(s2, fro2, mode);
            chk_out += s2;
        }
    }
    // Factorisation check over the cluster, as in jacobi_ring_kernel.
    {
        const double in_cta = block_total(chk_in, red);
        const double out_cta = block_total(chk_out, red);
        if (tid == 0) {
            ctl.chk_in = in_cta;
            ctl.chk_out = out_cta;
        }
        cluster.sync();
        if (rank == 0 && tid == 0) {
            double tin = 0, tout = 0;
            for (int r = 0; r < C; ++r) {
                const JacobiCtl* rc = cluster.map_shared_rank(&ctl, r);
                tin += rc->chk_in;
                tout += rc->chk_out;
            }
            if (pre) tin = S.pre_fro2;  // the matrix before its QR
            const double tol = kF64 ? kSvdCheckTol : kSvdCheckTolFp32;
            if (fabs(tout - tin) > tol * tin + 1e-28) atomicOr(status, kStatusSvdCheck);
        }
        cluster.sync();  // no CTA leaves while rank 0 reads its shared memory
    }
}

// ---------------------------------------------------------------------------
// The probe-vector half of the reference's factorisation check
// (svd_reproduces, svd_guard.rs:256-283): U Sigma V^H x must reproduce X x
// for the two fixed probes x_j = (sin t, cos t), t = (j + 1) (0.754877666 +
// p 0.56984029), to 1e-9 ||X||_F ||x|| + 1e-14.  The Jacobi keeps W = X V =
// U Sigma and no V, and U Sigma V^H x = U U^H X x over the columns with
// sigma > 0, so with y = X x the rebuilt vector is W diag(1/sigma^2) W^H y:
// it equals y only when W's columns are orthogonal and span X's range.  A
// Jacobi on R^H (jacobi_qr.cu) leaves X's right vectors in W: the same check
// on X^H, which covers the QR too.
// Columns at the storage's rounding level (the Jacobi's noise floor) are
// left out: their direction is noise and they carry less than the tolerance.
// One CTA per (job, probe); a failure sets the same status as the Frobenius
// check ("failed its check").
// ---------------------------------------------------------------------------
constexpr int kProbeMax = 512;

// out[i] = sum_c A(i, c) x[c] for i < M, c < N.  With `down` A(i, c) runs
// fastest in memory over i: a thread per row, the columns dealt to
// kProbeThreads / (M rounded up to a warp) groups of threads whose parts are
// added in order; else a warp per row, lanes along it.  Ends with a barrier.
template <typename At>
__device__ __forceinline__ void probe_matvec(int M, int N, bool down, At at, const double2* x, double2* out,
                                             double2* parts) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (down) {
        const int span = (M + 31) & ~31, groups = kProbeThreads / span;  // span <= 512
        const int g = tid / span, i = tid % span;
        double2 acc = cmake(0, 0);
        if (g < groups && i < M)
#pragma unroll 8
            for (int c = g; c < N; c += groups) cfma(acc, at(i, c), x[c]);
        if (g < groups) parts[tid] = acc;
        __syncthreads();
        for (int r = tid; r < M; r += kProbeThreads) {
            double2 t = parts[r];
            for (int q = 1; q < groups; ++q) t = cadd(t, parts[q * span + r]);
            out[r] = t;
        }
    } else {
        for (int i = wid; i < M; i += kProbeThreads / 32) {
            double2 acc = cmake(0, 0);
#pragma unroll 4
            for (int c = lane; c < N; c += 32) cfma(acc, at(i, c), x[c]);
            for (int o = 16; o > 0; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            if (lane == 0) out[i] = acc;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kProbeThreads) svd_probe_kernel(const SplitJob* jobs, const SplitState* st,
                                                                  const SlotBuffers* slots, int mode, int fp32,
                                                                  int* status) {
    const int j = blockIdx.x;
    const int probe = blockIdx.y;
    const SplitState S = st[j];
    if (!jacobi_active(S, mode)) return;
    const SplitJob& J = jobs[j];
    const SlotBuffers Bf = slots[J.slot];
    const double2* src;
    int sr, sc, ld, rows_of_src;
    jacobi_task(J, S, Bf, mode, src, sr, sc, ld, rows_of_src);
    // W's columns are left vectors of X, or with a preconditioned Jacobi left
    // vectors of X^H: the check is made on that matrix, M x N with K columns of W.
    const int K = rows_of_src ? sr : sc;
    if (jacobi_preconditioned(S, mode)) rows_of_src = !rows_of_src;
    const int M = rows_of_src ? sc : sr;
    const int N = rows_of_src ? sr : sc;
    if (M > kProbeMax || N > kProbeMax) {
        if (threadIdx.x == 0) atomicOr(status, kStatusBadShape);
        return;
    }
    __shared__ double2 xs[kProbeMax], ys[kProbeMax], zs[kProbeMax], parts[kProbeThreads];
    __shared__ double red[kProbeThreads / 32];
    const int tid = threadIdx.x;
    const double step = 0.754877666 + double(probe) * 0.56984029;
    double fro2_part = 0;
    for (int c = tid; c < N; c += kProbeThreads) {
        double sn, cs;
        sincos(double(c + 1) * step, &sn, &cs);
        xs[c] = cmake(sn, cs);
    }
    for (int c = tid; c < K; c += kProbeThreads) {
        const double sg = Bf.sigma[c];
        fro2_part += sg * sg;
    }
    const double fro2 = block_total(fro2_part, red);  // its barriers also publish xs
    const double floor2 = (fp32 ? 1e-12 : 1e-30) * fro2;
    // y = X x.
    if (rows_of_src)
        probe_matvec(M, N, true, [&](int i, int c) { return cconj(src[size_t(c) * ld + i]); }, xs, ys, parts);
    else
        probe_matvec(M, N, false, [&](int i, int c) { return src[size_t(i) * ld + c]; }, xs, ys, parts);
    // z = diag(1/sigma^2) W^H y.
    probe_matvec(K, M, false, [&](int c, int i) { return cconj(Bf.w[size_t(c) * M + i]); }, ys, zs, parts);
    for (int c = tid; c < K; c += kProbeThreads) {
        const double sg = Bf.sigma[c];
        zs[c] = sg * sg > floor2 ? cscale(zs[c], 1.0 / (sg * sg)) : cmake(0, 0);
    }
    __syncthreads();
    // |y - W z|^2.
    probe_matvec(M, K, true, [&](int i, int c) { return Bf.w[size_t(c) * M + i]; }, zs, xs, parts);
    double err2 = 0;
    for (int i = tid; i < M; i += kProbeThreads) err2 += cnorm2(csub(ys[i], xs[i]));
    const double e2 = block_total(err2, red);
    if (tid == 0) {
        const double tol = fp32 ? 1e-4 : 1e-9;  // the Frobenius check's tolerance of each form
        if (!(sqrt(e2) <= tol * sqrt(fro2) * sqrt(double(N)) + 1e-14)) atomicOr(status, kStatusSvdCheck);
    }
}

// ---------------------------------------------------------------------------
// The precision form's FP64 products between its Jacobi phases (see
// split_kernels.cuh), batched over the wave's jobs.  Waves of few jobs take
// 16 x 16 tiles (96 x 96 matrices: 7 us a product, against 14 with 32 x 32 tiles
// on 9 CTAs a job); waves that fill the device 32 x 32, four outputs a thread,
// which read shared memory half as often (a batch of 128 slices of bonds up to
// 128: 1.53 s, against 1.66 with the small tiles).  G lives
// in the slot's omega and y0 buffers and V' in zr and y (each pair holds
// 2 R ell >= R^2 entries); none of them is in use while an SVD of the job
// runs.
// ---------------------------------------------------------------------------
template <bool kSmall>
__global__ void __launch_bounds__(256) precond_gemm_kernel(const SplitJob* jobs, const SplitState* st,
                                                           const SlotBuffers* slots, int mode, int stage) {
    constexpr int kT = kSmall ? kTile : kPrecondTile;
    const int j = blockIdx.z;
    const SplitState S = st[j];
    if (!jacobi_active(S, mode)) return;
    const SplitJob& J = jobs[j];
    const SlotBuffers B = slots[J.slot];
    const JacobiMatrix X = jacobi_matrix(J, S, B, mode);
    const int M = X.M, N = X.N;
    const bool last = stage == kPrecondXV;
    const int m = last ? M : N, n = N, k = N;
    const int i0 = blockIdx.y * kT, n0 = blockIdx.x * kT;
    if (i0 >= m || n0 >= n) return;
    // Two Newton-Schulz steps: V (z) -> zr -> z; then X V from z.
    const bool second = stage >= kPrecondGram2;
    const double2* V = last ? B.z : (second ? B.zr : B.z);
    double2* G = B.omega;
    double2* Vout = second ? B.z : B.zr;
    const bool gram = stage == kPrecondGram1 || stage == kPrecondGram2;
    const double dust2 = jacobi_preconditioned(S, mode) ? 0.0 : kDustRel * kDustRel * S.fro2;
    auto a_at = [&](int i, int kk) -> double2 {
        if (gram) return cconj(V[size_t(i) * N + kk]);  // V^H
        if (!last) return V[size_t(kk) * N + i];
        const double2 x = X.at(i, kk);
        return cnorm2(x) < dust2 ? cmake(0, 0) : x;  // X, dust-zeroed as the first phase loaded it
    };
    auto b_at = [&](int kk, int jj) -> double2 {
        if (gram) return V[size_t(jj) * N + kk];
        if (!last) {
            const double2 g = G[size_t(jj) * N + kk];
            return cmake((kk == jj ? 1.5 : 0.0) - 0.5 * g.x, -0.5 * g.y);
        }
        return V[size_t(jj) * N + kk];
    };
    double2* C = gram ? G : last ? B.w : Vout;
    const int ldc = last ? M : N;
    if constexpr (kSmall) {
        __shared__ TileSmem sm;
        // C is column-major, so the transposed product is what stores in runs.
        tile_gemm(
            sm, n0, i0, n, m, k, true, gram, [&](int jj, int kk) { return b_at(kk, jj); },
            [&](int kk, int i) { return a_at(i, kk); },
            [&](int jj, int i, double2 v) { C[size_t(jj) * ldc + i] = v; });
    } else {
        constexpr int kK = 16;
        __shared__ double2 As[kT][kK + 1];
        __shared__ double2 Bs[kK][kT + 1];
        const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16;
        double2 acc[2][2] = {{cmake(0, 0), cmake(0, 0)}, {cmake(0, 0), cmake(0, 0)}};
        for (int k0 = 0; k0 < k; k0 += kK) {
            for (int e = tid; e < kT * kK; e += 256) {
                const int r = e / kK, c = e % kK;
                As[r][c] = (i0 + r < m && k0 + c < k) ? a_at(i0 + r, k0 + c) : cmake(0, 0);
            }
            for (int e = tid; e < kK * kT; e += 256) {
                const int r = e / kT, c = e % kT;
                Bs[r][c] = (k0 + r < k && n0 + c < n) ? b_at(k0 + r, n0 + c) : cmake(0, 0);
            }
            __syncthreads();
#pragma unroll 4
            for (int c = 0; c < kK; ++c) {
                const double2 a0 = As[tr][c], a1 = As[tr + 16][c];
                const double2 b0 = Bs[c][tc], b1 = Bs[c][tc + 16];
                cfma(acc[0][0], a0, b0);
                cfma(acc[0][1], a0, b1);
                cfma(acc[1][0], a1, b0);
                cfma(acc[1][1], a1, b1);
            }
            __syncthreads();
        }
        for (int x = 0; x < 2; ++x)
            for (int y = 0; y < 2; ++y) {
                const int i = i0 + tr + 16 * x, jj = n0 + tc + 16 * y;
                if (i < m && jj < n) C[size_t(jj) * ldc + i] = acc[x][y];
            }
    }
}
template __global__ void precond_gemm_kernel<true>(const SplitJob*, const SplitState*, const SlotBuffers*, int, int);
template __global__ void precond_gemm_kernel<false>(const SplitJob*, const SplitState*, const SlotBuffers*, int, int);

// ---------------------------------------------------------------------------
// The cut: stable descending sort, truncation rule, discarded weight and the
// split record, then both sides into the sites.
// ---------------------------------------------------------------------------
struct CutSmem {
    double vals[1024];  // singular values, descending, noise at zero
    int perm[1024];     // sorted position -> column of W
};

// rank_j = #{i : s_i > s_j or (s_i == s_j and i < j)}; every thread of the CTA.
__device__ __forceinline__ void sort_values(CutSmem& sm, const double* sigma, int N, int mode, double noise_rel) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int c = tid; c < N; c += nt) sm.perm[c] = c;  // a NaN among the values leaves places unwritten below
    __shared__ double raw[1024];
    for (int c = tid; c < N; c += nt) raw[c] = sigma[c];
    __syncthreads();
    for (int c = tid; c < N; c += nt) {
        const double sj = raw[c];
        int r = 0;
        for (int i = 0; i < N; ++i) {
            const double si = raw[i];
            r += (si > sj || (si == sj && i < c)) ? 1 : 0;
        }
        sm.perm[r] = c;
    }
    __syncthreads();
    const double floor_abs = N > 0 ? noise_rel * raw[sm.perm[0]] : 0.0;
    for (int c = tid; c < N; c += nt) {
        double v = raw[sm.perm[c]];
        if (mode == kJacobiRsvd && v < kRsvdZero) v = 0.0;
        if (v < floor_abs) v = 0.0;
        sm.vals[c] = v;
    }
    __syncthreads();
}

// retained_chi (svd_guard.rs:25-35); every thread of the CTA.
__device__ __forceinline__ int kept_bond(const CutSmem& sm, int N, const SplitJob& J, const SplitState& S, int chi_max) {
    int rank = 0;
    for (int base = 0; base < N; base += blockDim.x) {
        const int c = base + int(threadIdx.x);
        rank += __syncthreads_count(c < N && sm.vals[c] > kSingularCutoff);
    }
    return N == 0 ? 0 : min(min(max(rank, 1), J.chi_max > 0 ? J.chi_max : chi_max), min(S.rows, S.cols));
}

// The outcome of an exact SVD, or of a range finder that is accepted; one thread.
__device__ __forceinline__ void record_cut(const CutSmem& sm, int N, int chi, int final_kind, const SplitJob& J,
                                           SplitState& S, wqc_split_info* records, int* status) {
    bool bad = false;
    for (int i = 0; i < N; ++i)
        if (!isfinite(sm.vals[i]) || sm.vals[i] < 0.0) bad = true;
    if (final_kind == 0) {
        if (J.reject) {
            for (int i = chi; i < N; ++i)
                if (sm.vals[i] > kSingularCutoff) {
                    atomicOr(status, kStatusTruncationRejected);
                    break;
                }
        }
        if (bad) atomicOr(status, kStatusNonFinite);
    }
    double disc = 0;
    for (int i = chi; i < N; ++i) disc += sm.vals[i] * sm.vals[i];
    S.final_kind = final_kind;
    S.chi = chi;
    S.discarded = disc;
    wqc_split_info info;
    info.left_site = J.p;
    info.rows = S.rows;
    info.cols = S.cols;
    info.ell = S.ell;
    info.path = S.path;
    info.chi = chi;
    info.discarded_weight = disc;
    records[J.seq] = info;
}

// finalize: the cut of a wave in which range finders take part, with the
// ambiguity test that sends one back to the exact path.
__global__ void finalize_kernel(const SplitJob* jobs, SplitState* st, const SlotBuffers* slots, int mode,
                                int chi_max, double noise_rel, wqc_split_info* records, int* status) {
    const int j = blockIdx.x;
    SplitState& S = st[j];
    if (!jacobi_active(S, mode)) return;
    const SplitJob& J = jobs[j];
    const SlotBuffers B = slots[J.slot];
    const int N = mode == kJacobiRsvd ? S.ell : min(S.rows, S.cols);
    __shared__ CutSmem sm;
    sort_values(sm, B.sigma, N, mode, noise_rel);
    for (int c = threadIdx.x; c < N; c += blockDim.x) B.perm[c] = sm.perm[c];
    const int chi = kept_bond(sm, N, J, S, chi_max);
    if (threadIdx.x != 0) return;
    if (mode == kJacobiRsvd) {
        // needs_f64_fallback (svd_guard.rs:58-76)
        bool fb = chi == 0;
        for (int i = 0; i < N && !fb; ++i) {
            if (!isfinite(sm.vals[i]) || sm.vals[i] < 0.0) fb = true;
            if (sm.vals[i] > 0.0 && fabs(sm.vals[i] - kSingularCutoff) <= kCutoffAbsBand) fb = true;
        }
        if (!fb && chi > 0 && chi < N) {
            const double kept = sm.vals[chi - 1], dropped = sm.vals[chi];
            const double scale = fmax(fmax(kept, dropped), 1e-30);
            if (fabs(kept - dropped) / scale < kChiRelGap) fb = true;
        }
        if (fb) {
            S.need_exact = 1;
            S.path = WQC_SPLIT_RSVD_FALLBACK;
            return;
        }
    }
    record_cut(sm, N, chi, mode == kJacobiRsvd ? 1 : 0, J, S, records, status);
}

// ---------------------------------------------------------------------------
// Recovery of the side the Jacobi does not accumulate, as tiled batched
// GEMMs over the kept columns (m < chi, W column pc = perm[m]), with the
// s^-3/2 scale in the epilogue.  W = X V = U_X Sigma for X = theta, theta^H
// or B^H, so (kept columns, sigma > 0):
//   kRecoverBW:   T = B W_k                  (ell x chi, into the slot's z, column pc)
//   kRecoverQT:   L = Q T s^-3/2             (range finder, rows x chi, into site p)
//   kRecoverExact: R = s^-3/2 W_k^H theta    (W left vectors, into site p+1)
//                  L = theta W_k s^-3/2      (W right vectors, into site p)
// A range finder's Jacobi on R^H (jacobi_qr.cu) leaves B's left vectors in W:
//   kRecoverBW:   R = s^-3/2 W_k^H B         (chi x cols, into site p+1)
//   kRecoverQT:   L = Q W_k s^-1/2           (rows x chi, into site p)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double inv_s32(double sg) { return sg > 0.0 ? 1.0 / (sg * sqrt(sg)) : 0.0; }
__device__ __forceinline__ double inv_s12(double sg) { return sg > 0.0 ? 1.0 / sqrt(sg) : 0.0; }

// The recovered side of an exact SVD, one tile.
__device__ __forceinline__ void recover_exact(TileSmem& sm, int m0, int n0, const SplitJob& J, const SplitState& S,
                                              const SlotBuffers& B, const int* perm, int chi, const DeviceMps& mps) {
    const int rows = S.rows, cols = S.cols;
    if (!S.w_rows_of_src) {
        if (m0 >= chi || n0 >= cols) return;
        double2* R = mps.site[J.p + 1];
        tile_gemm(
            sm, m0, n0, chi, cols, rows, true, false,
            [&](int i, int k) { return cconj(B.w[size_t(perm[i]) * rows + k]); },
            [&](int k, int c) { return B.theta[size_t(k) * cols + c]; },
            [&](int i, int c, double2 v) { R[size_t(i) * cols + c] = cscale(v, inv_s32(B.sigma[perm[i]])); });
    } else {
        if (m0 >= rows || n0 >= chi) return;
        double2* L = mps.site[J.p];
        tile_gemm(
            sm, m0, n0, rows, chi, cols, true, true, [&](int i, int k) { return B.theta[size_t(i) * cols + k]; },
            [&](int k, int c) { return B.w[size_t(perm[c]) * cols + k]; },
            [&](int i, int c, double2 v) { L[size_t(i) * chi + c] = cscale(v, inv_s32(B.sigma[perm[c]])); });
    }
}

__global__ void __launch_bounds__(kTileThreads) recover_gemm_kernel(const SplitJob* jobs, const SplitState* st,
                                                                    const SlotBuffers* slots, DeviceMps mps,
                                                                    int stage) {
    const int j = blockIdx.z;
    const SplitJob& J = jobs[j];
    const SplitState S = st[j];
    if (S.skip) return;
    const bool rf = S.final_kind == 1;
    if ((stage == kRecoverExact) == rf) return;
    const SlotBuffers B = slots[J.slot];
    const int rows = S.rows, cols = S.cols, ell = S.ell, chi = S.chi;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    __shared__ TileSmem sm;
    if (stage == kRecoverExact) {
        recover_exact(sm, m0, n0, J, S, B, B.perm, chi, mps);
        return;
    }
    auto q_at = [&](int i, int k) { return B.q[size_t(k) * rows + i]; };
    if (stage == kRecoverBW && !S.pre_rsvd) {
        if (m0 >= ell || n0 >= chi) return;
        tile_gemm(
            sm, m0, n0, ell, chi, cols, true, true, [&](int i, int k) { return B.b[size_t(i) * cols + k]; },
            [&](int k, int c) { return B.w[size_t(B.perm[c]) * cols + k]; },
            [&](int i, int c, double2 v) { B.z[size_t(B.perm[c]) * ell + i] = v; });
    } else if (stage == kRecoverBW) {
        if (m0 >= chi || n0 >= cols) return;
        double2* R = mps.site[J.p + 1];
        tile_gemm(
            sm, m0, n0, chi, cols, ell, true, false,
            [&](int i, int k) { return cconj(B.w[size_t(B.perm[i]) * ell + k]); },
            [&](int k, int c) { return B.b[size_t(k) * cols + c]; },
            [&](int i, int c, double2 v) { R[size_t(i) * cols + c] = cscale(v, inv_s32(B.sigma[B.perm[i]])); });
    } else {
        if (m0 >= rows || n0 >= chi) return;
        double2* L = mps.site[J.p];
        const double2* T = S.pre_rsvd ? B.w : B.z;
        tile_gemm(
            sm, m0, n0, rows, chi, ell, false, true, q_at,
            [&](int k, int c) { return T[size_t(B.perm[c]) * ell + k]; },
            [&](int i, int c, double2 v) {
                const double sg = B.sigma[B.perm[c]];
                L[size_t(i) * chi + c] = cscale(v, S.pre_rsvd ? inv_s12(sg) : inv_s32(sg));
            });
    }
}

// The side that is a plain copy of W (L = W / sqrt(s) where W holds left
// vectors, R = W^H / sqrt(s) where it holds right ones; mps.rs:1156-1168,
// 1039-1051), entries t0, t0 + stride, ...
__device__ __forceinline__ void copy_side(const SplitJob& J, const SplitState& S, const SlotBuffers& B, bool left,
                                          const int* perm, int chi, const DeviceMps& mps, long t0, long stride) {
    const int rows = S.rows, cols = S.cols;
    if (left) {
        double2* Ls = mps.site[J.p];
        for (long e = t0; e < long(rows) * chi; e += stride) {
            const int r = int(e / chi), pc = perm[e % chi];
            Ls[e] = cscale(B.w[size_t(pc) * rows + r], inv_s12(B.sigma[pc]));  // L[(r/2)][r%2][m] at r*chi + m
        }
    } else {
        double2* Rs = mps.site[J.p + 1];
        for (long e = t0; e < long(chi) * cols; e += stride) {
            const int c = int(e % cols), pc = perm[e / cols];
            Rs[e] = cscale(cconj(B.w[size_t(pc) * cols + c]), inv_s12(B.sigma[pc]));  // R[m][c/dr][c%dr]
        }
    }
}

// absorb: the copied sides of a wave with range finders, and the new bonds.
__global__ void __launch_bounds__(256) absorb_kernel(const SplitJob* jobs, const SplitState* st,
                                                     const SlotBuffers* slots, DeviceMps mps) {
    const int j = blockIdx.y;
    const SplitJob& J = jobs[j];
    const SplitState S = st[j];
    if (S.skip) return;
    const SlotBuffers B = slots[J.slot];
    if (!(S.final_kind == 1 && S.pre_rsvd))  // both sides come from recover_gemm_kernel
        copy_side(J, S, B, S.final_kind == 0 && !S.w_rows_of_src, B.perm, S.chi, mps,
                  long(blockIdx.x) * blockDim.x + threadIdx.x, long(gridDim.x) * blockDim.x);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        mps.dr[J.p] = S.chi;
        mps.dl[J.p + 1] = S.chi;
    }
}

// The whole cut of a wave without range finders in one launch: every CTA sorts
// the values for itself (N^2 / 256 compares a thread, ~2 us at N = 256) and
// then computes a tile of the recovered side (blocks below `tiles`, tiles_n to
// a row) or copies a part of the other; block 0 records.  Three launches, two
// of them a few microseconds of work behind a launch each, took 27 us at 64
// columns and 87 us at 256.
__global__ void __launch_bounds__(kTileThreads) cut_kernel(const SplitJob* jobs, SplitState* st,
                                                           const SlotBuffers* slots, DeviceMps mps, int tiles,
                                                           int tiles_n, int chi_max, double noise_rel,
                                                           wqc_split_info* records, int* status) {
    const int j = blockIdx.y;
    const SplitJob& J = jobs[j];
    const SplitState S = st[j];
    if (!jacobi_active(S, kJacobiExact)) return;
    const SlotBuffers B = slots[J.slot];
    const int N = min(S.rows, S.cols);
    const int bx = blockIdx.x, m0 = (bx / tiles_n) * kTile, n0 = (bx % tiles_n) * kTile;
    // Tiles past what the largest kept bond can need leave before the sort.
    if (bx > 0 && bx < tiles &&
        (S.w_rows_of_src ? m0 >= S.rows || n0 >= min(N, J.chi_max) : m0 >= min(N, J.chi_max) || n0 >= S.cols))
        return;
    __shared__ CutSmem cut;
    sort_values(cut, B.sigma, N, kJacobiExact, noise_rel);
    const int chi = kept_bond(cut, N, J, S, chi_max);
    if (bx < tiles) {
        __shared__ TileSmem sm;
        recover_exact(sm, m0, n0, J, S, B, cut.perm, chi, mps);
    } else {
        copy_side(J, S, B, !S.w_rows_of_src, cut.perm, chi, mps, long(bx - tiles) * blockDim.x + threadIdx.x,
                  long(gridDim.x - tiles) * blockDim.x);
    }
    if (bx == 0) {
        for (int c = threadIdx.x; c < N; c += blockDim.x) B.perm[c] = cut.perm[c];
        if (threadIdx.x == 0) {
            record_cut(cut, N, chi, 0, J, st[j], records, status);
            mps.dr[J.p] = chi;
            mps.dl[J.p + 1] = chi;
        }
    }
}

}  // namespace wqc

namespace wqc {
const void* qr_cluster(bool global_cols) {
    return global_cols ? reinterpret_cast<const void*>(qr_cluster_kernel<true>)
                       : reinterpret_cast<const void*>(qr_cluster_kernel<false>);
}

cudaError_t launch_qr_cluster(bool global_cols, const cudaLaunchConfig_t& cfg, const SplitJob* jobs,
                              const SplitState* st, const SlotBuffers* slots) {
    if (global_cols) return cudaLaunchKernelEx(&cfg, qr_cluster_kernel<true>, jobs, st, slots);
    return cudaLaunchKernelEx(&cfg, qr_cluster_kernel<false>, jobs, st, slots);
}

const void* jacobi_staged(bool fp32) {
    return fp32 ? reinterpret_cast<const void*>(jacobi_staged_kernel<float2>)
                : reinterpret_cast<const void*>(jacobi_staged_kernel<double2>);
}

cudaError_t launch_jacobi_staged(bool fp32, const cudaLaunchConfig_t& cfg, const SplitJob* jobs, SplitState* st,
                                 const SlotBuffers* slots, const int* idx, int mode, int phase, int max_sweeps, int b,
                                 int* status, unsigned long long* counters) {
    if (fp32)
        return cudaLaunchKernelEx(&cfg, jacobi_staged_kernel<float2>, jobs, st, slots, idx, mode, phase, max_sweeps, b,
                                  status, counters);
    return cudaLaunchKernelEx(&cfg, jacobi_staged_kernel<double2>, jobs, st, slots, idx, mode, phase, max_sweeps, b,
                              status, counters);
}
}  // namespace wqc
