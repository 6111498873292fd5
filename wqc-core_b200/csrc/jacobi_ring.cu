// One-sided Hestenes Jacobi SVD of a two-site matrix on a thread-block
// cluster (svd_guard.rs:146-229), columns in registers and shared memory.
#include <cooperative_groups.h>

#include "common.cuh"
#include "jacobi_device.cuh"
#include "split_kernels.cuh"

namespace cg = cooperative_groups;

namespace wqc {

namespace {

// Rotates the columns u and v, both in registers (rows lane + 32 k; rows past
// the column's end are zero).  With kV only the first km row groups enter the
// dot products: the rest hold the accumulated V of the precision form's first
// phase and are rotated along.  Returns false when the pair is left alone.
template <typename T, int KR, bool kV>
__device__ __forceinline__ bool rotate_reg(T (&u)[KR], T (&v)[KR], int km, double tol2, double noise_floor,
                                           bool want_ratio, int lane, JacobiSweep& sw) {
    using R = typename JacobiReal<T>::R;
    R a0 = 0, b0 = 0, gr0 = 0, gi0 = 0, a1 = 0, b1 = 0, gr1 = 0, gi1 = 0;
#pragma unroll
    for (int k = 0; k < KR; k += 2) {
        if (kV && k >= km) break;
        a0 = fma(u[k].x, u[k].x, fma(u[k].y, u[k].y, a0));
        b0 = fma(v[k].x, v[k].x, fma(v[k].y, v[k].y, b0));
        gr0 = fma(u[k].x, v[k].x, fma(u[k].y, v[k].y, gr0));
        gi0 = fma(u[k].x, v[k].y, fma(-u[k].y, v[k].x, gi0));
        if (k + 1 < KR && (!kV || k + 1 < km)) {
            a1 = fma(u[k + 1].x, u[k + 1].x, fma(u[k + 1].y, u[k + 1].y, a1));
            b1 = fma(v[k + 1].x, v[k + 1].x, fma(v[k + 1].y, v[k + 1].y, b1));
            gr1 = fma(u[k + 1].x, v[k + 1].x, fma(u[k + 1].y, v[k + 1].y, gr1));
            gi1 = fma(u[k + 1].x, v[k + 1].y, fma(-u[k + 1].y, v[k + 1].x, gi1));
        }
    }
    a0 += a1;
    b0 += b1;
    gr0 += gr1;
    gi0 += gi1;
    warp_sum4(a0, b0, gr0, gi0, lane);
    double c64, wr64, wi64;
    if (!jacobi_params(a0, b0, gr0, gi0, tol2, noise_floor, want_ratio, sw, c64, wr64, wi64)) return false;
    const R wr = R(wr64), wi = R(wi64), c = R(c64);
#pragma unroll
    for (int k = 0; k < KR; ++k) {
        T p, q;
        p.x = fma(c, u[k].x, -fma(wr, v[k].x, wi * v[k].y));
        p.y = fma(c, u[k].y, -fma(wr, v[k].y, -wi * v[k].x));
        q.x = fma(wr, u[k].x, fma(-wi, u[k].y, c * v[k].x));
        q.y = fma(wr, u[k].y, fma(wi, u[k].x, c * v[k].y));
        u[k] = p;
        v[k] = q;
    }
    return true;
}

}  // namespace

// ---------------------------------------------------------------------------
// The tall working matrix W (M x N, N padded to 2 C b columns) is held by C
// CTAs (a power of two) of one cluster as 2C blocks of b columns, every
// column padded to 32 KR rows.  CTA r holds a top block, one column in the
// registers of each of its b warps, and a bottom block in shared memory.
//
// A sweep rotates the pairs inside every block, then the pairs between
// blocks by halving: in a group of g CTAs the bottom blocks go once round the
// ring of the group, so that every top block meets every bottom block in g
// steps; then the group's top blocks move to its lower half of CTAs and its
// bottom blocks to the upper half (half of each becoming the other kind), and
// both halves go on by themselves, down to g = 1.  That is 2C - 1 block steps
// of b rounds, every pair of columns once a sweep.  In round k of a step warp
// i rotates its top column with bottom column (i + k) mod b.
//
// What bounds a round is its chain (load, dot products, warp sum, two
// reciprocal square roots, update, CTA barrier), not the FP64 pipe, so what
// this layout takes off the chain is traffic: a block moves only once per
// step (the circle method moved two), and it moves in the step's last round,
// when each warp stores its rotated column straight into the next CTA's
// spare buffer; one cluster barrier ends the step.  The spare buffer is the
// one that CTA finished reading a step ago, before that barrier.
//
// Right rotations are not accumulated: at convergence W = X V = U Sigma, and
// the cut recovers the other side from W and X (recover_gemm_kernel).  The
// precision form's first phase carries V as rows under W.
// ---------------------------------------------------------------------------
template <typename T, int KR, bool kV>
__global__ void __launch_bounds__(jacobi_ring_warps(KR, sizeof(T)) * 32) jacobi_ring_kernel(
    const SplitJob* jobs, SplitState* st, const SlotBuffers* slots, const int* idx, int mode, int phase,
    int max_sweeps, int* status, unsigned long long* counters) {
    constexpr bool kF64 = sizeof(T) == sizeof(double2);
    constexpr int LD = 32 * KR;  // rows of a stored column
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int entry = idx[blockIdx.x / cluster.num_blocks()];
    const int j = jacobi_entry_job(entry);
    // The task's own cluster size; the launch's is the largest of its tasks.
    // CTAs past it leave at once (cluster barriers wait for non-exited
    // threads only, and nobody reads their shared memory).
    const int C = jacobi_entry_cluster(entry);
    if (rank >= C) return;
    const SplitState S = st[j];
    if (!jacobi_active(S, mode)) return;  // uniform over the task's CTAs
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
    const int M = X.M, N = X.N;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nthreads = blockDim.x, nwarps = nthreads >> 5;
    const int b = (N + 2 * C - 1) / (2 * C);
    const int km = (M + 31) / 32;          // row groups of W
    const int vrows = kV ? N : 0;          // V's rows start at row 32 km
    if (b > nwarps || km + (vrows + 31) / 32 > KR) {  // a launch shape this task does not fit (uniform)
        if (tid == 0 && rank == 0) atomicOr(status, kStatusBadShape);
        return;
    }
    const bool colmajor = X.contiguous();
    const bool dusted = pre || phase == kPhaseFinish;  // entries already dust-zeroed

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(smem_raw);
    const size_t blk = size_t(b) * LD;
    __shared__ JacobiCtl ctl;
    __shared__ double red[32];
    __shared__ int ids[2];  // block held by each buffer
    auto column = [&](int buffer, int c) { return smem + size_t(buffer) * blk + size_t(c) * LD; };

    // Frobenius norm over the columns this CTA loads, then over the cluster.
    double part = 0;
    for (int half = 0; half < 2; ++half) {
        const int id = half * C + rank;
        for (int e = tid; e < b * M; e += nthreads) {
            int c, i;
            if (colmajor) { c = e / M; i = e % M; } else { i = e / b; c = e % b; }
            const int col = id * b + c;
            if (col < N) part += cnorm2(X.at(i, col));
        }
    }
    const double cta_part = block_total(part, red);
    if (tid == 0) ctl.fro_part = cta_part;
    cluster.sync();
    double fro2 = 0;
    for (int r = 0; r < C; ++r) fro2 += cluster.map_shared_rank(&ctl, r)->fro_part;
    const double dust = sqrt(fro2) * kDustRel;
    const double dust2 = dust * dust;
    double chk_in = 0, chk_out = 0;
    // Load W (dust-zeroed; padding rows and columns zero): buffer 0 the
    // bottom block, buffer 1 the block that goes to the registers.
    for (int half = 0; half < 2; ++half) {
        const int id = half * C + rank;
        if (tid == 0) ids[half] = id;
        if (LD > M)
            for (int e = tid; e < b * (LD - M); e += nthreads) {
                const int c = e / (LD - M), i = M + e % (LD - M);
                const bool one = kV && i >= 32 * km && i - 32 * km == id * b + c && id * b + c < N;
                column(half, c)[i] = to_store<T>(cmake(one ? 1.0 : 0.0, 0.0));
            }
        for (int e = tid; e < b * M; e += nthreads) {
            int c, i;
            if (colmajor) { c = e / M; i = e % M; } else { i = e / b; c = e % b; }
            const int col = id * b + c;
            double2 x = col < N ? X.at(i, col) : cmake(0, 0);
            if (!dusted && cnorm2(x) < dust2) x = cmake(0, 0);
            chk_in += cnorm2(x);
            column(half, c)[i] = to_store<T>(x);
        }
    }
    const double tol2 = kF64 ? kJacobiTol2 : kJacobiTol2Fp32;
    const double noise_floor = (kF64 ? 1e-30 : 1e-12) * fro2;  // squared column norm: 1e-15 (1e-6) of ||W||_F
    const bool mine = wid < b;
    T u[KR], v[KR];
    auto load = [&](T (&x)[KR], const T* col) {
#pragma unroll
        for (int k = 0; k < KR; ++k) x[k] = col[lane + 32 * k];
    };
    auto store = [&](T* col, const T (&x)[KR]) {
#pragma unroll
        for (int k = 0; k < KR; ++k) col[lane + 32 * k] = x[k];
    };
    int sweep = 0, last_rot = 0;
    unsigned long long last_relmax_bits = 0ull;
    bool converged = false;
    int cur = 0;     // buffer of the bottom block
    int top_id = 0;  // block in the registers
    __syncthreads();
    for (; sweep < max_sweeps; ++sweep) {
        if (tid == 0) {
            ctl.rot = 0;
            ctl.ecos = ctl.esin = -8192;
            ctl.relmax_bits = 0ull;
        }
        JacobiSweep my;
        const bool want_ratio = sweep == max_sweeps - 1;
        if (sweep > 0) {  // the top block into the spare buffer
            if (mine) store(column(cur ^ 1, wid), u);
            if (tid == 0) ids[cur ^ 1] = top_id;
            __syncthreads();
        }
        // Pairs inside each block (circle method; an odd b has a dummy position).
        const int be = b + (b & 1);
        for (int step = 0; step < be - 1; ++step) {
            for (int pq = wid; pq < be; pq += nwarps) {
                const int i = pq < be / 2 ? pq : pq - be / 2;
                const int e1 = circle_at(i, step, be), e2 = circle_at(be - 1 - i, step, be);
                if (e1 < b && e2 < b) {
                    T* p = column(pq < be / 2 ? 1 : 0, e1);
                    T* q = column(pq < be / 2 ? 1 : 0, e2);
                    load(u, p);
                    load(v, q);
                    if (rotate_reg<T, KR, kV>(u, v, km, tol2, noise_floor, want_ratio, lane, my)) {
                        store(p, u);
                        store(q, v);
                    }
                }
            }
            __syncthreads();
        }
        cur = 0;
        top_id = ids[1];
        if (mine) load(u, column(1, wid));
        cluster.sync();  // every CTA has read its buffer 1: it may be stored into from outside
        // Pairs between blocks.
        for (int g = C; g >= 1; g >>= 1) {
            const int at = rank & (g - 1), base = rank - at;
            const bool lower = at < g / 2;
            for (int step = 0; step < g; ++step) {
                const bool regroup = step == g - 1;
                for (int k = 0; k < b; ++k) {
                    int c = wid + k;
                    if (c >= b) c -= b;
                    T* q = column(cur, c);
                    bool rotated = false;
                    if (mine) {
                        load(v, q);
                        rotated = rotate_reg<T, KR, kV>(u, v, km, tol2, noise_floor, want_ratio, lane, my);
                    }
                    if (k < b - 1) {
                        if (rotated) store(q, v);
                        __syncthreads();
                        continue;
                    }
                    // Last round: the bottom column goes where the next step needs it.
                    if (!regroup) {
                        const int to = base + ((at + 1) & (g - 1));
                        if (mine) store(cluster.map_shared_rank(column(cur ^ 1, c), to), v);
                        if (tid == 0) *cluster.map_shared_rank(&ids[cur ^ 1], to) = ids[cur];
                    } else if (g > 1) {
                        if (lower) {  // bottom block to the upper half, as a top block
                            if (mine) store(cluster.map_shared_rank(column(cur ^ 1, c), rank + g / 2), v);
                            if (tid == 0) *cluster.map_shared_rank(&ids[cur ^ 1], rank + g / 2) = ids[cur];
                        } else {  // top block to the lower half, as a bottom block
                            if (mine) {
                                if (rotated) store(q, v);
                                store(cluster.map_shared_rank(column(cur ^ 1, wid), rank - g / 2), u);
                            }
                            if (tid == 0) *cluster.map_shared_rank(&ids[cur ^ 1], rank - g / 2) = top_id;
                        }
                    } else if (rotated) {
                        store(q, v);
                    }
                }
                if (g == 1) {
                    __syncthreads();
                    break;
                }
                cluster.sync();
                if (!regroup) {
                    cur ^= 1;
                } else {
                    if (lower) {
                        cur ^= 1;
                    } else {
                        if (mine) load(u, column(cur ^ 1, wid));
                        top_id = ids[cur ^ 1];
                    }
                    // The upper half's spare buffer has been read before the
                    // next store from outside.
                    if (g > 2) cluster.sync();
                }
            }
        }
        // Cluster-wide findings decide convergence.
        jacobi_report(ctl, my, lane);
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
        last_rot = total;
        last_relmax_bits = relmax_bits;
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
                status[2] = last_rot;
                status[3] = int(last_relmax_bits >> 32);
                status[4] = int(last_relmax_bits & 0xffffffffull);
            }
        }
        if (phase != kPhaseFp32V) atomicAdd(counters + 0, 1ull);
        atomicAdd(counters + (phase == kPhaseFp32V ? 2 : 1), (unsigned long long)(converged ? sweep + 1 : sweep));
    }
    // The bottom block's columns join the top block's in registers: v from u's place.
    const int bot_id = ids[cur];
    if (mine) load(v, column(cur, wid));
    if constexpr (kV) {
        // The accumulated V (FP64) for the finishing phase, and ||X||_F^2
        // for its dust zeroing of X.
        for (int half = 0; half < 2; ++half) {
            const int col = (half ? bot_id : top_id) * b + wid;
            if (!mine || col >= N) continue;
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                const int r = lane + 32 * (k - km);
                if (k >= km && r < N) Bf.z[size_t(col) * N + r] = to_f64(half ? v[k] : u[k]);
            }
        }
        if (rank == 0 && tid == 0) st[j].fro2 = fro2;
        // (The last sweep's barrier ended every access to other CTAs' memory.)
    } else {
        // Write back: W columns and column norms (FP64 in both forms).
        for (int half = 0; half < 2; ++half) {
            const int col = (half ? bot_id : top_id) * b + wid;
            if (!mine || col >= N) continue;
            double s2 = 0;
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                const double2 x = to_f64(half ? v[k] : u[k]);
                const int r = lane + 32 * k;
                s2 = fma(x.x, x.x, fma(x.y, x.y, s2));
                if (r < M) Bf.w[size_t(col) * M + r] = x;
            }
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (lane == 0) {
                Bf.sigma[col] = jacobi_sigma(s2, fro2, mode);
                chk_out += s2;
            }
        }
        // Factorisation check over the cluster.
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

namespace {

using RingKernel = void (*)(const SplitJob*, SplitState*, const SlotBuffers*, const int*, int, int, int, int*,
                            unsigned long long*);

// The instance for columns of `kr` row groups (jacobi_ring_kr).
RingKernel ring_kernel(bool fp32, int kr) {
    if (fp32) {
        switch (kr) {
            case 2: return jacobi_ring_kernel<float2, 2, true>;
            case 4: return jacobi_ring_kernel<float2, 4, true>;
            case 8: return jacobi_ring_kernel<float2, 8, true>;
            case 16: return jacobi_ring_kernel<float2, 16, true>;
            default: return jacobi_ring_kernel<float2, 24, true>;
        }
    }
    switch (kr) {
        case 1: return jacobi_ring_kernel<double2, 1, false>;
        case 2: return jacobi_ring_kernel<double2, 2, false>;
        case 3: return jacobi_ring_kernel<double2, 3, false>;
        case 4: return jacobi_ring_kernel<double2, 4, false>;
        case 6: return jacobi_ring_kernel<double2, 6, false>;
        case 8: return jacobi_ring_kernel<double2, 8, false>;
        default: return jacobi_ring_kernel<double2, 12, false>;
    }
}

}  // namespace

std::vector<const void*> jacobi_ring_kernels() {
    std::vector<const void*> all;
    for (int kr : {2, 4, 8, 16, 24}) all.push_back(reinterpret_cast<const void*>(ring_kernel(true, kr)));
    for (int kr : {1, 2, 3, 4, 6, 8, 12}) all.push_back(reinterpret_cast<const void*>(ring_kernel(false, kr)));
    return all;
}

cudaError_t launch_jacobi(bool fp32, int kr, const cudaLaunchConfig_t& cfg, const SplitJob* jobs, SplitState* st,
                          const SlotBuffers* slots, const int* idx, int mode, int phase, int max_sweeps, int* status,
                          unsigned long long* counters) {
    return cudaLaunchKernelEx(&cfg, ring_kernel(fp32, kr), jobs, st, slots, idx, mode, phase, max_sweeps, status,
                              counters);
}

}  // namespace wqc
