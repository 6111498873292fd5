// QR of a Jacobi task's working matrix, so that the Jacobi runs on R^H.
#include <cooperative_groups.h>

#include "common.cuh"
#include "jacobi_device.cuh"
#include "split_kernels.cuh"

namespace cg = cooperative_groups;

namespace wqc {

// ---------------------------------------------------------------------------
// X P = Q R for the tall working matrix X (M x N, dust-zeroed), P ordering the
// columns by descending norm, Householder reflectors on a cluster.  Only R is
// kept: A = P R^H (N x N) goes to the slot, and the Jacobi orthogonalises A's
// columns instead of X's (Drmac and Veselic, SIAM J. Matrix Anal. Appl. 29
// (2008) 1322).  A = P (V' Sigma U'^H)^H, so its singular values are X's and
// its left singular vectors are X's right ones: the Jacobi's W then holds
// X's right vectors times sigma, and the cut recovers X's left side.
//
// Why: one-sided Jacobi on X itself takes 12-19 sweeps on the two-site
// matrices of random circuits (up to 30 on steeply graded ones); on the
// triangular factor the columns are near their final order and orthogonality,
// and it takes 8-11.  A tall X also loses its extra rows, and columns beyond
// its rank come out as noise-level columns of A, which the Jacobi leaves out.
//
// Column j of X P lives in the registers of one warp (rows lane + 32 k), NC
// columns per warp, each CTA a panel of NC NW consecutive columns.  The panels
// are factored one after another; a finished panel's reflectors reach the CTAs
// to its right through L2, behind one cluster barrier.  (Broadcasting every
// column through distributed shared memory instead took 8500 cycles a column
// at 256 x 256: one SM feeds all the others.)  A column's step is bound by
// its chain and by the FP64 pipe, so it is cut to one barrier and one
// reduction: the owner publishes the raw column x, and every warp forms
// ||x||^2 and <x, a_j> together; the reflector I - f v v^H (v = x +
// phase(alpha) ||x|| e_c, f = 1 / (||x||^2 + |alpha| ||x||), Hermitian, so R's
// diagonal is complex) follows from those sums without normalising first.
// ---------------------------------------------------------------------------
namespace {

// Warp totals of n values, every lane receiving all of them.  Halving: each
// level hands half of the values to the other half of the lanes, so eight
// values take 9 adds instead of 40.  n divides 32.
template <int n>
__device__ __forceinline__ void warp_totals(double (&v)[n], int lane) {
    static_assert(n == 2 || n == 4 || n == 8, "a power of two");
    int width = 16;
#pragma unroll
    for (int m = n / 2; m >= 1; m /= 2) {
        const bool upper = lane & width;
#pragma unroll
        for (int i = 0; i < n / 2; ++i)
            if (i < m) {
                const double keep = upper ? v[i + m] : v[i], give = upper ? v[i] : v[i + m];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, width);
            }
        width >>= 1;
    }
    for (int o = width; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    // Value i ended on the lanes whose top bits, first level first, spell i.
    const double mine = v[0];
#pragma unroll
    for (int i = 0; i < n; ++i) v[i] = __shfl_sync(0xffffffffu, mine, 32 / n * i);
}

// Column `slot` of a warp's registers into shared memory.  The branches are
// told apart by hand: merged into one indexed copy they would move the columns
// to local memory.
template <int s, int NC, int KR>
__device__ __forceinline__ void publish(const double2 (&a)[NC][KR], int slot, double2* to, int lane) {
    if (slot == s) {
        asm volatile("// slot %0" ::"n"(s));
#pragma unroll
        for (int k = 0; k < KR; ++k) to[lane + 32 * k] = a[s][k];
    }
    if constexpr (s + 1 < NC) publish<s + 1>(a, slot, to, lane);
}

}  // namespace

template <int KR, int NC, int NW>
__global__ void __launch_bounds__(NW * 32) jacobi_qr_kernel(const SplitJob* jobs, SplitState* st,
                                                            const SlotBuffers* slots, const int* idx, int mode,
                                                            int* status) {
    constexpr int LD = 32 * KR, kPer = NC * NW, kThreads = NW * 32;
    constexpr int kSums = NC == 1 ? 4 : 8;  // re, im of every product, then ||x||^2
    constexpr int kDots = 2 * NC;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const int j = jacobi_entry_job(idx[blockIdx.x / cluster.num_blocks()]);
    const SplitState S = st[j];
    if (!jacobi_active(S, mode) || !jacobi_preconditioned(S, mode)) return;
    const SplitJob& J = jobs[j];
    const SlotBuffers Bf = slots[J.slot];
    const double2* src;
    int sr, sc, ld, rows_of_src;
    jacobi_task(J, S, Bf, mode, src, sr, sc, ld, rows_of_src);
    const int M = rows_of_src ? sc : sr;
    const int N = rows_of_src ? sr : sc;
    const int panels = (N + kPer - 1) / kPer;
    const int C = min(panels, int(cluster.num_blocks()));  // CTAs that hold columns; the others leave
    if (M > LD) {  // a launch shape this task does not fit (uniform)
        if (threadIdx.x == 0 && rank == 0) atomicOr(status, kStatusBadShape);
        return;
    }
    if (rank >= C) return;
    extern __shared__ __align__(16) double2 panel[];  // a panel's columns or reflectors, kPer x LD
    __shared__ double norms[kJacobiQrMax];
    __shared__ int order[kJacobiQrMax];
    __shared__ double red[NW];
    __shared__ double part;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    auto src_at = [&](int i, int col) -> double2 {
        return rows_of_src ? cconj(src[size_t(col) * ld + i]) : src[size_t(i) * ld + col];
    };
    auto sync = [&]() {
        if (C > 1)
            cluster.sync();
        else
            __syncthreads();
    };
    sync();  // every CTA has started: its shared memory may be stored into
    // Squared column norms, on every CTA; the order of the columns.
    for (int col = rank * NW + wid; col < N; col += C * NW) {
        double s = 0;
        for (int i = lane; i < M; i += 32) s += cnorm2(src_at(i, col));
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane < C) *cluster.map_shared_rank(&norms[col], lane) = s;
    }
    sync();
    double fro2 = 0;
    for (int c = lane; c < N; c += 32) fro2 += norms[c];
    for (int o = 16; o > 0; o >>= 1) fro2 += __shfl_xor_sync(0xffffffffu, fro2, o);
    // Every place of `order` is written once: a NaN among the norms (and so in
    // their sum) leaves no ranks, and the columns stay where they are; the
    // result is rejected later.
    const bool ranked = fro2 == fro2;
    for (int c = tid; c < N; c += NW * 32) {
        const double nc = norms[c];
        int r = 0;
        for (int i = 0; i < N; ++i) r += (norms[i] > nc || (norms[i] == nc && i < c)) ? 1 : 0;
        order[ranked ? r : c] = c;
    }
    __syncthreads();
    const double dust = sqrt(fro2) * kDustRel;
    const double dust2 = dust * dust;
    double2 a[NC][KR];
    double chk = 0;
    double2* refl = Bf.omega;  // reflector c at refl + c M (omega and y0, not in use by now)
    double2* out = jacobi_pre_matrix(Bf, mode);
    // A panel per CTA at a time; a matrix of more columns than the cluster
    // holds goes in groups of C panels, each group first taking the
    // reflectors of all before it.
    for (int group = 0; group < panels; group += C) {
        const int first = (group + rank) * kPer;
#pragma unroll
        for (int s = 0; s < NC; ++s) {
            const int pos = first + s * NW + wid;
            const int col = pos < N ? order[pos] : 0;
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                const int i = lane + 32 * k;
                double2 x = pos < N && i < M ? src_at(i, col) : cmake(0, 0);
                if (cnorm2(x) < dust2) x = cmake(0, 0);
                chk += cnorm2(x);
                a[s][k] = x;
            }
        }
        for (int p = 0; p < min(panels, group + C); ++p) {
            const int c0 = p * kPer, c1 = min(N, c0 + kPer), q = p - group;
            if (q >= 0) {
                if (rank != q && p + 1 < panels) sync();  // panel p is factored
                if (rank < q) continue;
            }
            if (rank > q) {
                if (first >= N) continue;
                // The panel's reflectors, then each applied in turn; no barriers,
                // every warp has its own columns.
                for (int e = tid; e < (c1 - c0) * LD; e += kThreads) {
                    const int i = e % LD;
                    panel[e] = i < M ? __ldcg(refl + size_t(c0 + e / LD) * M + i) : cmake(0, 0);
                }
                for (int c = c0 + tid; c < c1; c += kThreads) norms[c] = __ldcg(Bf.sigma + c);
                __syncthreads();
                for (int c = c0; c < c1; ++c) {
                    const double f = norms[c];
                    if (f == 0.0) continue;
                    const double2* v = panel + (c - c0) * LD;
                    const int ck = c >> 5;
                    double2 x[KR];
                    double dots[NC == 1 ? 2 : kSums];
#pragma unroll
                    for (int i = 0; i < (NC == 1 ? 2 : kSums); ++i) dots[i] = 0;
#pragma unroll
                    for (int k = 0; k < KR; ++k) {
                        if (k < ck) continue;  // rows above the diagonal
                        x[k] = v[lane + 32 * k];
#pragma unroll
                        for (int s = 0; s < NC; ++s) {
                            double2 d = cmake(dots[2 * s], dots[2 * s + 1]);
                            cfma_conj(d, x[k], a[s][k]);
                            dots[2 * s] = d.x;
                            dots[2 * s + 1] = d.y;
                        }
                    }
                    warp_totals(dots, lane);
#pragma unroll
                    for (int s = 0; s < NC; ++s) {
                        const double2 w = cmake(f * dots[2 * s], f * dots[2 * s + 1]);
#pragma unroll
                        for (int k = 0; k < KR; ++k) {
                            if (k < ck) continue;
                            a[s][k].x = fma(-x[k].x, w.x, fma(x[k].y, w.y, a[s][k].x));
                            a[s][k].y = fma(-x[k].x, w.y, fma(-x[k].y, w.x, a[s][k].y));
                        }
                    }
                }
                __syncthreads();  // the next panel overwrites this one
                continue;
            }
            for (int c = c0; c < c1; ++c) {
                const int local = c - c0;
                double2* pub = panel + local * LD;
                if (wid == local % NW) publish<0>(a, local / NW, pub, lane);
                __syncthreads();
                // Warps whose columns are all finished leave the FP64 pipe to
                // the others (the step is bound by it while all take part).
                if (first + (NC - 1) * NW + wid < c || first + wid >= N) continue;
                const int ck = c >> 5, cl = c & 31;
                double2 x[KR];
                double sums[kSums];
#pragma unroll
                for (int i = 0; i < kSums; ++i) sums[i] = 0;
#pragma unroll
                for (int k = 0; k < KR; ++k) {
                    if (k < ck) continue;
                    const int row = lane + 32 * k;
                    x[k] = row > c ? pub[row] : cmake(0, 0);
                    sums[kDots] = fma(x[k].x, x[k].x, fma(x[k].y, x[k].y, sums[kDots]));
#pragma unroll
                    for (int s = 0; s < NC; ++s) {
                        double2 d = cmake(sums[2 * s], sums[2 * s + 1]);
                        cfma_conj(d, x[k], a[s][k]);
                        sums[2 * s] = d.x;
                        sums[2 * s + 1] = d.y;
                    }
                }
                warp_totals(sums, lane);
                const double tail = sums[kDots];
                // Already triangular here, or below what squares can hold.
                const bool trivial = tail <= 1e-290;
                double f = 0;
                if (!trivial) {
                    const double2 alpha = pub[c];
                    const double al2 = cnorm2(alpha);
                    const double s2 = tail + al2;
                    const double nrm = s2 * rsqrt(s2);
                    const double ia = al2 > 1e-290 ? rsqrt(al2) : 0.0;
                    const double aabs = al2 * ia;
                    const double2 phase = ia > 0.0 ? cscale(alpha, ia) : cmake(1.0, 0.0);
                    const double2 vc = cscale(phase, aabs + nrm);
                    f = 1.0 / fma(aabs, nrm, s2);
#pragma unroll
                    for (int k = 0; k < KR; ++k)
                        if (k == ck && lane == cl) x[k] = vc;
#pragma unroll
                    for (int s = 0; s < NC; ++s) {
                        const int pos = first + s * NW + wid;
                        if (pos < c || pos >= N) continue;  // a finished column, or none (uniform per warp)
                        if (pos == c) {  // the column itself: R's diagonal
#pragma unroll
                            for (int k = 0; k < KR; ++k)
                                if (k == ck && lane == cl) a[s][k] = cscale(phase, -nrm);
                            continue;
                        }
                        double2 ac = cmake(0, 0);  // the part of <v, a> on the diagonal row
#pragma unroll
                        for (int k = 0; k < KR; ++k)
                            if (k == ck) ac = a[s][k];
                        ac.x = __shfl_sync(0xffffffffu, ac.x, cl);
                        ac.y = __shfl_sync(0xffffffffu, ac.y, cl);
                        double2 w = cmake(sums[2 * s], sums[2 * s + 1]);
                        cfma_conj(w, vc, ac);
                        w = cscale(w, f);
#pragma unroll
                        for (int k = 0; k < KR; ++k) {
                            if (k < ck) continue;
                            a[s][k].x = fma(-x[k].x, w.x, fma(x[k].y, w.y, a[s][k].x));
                            a[s][k].y = fma(-x[k].x, w.y, fma(-x[k].y, w.x, a[s][k].y));
                        }
                    }
                }
                if (p + 1 < panels && wid == local % NW) {  // for the panels to the right
#pragma unroll
                    for (int k = 0; k < KR; ++k) {
                        const int row = lane + 32 * k;
                        if (row < M) refl[size_t(c) * M + row] = k < ck ? cmake(0, 0) : x[k];
                    }
                    if (lane == 0) Bf.sigma[c] = f;
                }
            }
            if (p + 1 < panels) {
                __threadfence();
                sync();
            }
        }
        // A = P R^H, column-major: A[order[j]][i] = conj(R[i][j]).
#pragma unroll
        for (int s = 0; s < NC; ++s) {
            const int pos = first + s * NW + wid;
            if (pos >= N) continue;
            const int row = order[pos];
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                const int i = lane + 32 * k;
                if (i < N) out[size_t(i) * N + row] = i <= pos ? cconj(a[s][k]) : cmake(0, 0);
            }
        }
    }
    // ||X||_F^2 of the dust-zeroed matrix, for the Jacobi's check.
    for (int o = 16; o > 0; o >>= 1) chk += __shfl_xor_sync(0xffffffffu, chk, o);
    if (lane == 0) red[wid] = chk;
    __syncthreads();
    if (tid == 0) {
        double t = 0;
        for (int w = 0; w < NW; ++w) t += red[w];
        part = t;
    }
    sync();
    if (rank == 0 && tid == 0) {
        double t = 0;
        for (int r = 0; r < C; ++r) t += *cluster.map_shared_rank(&part, r);
        st[j].pre_fro2 = t;
    }
    if (C > 1) cluster.sync();  // no CTA leaves while rank 0 reads its shared memory
}

namespace {

using QrKernel = void (*)(const SplitJob*, SplitState*, const SlotBuffers*, const int*, int, int*);

// Instances by row groups, kJacobiQrPerCta columns a CTA.  A step's
// instructions are issued by every warp at about five cycles each, so columns
// are better spread over warps and CTAs than stacked in a warp (256 x 256:
// 0.81 ms with 4 columns in each of 4 warps), as long as two columns' rows fit
// the registers (0.62 ms with one column in each of 16 warps, which spill;
// 0.55 with two in each of 8).
QrKernel qr_kernel(int kr) {
    switch (kr) {
        case 1: return jacobi_qr_kernel<1, 1, 16>;
        case 2: return jacobi_qr_kernel<2, 1, 16>;
        case 4: return jacobi_qr_kernel<4, 1, 16>;
        case 6: return jacobi_qr_kernel<6, 2, 8>;
        case 8: return jacobi_qr_kernel<8, 2, 8>;
        case 12: return jacobi_qr_kernel<12, 2, 8>;
        default: return jacobi_qr_kernel<16, 2, 8>;
    }
}

size_t qr_smem(int kr) { return size_t(kJacobiQrPerCta) * 32 * kr * sizeof(double2); }

}  // namespace

cudaError_t jacobi_qr_attributes() {
    cudaError_t e = cudaSuccess;
    for (int kr : {1, 2, 4, 6, 8, 12, 16}) {
        const void* f = reinterpret_cast<const void*>(qr_kernel(kr));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(qr_smem(kr)));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    return e;
}

cudaError_t launch_jacobi_qr(int kr, int C, int tasks, cudaStream_t stream, const SplitJob* jobs, SplitState* st,
                             const SlotBuffers* slots, const int* idx, int mode, int* status) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tasks * C);
    cfg.blockDim = dim3(kr > 4 ? 256 : 512);
    cfg.dynamicSmemBytes = qr_smem(kr);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, qr_kernel(kr), jobs, st, slots, idx, mode, status);
}

}  // namespace wqc
