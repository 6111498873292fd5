// Device code shared by the one-sided Jacobi SVD kernels: the pair rotation,
// the tasks' operands and the factorisation check's constants.
#pragma once

#include "common.cuh"
#include "split_kernels.cuh"

namespace wqc {

struct JacobiCtl {
    int rot;                         // rotations of this sweep
    int ecos, esin;                  // binary exponents of this sweep's largest cos^2 and sin^2 (JacobiSweep)
    unsigned long long relmax_bits;  // last allowed sweep: largest squared |gamma|^2 / (alpha beta) (double bits)
    double fro_part;
    double chk_in, chk_out;  // this CTA's share of ||X||_F^2 (after dust zeroing) and of sum sigma^2
};

// The Frobenius part of the reference's factorisation check (svd_reproduces,
// svd_guard.rs:234-255): sum sigma^2 must equal ||X||_F^2 of the dust-zeroed
// matrix to SVD_CHECK_TOL = 1e-9 relative (plus 1e-28).  The precision form's
// complex64 columns carry ~1e-6 of rounding, so it is held to 1e-4.  The
// probe-vector part needs V, which this Jacobi does not accumulate.
constexpr double kSvdCheckTol = 1e-9;
constexpr double kSvdCheckTolFp32 = 1e-4;

// Pairs count as orthogonal at |gamma| <= tol sqrt(alpha beta), just above
// the rounding of an M <= 512 dot product (sqrt(M) eps: 5e-15 in FP64, 3e-6
// in FP32), so the sweeps stop and the singular values are exact to second
// order.  Squared.
constexpr double kJacobiTol2 = 1e-28, kJacobiTol2Fp32 = 1.6e-11;

// What a sweep learns from its pairs: rotations, and of the rotated pairs the
// largest cos^2 = |gamma|^2 / (alpha beta) they entered with and the largest
// sin^2 of a rotation, as binary exponents (integer compares off the
// rotation's chain, in place of a division on it).  The ratio itself is taken
// on the last allowed sweep, where the error message reports it.
struct JacobiSweep {
    int rot = 0;
    int ecos = -8192, esin = -8192;
    double relmax = 0.0;
};

// A sweep ends the iteration when it leaves every pair orthogonal: a pair it
// made orthogonal is spoiled by later rotations of its columns, by at most
// about (largest sin) x (largest cos of what is mixed in).  With separated
// singular values sin is of cos's size and a cos below 1e-8 leaves 1e-16; but
// in a cluster of equal ones any small gamma turns the pair by a large angle,
// and the sweep would leave what it entered with (1e-9 was seen on the
// doubly degenerate theta of Clifford-like circuits).  FP64: cos < 2^-26.5 and
// sin cos < 2^-50.  The complex64 phase only prepares the FP64 one: cos < 2e-3.
__device__ __forceinline__ bool jacobi_done(bool f64, int rot, int ecos, int esin) {
    if (rot == 0) return true;
    return f64 ? ecos < -53 && ecos + esin < -100 : ecos < -18;
}

// Singular values of an exact SVD at or below 18 eps ||X||_F are reported as
// zero: rounding leaves such values where X has none, their W columns are not
// orthogonal to the others, and one that a state of large norm lifts over the
// absolute cutoff of 1e-12 would enter the cut as a vector (a rank 20 theta of
// norm 1600 kept 250 vectors and a product off by ten times its norm).  At
// norm 1 the bound is 4e-15 and decides nothing.  Squared.
constexpr double kJacobiZero2 = 1.6e-29;
__device__ __forceinline__ double jacobi_sigma(double s2, double fro2, int mode) {
    return mode != kJacobiRsvd && s2 <= kJacobiZero2 * fro2 ? 0.0 : sqrt(s2);
}

__device__ __forceinline__ double block_total(double v, double* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double t = 0;
    for (int w = 0; w < int(blockDim.x >> 5); ++w) t += red[w];
    return t;
}

// Position pos of the circle method on b items after `step` < b - 1 turns.
__device__ __forceinline__ int circle_at(int pos, int step, int b) {
    if (pos == 0) return 0;
    const int v = pos - 1 - step;
    return (v < 0 ? v + b - 1 : v) + 1;
}

// Rotates columns xp, xq (each W then Z, `len` entries, W part `M`).  All
// lanes compute bitwise-identical reductions (xor butterfly), so the branch is
// warp-uniform.
//
// Two guards keep every applied rotation unitary and the sweep finite:
// |gamma| is taken with hypot when |gamma|^2 nears the subnormal range, so
// the phase stays of unit modulus; and a pair whose smaller column has
// alpha <= floor = (1e-15 ||W||_F)^2 (FP32 columns: (1e-6 ||W||_F)^2) is left
// alone.  Such a column is at the storage's rounding level: its direction is
// noise, rotating it against another column changes nothing above
// floor * ||W||_F^2, and rotating it anyway lets exactly parallel columns (a
// rank-deficient theta) be re-rotated every sweep until their products go
// subnormal, and pairs of noise columns keep |gamma|/sqrt(alpha beta) near
// 1e-8 forever (seen on a 256 x 144 range-finder matrix of the 50-qubit
// circuit, which then never met the stop test).
//
// The columns are complex128 (double2) in the plain form and complex64
// (float2) in the precision form.  The precision form accumulates the dot
// products and applies the rotation in FP32; the rotation parameters, the
// tests against tol and the noise floor, and the convergence measure are
// FP64 in both.
template <typename T>
struct JacobiReal;
template <>
struct JacobiReal<double2> {
    using R = double;
};
template <>
struct JacobiReal<float2> {
    using R = float;
};

// Warp sums of four values, every lane receiving the same four totals (so
// branches on them stay warp-uniform).  Instead of four butterflies (20
// shuffles) the first two levels split the values between the lane halves
// (lanes with bit 4 clear keep a, b and pass g, h; then bit 3 picks one of
// the two), three more levels finish one value per quarter of the warp, and
// four broadcasts from lanes 0, 8, 16, 24 hand out the totals: 10 shuffles,
// on the dependent chain of every rotation round.
template <typename R>
__device__ __forceinline__ void warp_sum4(R& a, R& b, R& g, R& h, int lane) {
    const bool hi = lane & 16;
    R k0 = hi ? g : a, k1 = hi ? h : b;
    k0 += __shfl_xor_sync(0xffffffffu, hi ? a : g, 16);
    k1 += __shfl_xor_sync(0xffffffffu, hi ? b : h, 16);
    const bool b3 = lane & 8;
    R v = b3 ? k1 : k0;
    v += __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    a = __shfl_sync(0xffffffffu, v, 0);
    b = __shfl_sync(0xffffffffu, v, 8);
    g = __shfl_sync(0xffffffffu, v, 16);
    h = __shfl_sync(0xffffffffu, v, 24);
}

// A warp's findings into its CTA's control block.
__device__ __forceinline__ void jacobi_report(JacobiCtl& ctl, const JacobiSweep& sw, int lane) {
    if (lane != 0) return;
    if (sw.rot) atomicAdd(&ctl.rot, sw.rot);
    atomicMax(&ctl.ecos, sw.ecos);
    atomicMax(&ctl.esin, sw.esin);
    if (sw.relmax > 0.0) atomicMax(&ctl.relmax_bits, (unsigned long long)__double_as_longlong(sw.relmax));
}

// Rotation parameters from alpha = |p|^2, beta = |q|^2, gamma = <p, q>:
// returns false when the pair is left alone (noise-level column, or already
// orthogonal to tol), else c and w = s * phase of the rephased rotation
// (svd_guard.rs:189-197) xp' = c xp - conj(w) xq, xq' = w xp + c xq.
//
// With d = (beta - alpha) / 2 and r = sqrt(d^2 + |gamma|^2) the half-angle
// form is c^2 = (1 + |d| / r) / 2 and w = sign(d) gamma / (2 r c): two
// dependent reciprocal square roots (85 cycles each on B200) and no
// division, where the tangent form took three and its phase a fourth.
__device__ __forceinline__ bool jacobi_params(double a, double bb, double gr, double gi, double tol2,
                                              double noise_floor, bool want_ratio, JacobiSweep& sw, double& c,
                                              double& wr, double& wi) {
    const double g2 = fma(gr, gr, gi * gi);
    const double ab = a * bb;
    // Left alone: the smaller column is at the storage's rounding level, or
    // the pair is orthogonal to tol.  (A NaN is rotated, and rejected later.)
    if (fmin(a, bb) <= noise_floor || g2 <= tol2 * ab) return false;
    if (want_ratio) sw.relmax = fmax(sw.relmax, g2 / ab);
    const double d = 0.5 * (bb - a);
    const double r2 = fma(d, d, g2);
    if (g2 > 1e-290) {
        const double ir = rsqrt(r2);
        const double c2 = fma(0.5 * fabs(d), ir, 0.5);
        const double ic = rsqrt(c2);
        c = c2 * ic;
        const double f = copysign(0.5 * ir * ic, d);
        wr = gr * f;
        wi = gi * f;
    } else {  // |gamma|^2 near the subnormal range: hypot keeps the rotation unitary
        const double r = hypot(d, hypot(gr, gi));
        c = sqrt(0.5 + 0.5 * (fabs(d) / r));
        const double f = copysign(0.5 / c, d);
        wr = (gr / r) * f;
        wi = (gi / r) * f;
    }
    ++sw.rot;
    auto exponent = [](double x) { return __double2hiint(x) >> 20; };
    sw.ecos = max(sw.ecos, exponent(g2) - exponent(ab));
    sw.esin = max(sw.esin, exponent(fma(wr, wr, wi * wi)) - 1023);
    return true;
}

// The original working matrix X of a task: column j of X (M x N, M >= N) is
// column j of src, or with rows_of_src the conjugate of src's row j.
__device__ __forceinline__ void jacobi_task(const SplitJob& J, const SplitState& S, const SlotBuffers& B, int mode,
                                            const double2*& src, int& sr, int& sc, int& ld, int& rows_of_src) {
    if (mode == kJacobiRsvd) {  // W = B^H, B is ell x cols row-major
        src = B.b;
        sr = S.ell;
        sc = S.cols;
        ld = S.cols;
        rows_of_src = 1;
    } else {  // exact: theta (rows >= cols) or theta^H
        src = B.theta;
        sr = S.rows;
        sc = S.cols;
        ld = S.cols;
        rows_of_src = S.rows < S.cols ? 1 : 0;
    }
}

__device__ __forceinline__ bool jacobi_active(const SplitState& S, int mode) {
    if (mode == kJacobiRsvd) return S.use_rsvd != 0;
    // The exact path's two modes never overlap: prepare sets path EXACT, and a
    // fallback changes a range-finder split's path to RSVD_FALLBACK only.
    if (mode == kJacobiExact) return S.need_exact != 0 && S.path == WQC_SPLIT_EXACT;
    return S.need_exact != 0 && S.path == WQC_SPLIT_RSVD_FALLBACK;
}

// Whether the task's Jacobi runs on A = P R^H (jacobi_qr.cu), N x N and
// column-major in a buffer that nothing else of the split uses by then: Y
// once Q is formed; the range finder's Q and B for the splits that are not
// its own (2 R E >= R^2 entries).  W then holds X's right vectors.
__device__ __forceinline__ bool jacobi_preconditioned(const SplitState& S, int mode) {
    return mode == kJacobiRsvd ? S.pre_rsvd != 0 : S.pre_exact != 0;
}
__device__ __forceinline__ double2* jacobi_pre_matrix(const SlotBuffers& B, int mode) {
    return mode == kJacobiRsvd ? B.y : B.q;
}

// The matrix whose columns a Jacobi task orthogonalises.
struct JacobiMatrix {
    const double2* p;
    int M, N, ld;
    int by_rows;  // column j is the conjugate of row j
    int by_cols;  // column-major
    __device__ __forceinline__ double2 at(int i, int col) const {
        if (by_cols) return p[size_t(col) * ld + i];
        return by_rows ? cconj(p[size_t(col) * ld + i]) : p[size_t(i) * ld + col];
    }
    __device__ __forceinline__ bool contiguous() const { return by_cols || by_rows; }
};
__device__ __forceinline__ JacobiMatrix jacobi_matrix(const SplitJob& J, const SplitState& S, const SlotBuffers& B,
                                                      int mode) {
    JacobiMatrix x;
    int sr, sc;
    jacobi_task(J, S, B, mode, x.p, sr, sc, x.ld, x.by_rows);
    x.M = x.by_rows ? sc : sr;
    x.N = x.by_rows ? sr : sc;
    x.by_cols = 0;
    if (jacobi_preconditioned(S, mode)) {
        x.p = jacobi_pre_matrix(B, mode);
        x.M = x.ld = x.N;
        x.by_rows = 0;
        x.by_cols = 1;
    }
    return x;
}

template <typename T>
__device__ __forceinline__ T to_store(double2 x);
template <>
__device__ __forceinline__ double2 to_store<double2>(double2 x) {
    return x;
}
template <>
__device__ __forceinline__ float2 to_store<float2>(double2 x) {
    return make_float2(float(x.x), float(x.y));
}
__device__ __forceinline__ double2 to_f64(double2 x) { return x; }
__device__ __forceinline__ double2 to_f64(float2 x) { return make_double2(x.x, x.y); }

}  // namespace wqc
