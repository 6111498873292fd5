// Transfer environments of <psi|psi> and of Pauli strings as batched tiled
// GEMMs: Pauli expectations (src/expectation.rs:98-200) and the right
// environments of shot sampling.
#include "common.cuh"
#include "split_kernels.cuh"
#include "tile_gemm.cuh"

namespace wqc {

namespace {

// (P t)[so] for the row t = (t0, t1) over the physical index.
__device__ __forceinline__ double2 pauli_row(char ch, int so, double2 t0, double2 t1) {
    switch (ch) {
        case 'X': return so ? t0 : t1;
        case 'Y': return so ? cmake(-t0.y, t0.x) : cmake(t1.y, -t1.x);
        case 'Z': return so ? cmake(-t1.x, -t1.y) : t0;
        default: return so ? t1 : t0;
    }
}

// T[a'][s][b] = sum_a E[a][a'] A[a][s][b]; E is [1] at the left end.
__device__ __forceinline__ void left_half(TileSmem& sm, const DeviceMps& mps, int q, const double2* env, bool first,
                                          double2* T, int m0, int n0) {
    const int l = mps.dl[q], r = mps.dr[q];
    if (m0 >= l || n0 >= 2 * r) return;
    const double2* s = mps.site[q];
    tile_gemm(
        sm, m0, n0, l, 2 * r, l, false, false,
        [&](int ap, int a) { return first ? cmake(1.0, 0.0) : env[size_t(a) * l + ap]; },
        [&](int a, int x) { return s[size_t(a) * 2 * r + x]; },
        [&](int ap, int x, double2 v) { T[size_t(ap) * 2 * r + x] = v; });
}

// E'[b][b'] = sum_{a', s} (P T)[a'][s][b] conj(A[a'][s][b']).
__device__ __forceinline__ void left_next(TileSmem& sm, const DeviceMps& mps, int q, const double2* T, char ch,
                                          double2* out, int m0, int n0) {
    const int l = mps.dl[q], r = mps.dr[q];
    if (m0 >= r || n0 >= r) return;
    const double2* s = mps.site[q];
    tile_gemm(
        sm, m0, n0, r, r, 2 * l, false, false,
        [&](int b, int x) {
            const double2* t = T + size_t(x >> 1) * 2 * r + b;
            return pauli_row(ch, x & 1, t[0], t[r]);
        },
        [&](int x, int bp) { return cconj(s[size_t(x) * r + bp]); },
        [&](int b, int bp, double2 v) { out[size_t(b) * r + bp] = v; });
}

}  // namespace

// One half of a step of the identity chains of every segment: blockIdx.z
// below nseg takes the left chain at site `step` from the left, the rest the
// right chain at the mirrored site.  phase 0 multiplies the environment into
// the site, phase 1 closes it with the conjugate site.
__global__ void __launch_bounds__(kTileThreads) env_chain_kernel(DeviceMps mps, EnvChains ch, int step, int phase) {
    __shared__ TileSmem sm;
    const int seg = blockIdx.z % ch.nseg;
    const bool right = int(blockIdx.z) / ch.nseg + (ch.left ? 0 : 1) == 1;
    const int first = ch.firsts[seg];
    const size_t E = size_t(ch.cap) * ch.cap;
    double2* base = ch.base + size_t(seg) * ch.seg_stride;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    if (!right) {
        const int q = first + step;
        double2* T = base + ch.t_off + size_t(step) * 2 * E;
        double2* L = base + ch.l_off;
        if (phase == 0)
            left_half(sm, mps, q, L + (step & 1) * E, step == 0, T, m0, n0);
        else if (step + 1 < ch.width)
            left_next(sm, mps, q, T, 'I', L + ((step + 1) & 1) * E, m0, n0);
        return;
    }
    // R_q[b][b'] contracts the sites right of q; R of the last site is [1].
    const int at = ch.width - 1 - step, q = first + at;
    auto right_of = [&](int x) { return base + (ch.r_at ? size_t(ch.r_at[x]) : ch.r_off + size_t(x) * E); };
    double2* R = right_of(at);
    double2* H = base + ch.h_off;
    const int l = mps.dl[q], r = mps.dr[q];
    const double2* s = mps.site[q];
    if (phase == 0) {
        if (step == 0 && m0 == 0 && n0 == 0 && threadIdx.x == 0) R[0] = cmake(1.0, 0.0);
        if (at == 0 || m0 >= 2 * l || n0 >= r) return;
        tile_gemm(  // H[a, s][b'] = sum_b A[a, s][b] R[b][b']
            sm, m0, n0, 2 * l, r, r, true, false, [&](int x, int b) { return s[size_t(x) * r + b]; },
            [&](int b, int bp) { return step == 0 ? cmake(1.0, 0.0) : R[size_t(b) * r + bp]; },
            [&](int x, int bp, double2 v) { H[size_t(x) * r + bp] = v; });
    } else {
        if (at == 0 || m0 >= l || n0 >= l) return;
        double2* out = right_of(at - 1);
        tile_gemm(  // R[a][a'] = sum_{s, b'} H[a][s, b'] conj(A[a'][s, b'])
            sm, m0, n0, l, l, 2 * r, true, true, [&](int a, int x) { return H[size_t(a) * 2 * r + x]; },
            [&](int x, int ap) { return cconj(s[size_t(ap) * 2 * r + x]); },
            [&](int a, int ap, double2 v) { out[size_t(a) * l + ap] = v; });
    }
}

// One half of step `step` of the terms t0 .. t0 + count - 1 of every segment:
// a term starts from the left chain's T at its first non-identity site, so
// its first step has no half of phase 0.
__global__ void __launch_bounds__(kTileThreads) env_term_kernel(DeviceMps mps, EnvChains ch, EnvTerms tm, int t0,
                                                               int count, int step, int phase) {
    __shared__ TileSmem sm;
    const int local = blockIdx.z % count, seg = blockIdx.z / count, t = t0 + local;
    if (step >= tm.span[t]) return;
    const size_t E = size_t(ch.cap) * ch.cap;
    const double2* base = ch.base + size_t(seg) * ch.seg_stride;
    double2* mine = tm.work + (size_t(seg) * count + local) * 4 * E;  // two environments, then T
    const int at = tm.start[t] + step, q = ch.firsts[seg] + at;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    if (phase == 0) {
        left_half(sm, mps, q, mine + (step & 1) * E, false, mine + 2 * E, m0, n0);
    } else {
        const double2* T = step == 0 ? base + ch.t_off + size_t(at) * 2 * E : mine + 2 * E;
        left_next(sm, mps, q, T, tm.labels[size_t(t) * ch.width + (ch.width - 1 - at)], mine + ((step + 1) & 1) * E, m0, n0);
    }
}

// <psi|P_t|psi> = sum_{b, b'} E[b][b'] R_q[b][b'] at the term's last site q.
__global__ void __launch_bounds__(256) env_dot_kernel(DeviceMps mps, EnvChains ch, EnvTerms tm, int t0, int count,
                                                      int nterms, double2* out) {
    const int local = blockIdx.x, seg = blockIdx.y, t = t0 + local;
    const size_t E = size_t(ch.cap) * ch.cap;
    const int at = tm.start[t] + tm.span[t] - 1, r = mps.dr[ch.firsts[seg] + at];
    const double2* env = tm.work + (size_t(seg) * count + local) * 4 * E + (tm.span[t] & 1) * E;
    const double2* R = ch.base + size_t(seg) * ch.seg_stride + ch.r_off + size_t(at) * E;
    __shared__ double2 red[8];
    double2 acc = cmake(0, 0);
    for (int e = threadIdx.x; e < r * r; e += 256) cfma(acc, env[e], R[e]);
    for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 v = red[0];
        for (int w = 1; w < 8; ++w) v = cadd(v, red[w]);
        out[size_t(seg) * nterms + t] = v;
    }
}

// Every step of the identity chains; `bond` bounds the bonds.  Two launches a
// site for both chains of every segment, instead of a walk over all sites on
// one CTA per Pauli term (50 sites, chi 128, 99 terms: 141 ms).
int launch_env_chains(const DeviceMps& mps, const EnvChains& ch, bool right, int bond, cudaStream_t stream) {
    const unsigned z = unsigned(ch.nseg) * ((ch.left ? 1 : 0) + (right ? 1 : 0));
    const unsigned b1 = unsigned(bond + kTile - 1) / kTile, b2 = unsigned(2 * bond + kTile - 1) / kTile;
    const unsigned both = ch.left && right ? b2 : 0;  // the chains' halves are b1 x b2 and b2 x b1 tiles
    for (int step = 0; step < ch.width; ++step) {
        env_chain_kernel<<<dim3(std::max(ch.left ? b2 : b1, both), std::max(right ? b2 : b1, both), z), kTileThreads, 0,
                           stream>>>(mps, ch, step, 0);
        env_chain_kernel<<<dim3(b1, b1, z), kTileThreads, 0, stream>>>(mps, ch, step, 1);
    }
    return 2 * ch.width;
}

int launch_env_terms(const DeviceMps& mps, const EnvChains& ch, const EnvTerms& tm, int t0, int count, int nterms,
                     int longest, int bond, double2* out, cudaStream_t stream) {
    const unsigned z = unsigned(ch.nseg) * unsigned(count);
    const unsigned b1 = unsigned(bond + kTile - 1) / kTile, b2 = unsigned(2 * bond + kTile - 1) / kTile;
    int launches = 1;
    for (int step = 0; step < longest; ++step) {
        if (step > 0) {
            env_term_kernel<<<dim3(b2, b1, z), kTileThreads, 0, stream>>>(mps, ch, tm, t0, count, step, 0);
            ++launches;
        }
        env_term_kernel<<<dim3(b1, b1, z), kTileThreads, 0, stream>>>(mps, ch, tm, t0, count, step, 1);
        ++launches;
    }
    env_dot_kernel<<<dim3(count, ch.nseg), 256, 0, stream>>>(mps, ch, tm, t0, count, nterms, out);
    return launches;
}

}  // namespace wqc
