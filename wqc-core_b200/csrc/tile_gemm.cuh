// A small tile of a complex FP64 product, for the batched GEMMs of a few
// hundred rows that a split, its adjoint and the environments are made of.
#pragma once

#include "common.cuh"

namespace wqc {

constexpr int kTile = 16, kTileK = 32, kTileThreads = kTile * kTile;

struct TileSmem {
    double2 a[kTileK][kTile + 1], b[kTileK][kTile + 1];
};

// One 16 x 16 tile of C = A B, one output per thread, summed over k in order.
// at_a(m, k) and at_b(k, n) are called inside the operands only; `a_along_k`
// (`b_along_k`) says that k runs fastest in A's (B's) memory, and the threads
// of a load follow it.  The next K block is fetched while this one is
// multiplied.  These products have up to 512 x 512 outputs and there are few of
// them at a time, so they are bound by how many SMs they reach: 32 x 32 tiles
// put a 256 x 128 product with k = 256 on 32 CTAs and took 66 us.
template <class FA, class FB, class FS>
__device__ __forceinline__ void tile_gemm(TileSmem& sm, int m0, int n0, int m, int n, int k, bool a_along_k,
                                          bool b_along_k, FA at_a, FB at_b, FS store) {
    constexpr int kLoads = kTileK * kTile / kTileThreads;
    const int tid = threadIdx.x, tm = tid / kTile, tn = tid % kTile;
    double2 fa[kLoads], fb[kLoads];
    auto place = [&](int e, bool along_k, int& i, int& kk) {
        if (along_k) {
            i = e / kTileK;
            kk = e % kTileK;
        } else {
            i = e % kTile;
            kk = e / kTile;
        }
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            int i, kk;
            place(tid + u * kTileThreads, a_along_k, i, kk);
            fa[u] = m0 + i < m && k0 + kk < k ? at_a(m0 + i, k0 + kk) : cmake(0, 0);
            place(tid + u * kTileThreads, b_along_k, i, kk);
            fb[u] = n0 + i < n && k0 + kk < k ? at_b(k0 + kk, n0 + i) : cmake(0, 0);
        }
    };
    double2 acc = cmake(0, 0);
    fetch(0);
    for (int k0 = 0; k0 < k; k0 += kTileK) {
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            int i, kk;
            place(tid + u * kTileThreads, a_along_k, i, kk);
            sm.a[kk][i] = fa[u];
            place(tid + u * kTileThreads, b_along_k, i, kk);
            sm.b[kk][i] = fb[u];
        }
        __syncthreads();
        if (k0 + kTileK < k) fetch(k0 + kTileK);
#pragma unroll 8
        for (int kk = 0; kk < kTileK; ++kk) cfma(acc, sm.a[kk][tm], sm.b[kk][tn]);
        __syncthreads();
    }
    if (m0 + tm < m && n0 + tn < n) store(m0 + tm, n0 + tn, acc);
}

}  // namespace wqc
