// simt_gemm.cuh -- the register-tiled FP32 SIMT GEMM of the plain FP32 path (inference and
// training kernels).
//
// A CTA holds the activations of 64 samples in one shared-memory tile, K-major: value (k, m) of
// feature k and sample m sits at k * 64 + (m ^ (k & 28)). The swizzle moves a row's 16-byte groups
// by its row number / 4, so that the epilogue's stores (rows 4 apart) and the per-sample column
// accesses (consecutive m) are both free of bank conflicts, without padding. A layer
// out[n][m] = epi(sum_k B[k][n] in[k][m]) is computed in place on that tile: each thread owns an
// 8 x C block of outputs (8 samples x C neurons) and, per k, reads 8 activations and C values of B
// as 16-byte words and issues 4 C paired FMAs (fma.rn.f32x2: two samples each, IEEE FMAs at half
// the issue slots; plain FMAs reached 59 of 74 TFLOP/s with distinct register operands, paired
// ones 68).
// B ([k_rows][ldb] in global memory: a layer's transposed weights for a forward step, its
// row-major weights for a backward step) comes from L2 in chunks of 16 rows, double-buffered with
// cp.async.
// Every output is accumulated as fmaf(B[k][n], in[k][m], acc) over k ascending, so the results do
// not depend on the launch shape.
//
// Threads: 64 for the 64- and 32-wide networks (8 x 8 and 8 x 4 outputs per thread, one thread
// per sample in the per-sample phases, 8 small CTAs per SM whose phases interleave), 128 for the
// 128-wide one.
#pragma once
#include "kernels.hpp"

namespace nrrs {
namespace simt {

constexpr int kTM = 64;        // samples (vertices) per tile
constexpr int kKC = 16;        // B rows per chunk

constexpr int imax(int a, int b) { return a > b ? a : b; }
// threads per CTA of a W-wide network's kernels
constexpr int threads_of(int w) { return w == 128 ? 128 : 64; }

// offset of value (k, m) in the tile
__device__ __forceinline__ int at(int k, int m) { return k * kTM + (m ^ (k & 28)); }

__device__ __forceinline__ void cp_async16(float* smem_dst, const float* gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
// the first src_bytes (0, 4, 8, 12 or 16) of 16; the rest is zero-filled
__device__ __forceinline__ void cp_async16_n(float* smem_dst, const float* gmem_src,
                                             unsigned src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem_src),
                 "r"(src_bytes)
                 : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// two FP32 FMAs: the low and the high halves of the 64-bit registers
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long dup2(float x) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ void unpack2f(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// rows x W floats of B (row stride ldb) into a shared-memory chunk
template <int W, int NT>
__device__ __forceinline__ void load_chunk(float* dst, const float* __restrict__ src, int ldb,
                                           int rows, int tid) {
    const int n4 = rows * (W / 4);
    for (int q = tid; q < n4; q += NT)
        cp_async16(dst + 4 * q, src + (size_t)(q / (W / 4)) * ldb + 4 * (q % (W / 4)));
}

// out[n][m] = epi(j, n, m0, v[8]) with v[i] = sum_{k < k_eff} B[k][n] act[k][m] for the 8 samples
// m = m0 .. m0+3 and m0+32 .. m0+35 and the C neurons n each thread owns (j = 0 .. C-1 counts
// them). Four samples each from both halves: the threads of a warp that share a neuron then hold
// 64 consecutive bytes, whole sectors when they store to global memory. Every read
// of the tile ends at the chunk loop's last barrier, so epi may overwrite it in place; a barrier
// follows epi. wch holds two chunks of kKC x W floats.
template <int W, int NT, class Epi>
__device__ __forceinline__ void tile_gemm(const float* __restrict__ B, int ldb, int k_eff,
                                          const float* act, float* wch, int tid, Epi&& epi) {
    constexpr int C = kTM * W / (8 * NT);     // neurons per thread
    constexpr int TX = W / C;
    constexpr int CW = C < 4 ? C : 4;         // consecutive neurons of a thread's group
    static_assert(C == 2 || C == 4 || C == 8, "tile widths");
    const int tx = tid % TX, ty = tid / TX;   // ty 0..7: samples 4 ty .. +3 and 32 + 4 ty .. +3
    unsigned long long acc[4][C];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) acc[i][j] = 0ull;
    const int nch = (k_eff + kKC - 1) / kKC;
    load_chunk<W, NT>(wch, B, ldb, k_eff < kKC ? k_eff : kKC, tid);
    cp_async_commit();
#pragma unroll 1
    for (int c = 0; c < nch; ++c) {
        if (c + 1 < nch) {
            const int r = k_eff - (c + 1) * kKC;
            load_chunk<W, NT>(wch + ((c + 1) & 1) * kKC * W, B + (size_t)(c + 1) * kKC * ldb, ldb,
                              r < kKC ? r : kKC, tid);
        }
        cp_async_commit();
        cp_async_wait<1>();   // every group but the newest: chunk c has landed
        __syncthreads();
        const float* Bc = wch + (c & 1) * kKC * W + tx * CW;
        const float* A = act + (size_t)(c * kKC) * kTM;
        auto step = [&](int kk) {
            const int sw = (c * kKC + kk) & 28;
            const ulonglong2 a0 =
                *reinterpret_cast<const ulonglong2*>(A + kk * kTM + ((ty * 4) ^ sw));
            const ulonglong2 a1 =
                *reinterpret_cast<const ulonglong2*>(A + kk * kTM + 32 + ((ty * 4) ^ sw));
            const unsigned long long av[4] = {a0.x, a0.y, a1.x, a1.y};
            float bv[C];
            if constexpr (C == 2) {
                const float2 b0 = *reinterpret_cast<const float2*>(Bc + kk * W);
                bv[0] = b0.x; bv[1] = b0.y;
            } else {
                const float4 b0 = *reinterpret_cast<const float4*>(Bc + kk * W);
                bv[0] = b0.x; bv[1] = b0.y; bv[2] = b0.z; bv[3] = b0.w;
            }
            if constexpr (C == 8) {
                const float4 b1 = *reinterpret_cast<const float4*>(Bc + kk * W + W / 2);
                bv[4] = b1.x; bv[5] = b1.y; bv[6] = b1.z; bv[7] = b1.w;
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const unsigned long long b2 = dup2(bv[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[i][j] = fma2(b2, av[i], acc[i][j]);
            }
        };
        if (k_eff - c * kKC >= kKC) {
#pragma unroll
            for (int kk = 0; kk < kKC; ++kk) step(kk);
        } else {
#pragma unroll 1
            for (int kk = 0; kk < k_eff - c * kKC; ++kk) step(kk);
        }
        __syncthreads();    // the buffer read here is refilled by the next iteration's prefetch
    }
#pragma unroll
    for (int j = 0; j < C; ++j) {
        const int n = (j < 4 ? 0 : W / 2) + tx * CW + (j & 3);
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) unpack2f(acc[i][j], v[2 * i], v[2 * i + 1]);
        epi(j, n, ty * 4, v);
    }
    __syncthreads();
}

// 8 values of tile row n: samples m0 .. m0+3 and m0+32 .. m0+35
__device__ __forceinline__ void tile_store8(float* act, int n, int m0, const float* v) {
    *reinterpret_cast<float4*>(act + at(n, m0)) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(act + at(n, m0 + 32)) = make_float4(v[4], v[5], v[6], v[7]);
}

// y[o] = sum_k wt[k][o] tile[k][m] for a narrow output layer (wt is [W][OUT rounded up to 4]), k
// ascending
template <int W, int OUT>
__device__ __forceinline__ void narrow_out(const float* __restrict__ wt, const float* tile, int m,
                                           float* y) {
    constexpr int OP = (OUT + 3) / 4 * 4;
    float acc[OUT];
#pragma unroll
    for (int o = 0; o < OUT; ++o) acc[o] = 0.f;
#pragma unroll 8
    for (int k = 0; k < W; ++k) {
        const float x = tile[at(k, m)];
#pragma unroll
        for (int q = 0; q < OP / 4; ++q) {
            const float4 w = __ldg(reinterpret_cast<const float4*>(wt + OP * k + 4 * q));
            const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (4 * q + e < OUT) acc[4 * q + e] = fmaf(wv[e], x, acc[4 * q + e]);
        }
    }
#pragma unroll
    for (int o = 0; o < OUT; ++o) y[o] = acc[o];
}

// Hash-grid features of one level from the FP32 table: trilinear over the 8 corners in corner
// order. For each (y, z) the aligned 32-byte sector holding corner x is loaded whole; corner x+1
// comes from it when it lies there (the hash multiplies x by 1, so x and x+1 differ in the low
// bits) and from a predicated 8-byte load otherwise. Each request from L1 to L2 carries one
// sector, so this makes about 5 of the 8 that one load per corner makes. The parameters follow
// the table, so the last sector is whole.
__device__ __forceinline__ float2 level_features_f(const float2* table, const LevelDev& L,
                                                   uint32_t mask, const CellCoord& c) {
    float2 t[8];
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
        const uint32_t y = c.iy + (k2 & 1), z = c.iz + ((k2 >> 1) & 1);
        const float2* p0 = table + grid_row(L, mask, c.ix, y, z);
        const float2* p1 = table + grid_row(L, mask, c.ix + 1, y, z);
        const uint32_t lo0 = (uint32_t)reinterpret_cast<uintptr_t>(p0);
        const uint32_t lo1 = (uint32_t)reinterpret_cast<uintptr_t>(p1);
        const float* q = reinterpret_cast<const float*>(reinterpret_cast<uintptr_t>(p0) &
                                                        ~uintptr_t(31));
        float s[8];
        asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(s[0]), "=f"(s[1]), "=f"(s[2]), "=f"(s[3]), "=f"(s[4]), "=f"(s[5]), "=f"(s[6]),
              "=f"(s[7])
            : "l"(q));
        const bool same = ((lo0 ^ lo1) & ~31u) == 0;
        float2 v1 = make_float2(0.f, 0.f);
        if (!same) v1 = __ldg(p1);
        auto pick = [&](uint32_t lo) {
            const bool e1 = lo & 8u, e2 = lo & 16u;
            const float ax = e1 ? s[2] : s[0], ay = e1 ? s[3] : s[1];
            const float bx = e1 ? s[6] : s[4], by = e1 ? s[7] : s[5];
            return make_float2(e2 ? bx : ax, e2 ? by : ay);
        };
        t[2 * k2] = pick(lo0);
        t[2 * k2 + 1] = same ? pick(lo1) : v1;
    }
    float f0 = 0.f, f1 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float w = corner_weight(c, k);
        f0 += w * t[k].x;
        f1 += w * t[k].y;
    }
    return make_float2(f0, f1);
}

// rows 0 .. ROWS-1 of 64 samples (row stride ld) into the tile, as 16-byte copies; the caller waits
// for the copies and synchronises
template <int ROWS, int NT>
__device__ __forceinline__ void load_rows(const float* src, size_t ld, float* tile, int tid) {
    for (int q = tid; q < ROWS * (kTM / 4); q += NT) {
        const int k = q / (kTM / 4), m = 4 * (q % (kTM / 4));
        cp_async16(tile + at(k, m), src + k * ld + m);
    }
}

}  // namespace simt
}  // namespace nrrs
