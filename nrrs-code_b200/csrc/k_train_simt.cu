// k_train_simt.cu -- one training step of StatNet and RRSNet (replaces NRRSNetwork::train,
// src/render/nrrs/net/network.cpp:196-295, and the two tcnn Trainer::training_step calls it makes:
// myNetworkLL2.cpp:51 for StatNet, network.cpp:274 for RRSNet).
//
// Losses (the reference's NRRS_LL2 / NRRS_RRS live in the absent tiny-cuda-nn fork; these are
// the workload's written definitions):
//   StatNet: loss_S = mean over samples and RGB of (y_c - log(L_c + stat_eps))^2
//   RRSNet:  q = activationSigma(raw), r = min(mean_c(thp_c L_c)/(ref + ref_eps), clamp),
//            V = mean(r^2 / q), C = mean(cost_offset + q), loss_R = V * C
//   RRSNet inputs come from the detached StatNet forward of the same step (the reference trains
//   the networks separately and builds RRSNet's input after StatNet's step, train.cu:155-240).
//
// Pipeline (forked from and joined into the caller's stream, no host synchronisation):
//   k_encode_f32  hash features of the batch, level-major (k_encode.cu).
//   k_train_stat  per sample: StatNet forward, loss gradient, backward to the hash lanes, glue;
//                 RRSNet forward for the batch sums V and C (FP64 per-CTA partials). Activations
//                 and deltas go to feature-major scratch for the weight gradients.
//   k_scatter_levels  the lane gradients into the table (FP32 reductions, k_train_tc.cu), beside
//   k_train_rrs   per sample: RRSNet forward and backward with the final V and C.
//   k_wgrad       dW = sum_i delta_i (x) a_i for every layer, split over sample chunks.
//   k_wreduce     chunk partials -> gradients, in fixed order (deterministic).
//   k_adam        Adam on FP32 master weights/moments; writes the FP16 table copy in the same pass.
#include "context.hpp"
#include "simt_gemm.cuh"

namespace nrrs {

namespace {


struct TrainArgs {
    VertexPtrs v;
    const float* target;
    uint32_t n;
    uint32_t ld;                   // row stride of the feature-major scratch
    FactorParams fp;
    float loss_clamp, cost_offset;
    int32_t train_rrs;
    const float* wt_stat;          // transposed [in][out4] (forward)
    const float* wt_rrs;
    const float* w_stat;           // row-major master [out][in] (backward)
    const float* w_rrs;
    float* act;                    // feature-major scratch
    uint32_t r_x0, r_hs, r_dhs, r_dx, r_dy, r_x1, r_hr, r_dhr, r_draw;
    double* part;                  // [grid][4]: loss_S sum, V sum, C sum, R sum
    uint32_t part_n;               // CTAs of k_train_stat
    double* loss_out;              // [2]
    LossWeights lw;                // per-sample loss weights (inactive: plain means)
};

__device__ __forceinline__ double block_sum_d(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    return t;  // valid on thread 0
}

// relative contribution used by the RRS loss
__device__ __forceinline__ float rel_contrib(const TrainArgs& a, uint32_t i) {
    const size_t i3 = 3 * (size_t)i;
    float acc = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) acc += a.v.thp[i3 + c] * a.target[i3 + c];
    const float ref = (a.v.ref ? a.v.ref[i] : 0.5f) + a.fp.ref_eps;
    const float r = acc / 3.0f / ref;
    return r < a.loss_clamp ? r : a.loss_clamp;
}

using simt::at;
using simt::kTM;

// activation tile rows and weight-chunk floats of the training kernels
template <int W>
struct TrShape {
    static constexpr int kThr = simt::threads_of(W);
    static constexpr int kRows = simt::imax(stat_in_of(W), W);
    static constexpr int kChunk = simt::kKC * W;
    static constexpr size_t kSmem = sizeof(float) * ((size_t)kRows * kTM + 2 * kChunk);
};

// forward layer: ReLU (LeakyReLU for the reference network, W = 32) in place, and the activations
// to scratch rows row0 + n (samples i0 ..). Bit 8 j + i of `pos` tells whether the thread's j-th
// neuron is positive for its i-th sample: the backward layers give a thread the same neurons and
// samples, so their masks come from these registers.
template <int W>
__device__ __forceinline__ void fwd_layer(const float* __restrict__ wt, int k_eff, float* tile,
                                          float* wch, int tid, float* scr, uint32_t ld, uint32_t i0,
                                          uint32_t row0, bool store, unsigned long long& pos) {
    unsigned long long bits = 0;
    simt::tile_gemm<W, TrShape<W>::kThr>(
        wt, W, k_eff, tile, wch, tid, [&](int j, int n, int m0, const float* v) {
            float r[8];
            uint32_t b = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                r[i] = W == 32 ? leaky(v[i]) : fmaxf(v[i], 0.f);
                b |= (v[i] > 0.f ? 1u : 0u) << i;
            }
            bits |= (unsigned long long)b << (8 * j);
            simt::tile_store8(tile, n, m0, r);
            if (store) {
                float* g = scr + (size_t)(row0 + n) * ld + i0 + m0;
                *reinterpret_cast<float4*>(g) = make_float4(r[0], r[1], r[2], r[3]);
                *reinterpret_cast<float4*>(g + 32) = make_float4(r[4], r[5], r[6], r[7]);
            }
        });
    pos = bits;
}

// backward layer through row-major W [outputs of the forward layer][W = its inputs]:
// delta_in[n][m] = (sum_k W[k][n] delta_out[k][m]) times the activation's slope (ReLU: 1 or 0;
// LeakyReLU: 1 or 0.01) by the forward layer's `pos` bits; in place, and to scratch rows out0 + n
template <int W>
__device__ __forceinline__ void bwd_layer(const float* __restrict__ w, float* tile, float* wch,
                                          int tid, float* scr, uint32_t ld, uint32_t i0,
                                          uint32_t out0, unsigned long long pos) {
    simt::tile_gemm<W, TrShape<W>::kThr>(
        w, W, W, tile, wch, tid, [&](int j, int n, int m0, const float* v) {
            float r[8];
            const uint32_t b = (uint32_t)(pos >> (8 * j));
#pragma unroll
            for (int i = 0; i < 8; ++i)
                r[i] = (b >> i) & 1u ? v[i] : (W == 32 ? 0.01f * v[i] : 0.f);
            simt::tile_store8(tile, n, m0, r);
            float* g = scr + (size_t)(out0 + n) * ld + i0 + m0;
            *reinterpret_cast<float4*>(g) = make_float4(r[0], r[1], r[2], r[3]);
            *reinterpret_cast<float4*>(g + 32) = make_float4(r[4], r[5], r[6], r[7]);
        });
}

// The delta of the last hidden layer in column m of the tile (which holds that layer's
// activations): d[k] = sum_o w[o][k] g[o] times the activation's slope; w is the row-major output
// layer [OUT][W]. Also to scratch rows at dl (stride ld) when store is set.
template <int W, int OUT>
__device__ __forceinline__ void last_delta(const float* __restrict__ w, const float* g, float* tile,
                                           int m, float* dl, uint32_t ld, bool store) {
    constexpr bool REF = W == 32;
#pragma unroll 2
    for (int k = 0; k < W; k += 4) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int o = 0; o < OUT; ++o) {
            const float4 wv = __ldg(reinterpret_cast<const float4*>(w + o * W + k));
            acc[0] = fmaf(wv.x, g[o], acc[0]);
            acc[1] = fmaf(wv.y, g[o], acc[1]);
            acc[2] = fmaf(wv.z, g[o], acc[2]);
            acc[3] = fmaf(wv.w, g[o], acc[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float& x = tile[at(k + e, m)];
            const float d = x > 0.f ? acc[e] : (REF ? 0.01f * acc[e] : 0.f);
            x = d;
            if (store) dl[(size_t)(k + e) * ld] = d;
        }
    }
}

// The StatNet step and the RRSNet forward sums on 64-sample tiles: the hash lanes copied from the
// encoding kernel's rows and the other input lanes made here, the forward layers as tile GEMMs
// storing every activation, the loss gradient, the backward layers as tile GEMMs through the
// row-major weights, the gradient of the hash lanes to scratch rows (the scatter kernel adds them
// into the table), then the glue and the RRSNet forward for the sums. Per-sample phases run one
// thread per sample (64 threads per CTA); the 128-wide networks' CTAs have 128 threads and split the
// other input lanes over two per sample.
// 64 x 2, 262,144 samples: 315 us beside 89 us of encoding and 185 us of scatter (kernels of their
// own, the scatter overlapped), against 735 us for one kernel that did all three with 24 warps per
// SM waiting for the gathers (330 us of it) and for the reductions (175 us).
template <int WS, int HS, int WR, int HR>
__global__ void __launch_bounds__(TrShape<WS>::kThr, WS == 128 ? 4 : 8)
    k_train_stat(const __grid_constant__ TrainArgs a) {
    static_assert(WS == WR, "one tile shape for both networks");
    constexpr bool REF = WS == 32;             // the reference's shipped network
    constexpr int SIN = stat_in_of(WS), SOUT = stat_out_of(WS);
    constexpr int X1 = REF ? kRefRrsLanes : 10;     // live RRSNet input lanes
    using S = TrShape<WS>;
    constexpr int TPS = S::kThr / kTM;              // threads per sample
    extern __shared__ float4 smem4[];
    float* tile = reinterpret_cast<float*>(smem4);
    float* wch = tile + S::kRows * kTM;
    __shared__ double red[S::kThr / 32];
    wait_for_stream();
    const int tid = threadIdx.x;
    const int m = tid & (kTM - 1);
    const bool lead = tid < kTM;
    const bool lo = TPS == 1 || lead, hi = TPS == 1 || !lead;   // this thread's share of the lanes
    const uint32_t ld = a.ld;
    float* scr = a.act;
    double lossS = 0.0, sumV = 0.0, sumC = 0.0, sumR = 0.0;
    // forward (transposed) and backward (row-major) layer images
    const float* ts = a.wt_stat;
    const float* ts_out = ts + (size_t)SIN * WS + (size_t)(HS - 1) * WS * WS;
    const float* rs = a.w_stat;
    const float* rs_out = rs + (size_t)SIN * WS + (size_t)(HS - 1) * WS * WS;   // [SOUT][WS]
    const float* tr = a.wt_rrs;
    const float* tr_out = tr + (size_t)kRrsIn * WR + (size_t)(HR - 1) * WR * WR;
    const uint32_t items = (a.n + kTM - 1) / kTM;
#pragma unroll 1
    for (uint32_t u = blockIdx.x; u < items; u += gridDim.x) {
        const uint32_t i0 = u * kTM, i = i0 + m;
        const bool valid = i < a.n;
        __syncthreads();   // the previous tile's column reads are over
        // ---- the input tile: hash lanes from the encoding kernel's x0 rows, the other lanes here
        //      (and to their x0 rows) ----
        constexpr int LANES = REF ? 32 : 56, HL = REF ? 16 : 32;
        simt::load_rows<HL, S::kThr>(scr + (size_t)a.r_x0 * ld + i0, ld, tile, tid);
        simt::cp_async_commit();
        if (valid) {
            float* x0 = scr + (size_t)(a.r_x0 + HL) * ld + i;
            auto put = [&](int k, float x) {
                tile[at(HL + k, m)] = x;
                x0[(size_t)k * ld] = x;
            };
            if (REF) {
                // the reference network: direction blobs (lo) and roughness blob (hi)
                float blob[16];
                ref_blob_lanes(a.v, i, blob);
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    if (k < 8 ? lo : hi) put(k, blob[k]);
            } else {
                if (lo) {
                    float sh[16];
                    const size_t i3 = 3 * (size_t)i;
                    sh16(a.v.wi[i3], a.v.wi[i3 + 1], a.v.wi[i3 + 2], sh);
#pragma unroll
                    for (int k = 0; k < 16; ++k) put(k, sh[k]);
                }
                if (hi) {
                    float mm[16];
                    misc_lanes(a.v, i, mm);
#pragma unroll
                    for (int k = 0; k < 8; ++k) put(16 + k, mm[k]);
                }
            }
        } else {
            constexpr int NO = LANES - HL;       // non-hash lanes; `hi` owns the last 8
            for (int k = lo ? 0 : NO - 8; k < (hi ? NO : NO - 8); ++k) tile[at(HL + k, m)] = 0.f;
        }

        // ---- StatNet forward, every hidden activation to scratch ----
        unsigned long long pos[HS];
        fwd_layer<WS>(ts, LANES, tile, wch, tid, scr, ld, i0, a.r_hs, true, pos[0]);
#pragma unroll
        for (int h = 1; h < HS; ++h)
            fwd_layer<WS>(ts + (size_t)SIN * WS + (size_t)(h - 1) * WS * WS, WS, tile, wch, tid,
                          scr, ld, i0, a.r_hs + h * WS, true, pos[h]);

        // ---- output, loss gradient, and the delta of the last hidden layer (own column) ----
        float y[SOUT];
#pragma unroll
        for (int k = 0; k < SOUT; ++k) y[k] = 0.f;
        SampleMul mu{1.f, 1.f, 1.f, 0.f};
        if (lead) {
            simt::narrow_out<WS, SOUT>(ts_out, tile, m, y);
            float g[SOUT];
#pragma unroll
            for (int k = 0; k < SOUT; ++k) g[k] = 0.f;
            if (valid) {
                const size_t i3 = 3 * (size_t)i;
                mu = sample_mul(a.lw, i, a.n);
                if (REF) {
                    // relative squared error of L and L^2 against the target L and its square
#pragma unroll
                    for (int c = 0; c < 6; ++c) {
                        const float L = a.target[i3 + (c % 3)];
                        const float T = c < 3 ? L : L * L;
                        const float den = T * T + 0.01f;
                        const float d = y[c] - T;
                        lossS += (double)mu.stat * (double)d * (double)d / (double)den;
                        g[c] = mu.stat * (2.0f * d) / (den * 6.0f * (float)a.n);
                        scr[(size_t)(a.r_dy + c) * ld + i] = g[c];
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float d = y[c] - logf(a.target[i3 + c] + a.fp.stat_eps);
                        if (a.lw.active) {
                            lossS += (double)mu.stat * (double)d * (double)d;
                            g[c] = mu.stat * (2.0f * d) / (3.0f * (float)a.n);
                        } else {
                            lossS += (double)d * (double)d;
                            g[c] = 2.0f * d / (3.0f * (float)a.n);
                        }
                        scr[(size_t)(a.r_dy + c) * ld + i] = g[c];
                    }
                }
            }
            last_delta<WS, SOUT>(rs_out, g, tile, m,
                                 scr + (size_t)(a.r_dhs + (HS - 1) * WS) * ld + i, ld, valid);
        }

        // ---- backward through the hidden layers, then the hash-lane gradients ----
#pragma unroll
        for (int h = HS - 1; h >= 1; --h)
            bwd_layer<WS>(rs + (size_t)SIN * WS + (size_t)(h - 1) * WS * WS, tile, wch, tid, scr,
                          ld, i0, a.r_dhs + (h - 1) * WS, pos[h - 1]);
        // straight to scratch: the level-major scatter applies them
        simt::tile_gemm<32, S::kThr>(rs, SIN, WS, tile, wch, tid,
                                     [&](int, int n, int m0, const float* v) {
            if (n >= HL) return;
            float* g = scr + (size_t)(a.r_dx + n) * ld + i0 + m0;
            *reinterpret_cast<float4*>(g) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(g + 32) = make_float4(v[4], v[5], v[6], v[7]);
        });

        // ---- glue and the RRSNet forward for the batch sums ----
        if (a.train_rrs) {
            if (lead) {
                float x1[16];
                if (REF) glue16_ref_aux(y, load_aux(a.v, valid ? i : 0u), x1);
                else glue16(a.fp, y, a.v, valid ? i : 0u, x1);
#pragma unroll
                for (int k = 0; k < X1; ++k) {
                    tile[at(k, m)] = valid ? x1[k] : 0.f;
                    if (valid) scr[(size_t)(a.r_x1 + k) * ld + i] = x1[k];
                }
            }
            unsigned long long unused;
            fwd_layer<WR>(tr, X1, tile, wch, tid, scr, ld, i0, 0, false, unused);
#pragma unroll 1
            for (int h = 1; h < HR; ++h)
                fwd_layer<WR>(tr + (size_t)kRrsIn * WR + (size_t)(h - 1) * WR * WR, WR, tile, wch,
                              tid, scr, ld, i0, 0, false, unused);
            if (lead && valid) {
                float raw;
                simt::narrow_out<WR, 1>(tr_out, tile, m, &raw);
                const float q = act_sigma(raw);
                const float r = rel_contrib(a, i);
                if (a.lw.active) {
                    const float lq = logf(q);
                    sumV += (double)(mu.var * (r * r / q));
                    sumC += (double)(mu.cost * (a.cost_offset + q));
                    sumR += (double)(mu.reg * (lq * lq));
                } else {
                    sumV += (double)(r * r / q);
                    sumC += (double)(a.cost_offset + q);
                }
            }
        }
    }
    const double s0 = block_sum_d(lossS, red);
    const double s1 = block_sum_d(sumV, red);
    const double s2 = block_sum_d(sumC, red);
    const double s3 = block_sum_d(sumR, red);
    if (threadIdx.x == 0) {
        a.part[4 * blockIdx.x + 0] = s0;
        a.part[4 * blockIdx.x + 1] = s1;
        a.part[4 * blockIdx.x + 2] = s2;
        a.part[4 * blockIdx.x + 3] = s3;
    }
}

// The RRSNet step on 64-sample tiles: the forward layers again (activations to scratch), the
// loss gradient with the batch's V and C, and the backward layers.
template <int WR, int HR>
__global__ void __launch_bounds__(TrShape<WR>::kThr, WR == 128 ? 4 : 8)
    k_train_rrs(const __grid_constant__ TrainArgs a) {
    constexpr bool REF = WR == 32;             // the reference's shipped network
    constexpr int X1 = REF ? kRefRrsLanes : 10;
    using S = TrShape<WR>;
    extern __shared__ float4 smem4[];
    float* tile = reinterpret_cast<float*>(smem4);
    float* wch = tile + S::kRows * kTM;
    __shared__ double s_tot[4], s_red[4][S::kThr / 4];
    wait_for_stream();
    const int tid = threadIdx.x;
    const int m = tid & (kTM - 1);
    const bool lead = tid < kTM;
    const uint32_t ld = a.ld;
    float* scr = a.act;
    // the batch sums of the StatNet kernel's CTA partials, in the same order in every CTA: slices of
    // rows b = tid / 4 (mod threads / 4), then the slices (one serial sum per column took 40 us)
    {
        double t = 0.0;
#pragma unroll 8
        for (uint32_t b = tid >> 2; b < a.part_n; b += S::kThr / 4) t += a.part[4 * b + (tid & 3)];
        s_red[tid & 3][tid >> 2] = t;
        __syncthreads();
        if (tid < 4) {
            t = 0.0;
            for (int k = 0; k < S::kThr / 4; ++k) t += s_red[tid][k];
            s_tot[tid] = t;
        }
    }
    __syncthreads();
    const double Vm = s_tot[1] / (double)a.n, Cm = s_tot[2] / (double)a.n;
    if (blockIdx.x == 0 && tid == 0) {
        a.loss_out[0] = s_tot[0] / ((REF ? 6.0 : 3.0) * (double)a.n);
        a.loss_out[1] = a.train_rrs ? (a.lw.active ? Vm * Cm + s_tot[3] / (double)a.n : Vm * Cm)
                                    : 0.0;
    }
    if (!a.train_rrs) return;
    const float Vf = (float)Vm, Cf = (float)Cm;
    const float* tr = a.wt_rrs;
    const float* tr_out = tr + (size_t)kRrsIn * WR + (size_t)(HR - 1) * WR * WR;
    const float* rr = a.w_rrs;
    const float* rr_out = rr + (size_t)kRrsIn * WR + (size_t)(HR - 1) * WR * WR;   // [1][WR]
    const uint32_t items = (a.n + kTM - 1) / kTM;
#pragma unroll 1
    for (uint32_t u = blockIdx.x; u < items; u += gridDim.x) {
        const uint32_t i0 = u * kTM, i = i0 + m;
        const bool valid = i < a.n;
        __syncthreads();
        if (lead) {
#pragma unroll
            for (int k = 0; k < X1; ++k)
                tile[at(k, m)] = valid ? scr[(size_t)(a.r_x1 + k) * ld + i] : 0.f;
        }
        unsigned long long pos[HR];
        fwd_layer<WR>(tr, X1, tile, wch, tid, scr, ld, i0, a.r_hr, true, pos[0]);
#pragma unroll
        for (int h = 1; h < HR; ++h)
            fwd_layer<WR>(tr + (size_t)kRrsIn * WR + (size_t)(h - 1) * WR * WR, WR, tile, wch, tid,
                          scr, ld, i0, a.r_hr + h * WR, true, pos[h]);
        if (lead) {
            float draw = 0.f;
            if (valid) {
                float raw;
                simt::narrow_out<WR, 1>(tr_out, tile, m, &raw);
                const float q = act_sigma(raw);
                const float r = rel_contrib(a, i);
                float dq;
                if (a.lw.active) {
                    const SampleMul mu = sample_mul(a.lw, i, a.n);
                    dq = (mu.var * (-(r * r) / (q * q)) * Cf + mu.cost * Vf +
                          mu.reg * (2.0f * logf(q) / q)) / (float)a.n;
                } else {
                    dq = (-(r * r) / (q * q) * Cf + Vf) / (float)a.n;
                }
                draw = dq * act_sigma_grad(raw);
                scr[(size_t)a.r_draw * ld + i] = draw;
            }
            last_delta<WR, 1>(rr_out, &draw, tile, m,
                              scr + (size_t)(a.r_dhr + (HR - 1) * WR) * ld + i, ld, valid);
        }
#pragma unroll
        for (int h = HR - 1; h >= 1; --h)
            bwd_layer<WR>(rr + (size_t)kRrsIn * WR + (size_t)(h - 1) * WR * WR, tile, wch, tid, scr,
                          ld, i0, a.r_dhr + (h - 1) * WR, pos[h - 1]);
    }
}

// ---- batch sums of the loss weights (fixed slices and order: deterministic) ----
// out[0] = sum s_i, out[1] = sum w_i, out[2] = the mean pixel error error_sum / n_pixels (1 when
// no error sum is given). kSumBlocks CTAs each sum a fixed slice into part[b]; the last one to
// finish (a counter, which it resets) adds the slices in order. One CTA for the whole batch took
// 28 us at 50,021 samples; this takes 4.9.
constexpr int kSumThr = 512;
__global__ void __launch_bounds__(kSumThr) k_loss_sums(const __grid_constant__ LossWeights w,
                                                       uint32_t n, const float* error_sum,
                                                       uint32_t n_pixels, double* out, double* part,
                                                       unsigned* done) {
    __shared__ double red[2][kSumThr / 32];
    __shared__ bool s_last;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    auto block_pair = [&](double& s, double& ww) {   // sums over the CTA, valid on thread 0
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            ww += __shfl_xor_sync(0xffffffffu, ww, o);
        }
        if (lane == 0) red[0][wid] = s, red[1][wid] = ww;
        __syncthreads();
        if (threadIdx.x == 0) {
            s = ww = 0.0;
            for (int k = 0; k < kSumThr / 32; ++k) s += red[0][k], ww += red[1][k];
        }
    };
    double s = 0.0, ww = 0.0;
    for (uint32_t i = blockIdx.x * kSumThr + threadIdx.x; i < n; i += gridDim.x * kSumThr) {
        s += (double)loss_w_stat(w, i);
        ww += (double)loss_w_rrs(w, i);
    }
    block_pair(s, ww);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = s;
        part[2 * blockIdx.x + 1] = ww;
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    s = ww = 0.0;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += kSumThr) {
        s += __ldcg(part + 2 * b);
        ww += __ldcg(part + 2 * b + 1);
    }
    __syncthreads();
    block_pair(s, ww);
    if (threadIdx.x == 0) {
        *done = 0;
        out[0] = s;
        out[1] = ww;
        double em = 1.0;
        if (error_sum && n_pixels) {
            em = (double)*error_sum / (double)n_pixels;
            if (!(em > 1e-30)) em = 1e-30;
        }
        out[2] = em;
    }
}

}  // namespace

cudaError_t launch_loss_sums(const LossWeights& w, uint32_t n, const float* error_sum,
                             uint32_t n_pixels, double* out, cudaStream_t s) {
    // out[4] on: a pair per CTA, then the counter
    const uint32_t need = (n + kSumThr - 1) / kSumThr;
    k_loss_sums<<<need < kLossSumBlocks ? need : kLossSumBlocks, kSumThr, 0, s>>>(
        w, n, error_sum, n_pixels, out, out + 4,
        reinterpret_cast<unsigned*>(out + 4 + 2 * kLossSumBlocks));
    return cudaGetLastError();
}

namespace {

// ---- weight gradients: dW[o][k] = sum_i D[o][i] * A[k][i] over the batch ----
// One job is one output tile (at most 64 x 64) of one layer; a CTA computes it over one sample
// chunk. Tile shapes are thread grids TY x TX of RU x 4 outputs each (kWShapes below); a thread
// grid smaller than the CTA is repeated as sample groups, whose sums are added at the end in
// group order.
struct WJob {
    uint32_t d_row, a_row;   // first scratch row of the tile's deltas / activations
    uint32_t M, N;           // rows that exist in the scratch (the rest of the tile is zero)
    uint32_t store_n;        // columns written: N and the layer's zero input lanes
    uint32_t ldw;            // input width of the layer (row stride of W)
    uint32_t out;            // offset of the tile in the MLP gradient vector
    uint32_t shape;          // index into kWShapes
};
constexpr int kMaxJobs = 32;

struct WGradArgs {
    const float* act;
    uint32_t ld, n;
    uint32_t chunk;          // samples per chunk, a multiple of kWS
    float* partial;          // [chunks][total]
    uint32_t total;          // MLP gradient length
    WJob job[kMaxJobs];
};

constexpr int kWThr = 256;
constexpr int kWS = 64;          // samples per stage
constexpr int kWStages = 3;
// row pitch of a stage: 64 samples and 4 floats, so that rows r, r+1, .. r+7 start 4 banks apart
// and eight 16-byte reads of consecutive rows take one pass
constexpr int kWPitch = kWS + 4;
constexpr int kWRows = 128;      // largest tile: 64 delta + 64 activation rows
constexpr size_t kWSmem = sizeof(float) * (size_t)kWStages * kWRows * kWPitch;

// The whole (job, chunk): rows arrive as 16-byte cp.async copies (samples past the chunk's end
// zero-filled), three stages deep; a thread reads 4 samples of its RU delta and 4 activation rows
// as 16-byte words and adds the products of the even and odd samples as FP32 pairs (two FMAs per
// issue slot).
template <int RU, int TY, int TX>
__device__ __forceinline__ void wgrad_tile(const WGradArgs& a, const WJob& j, float* sm,
                                           uint32_t i0, uint32_t i1, float* out) {
    constexpr int TM = RU * TY, TN = 4 * TX, ROWS = TM + TN;
    constexpr int G = TY * TX, GROUPS = kWThr / G;
    static_assert(ROWS <= kWRows && kWThr % G == 0 && GROUPS <= kWS / 4, "tile shape");
    static_assert(GROUPS * TM * TN <= kWStages * kWRows * kWPitch, "group sums fit the stages");
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = (tid / TX) % TY, grp = tid / G;
    constexpr int kStage = ROWS * kWPitch;
    // rows of the tile that no layer row backs stay zero in every stage
    for (int e = tid; e < kWStages * ROWS * (kWS / 4); e += kWThr) {
        const int st = e / (ROWS * (kWS / 4)), r = (e / (kWS / 4)) % ROWS, q = e % (kWS / 4);
        const bool live = r < TM ? (uint32_t)r < j.M : (uint32_t)(r - TM) < j.N;
        if (!live)
            *reinterpret_cast<float4*>(sm + st * kStage + r * kWPitch + 4 * q) =
                make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const uint32_t stages = (i1 - i0 + kWS - 1) / kWS;
    // a thread copies the same 16 bytes of rows r0, r0 + 16, .. in every stage
    const int r0 = tid / (kWS / 4), q0 = 4 * (tid % (kWS / 4));
    constexpr int kStep = kWThr / (kWS / 4);
    const float* gd = a.act + (size_t)(j.d_row + r0) * a.ld + i0 + q0;
    const float* ga = a.act + (size_t)(j.a_row + r0) * a.ld + i0 + q0;
    const size_t gstep = (size_t)kStep * a.ld;
    auto issue = [&](uint32_t s) {
        if (s < stages) {
            float* dst = sm + (s % kWStages) * kStage + r0 * kWPitch + q0;
            const uint32_t i = i0 + s * kWS + q0;
            const uint32_t left = i < i1 ? i1 - i : 0u;
            const uint32_t bytes = left >= 4u ? 16u : 4u * left;
            const size_t o = left ? s * kWS : 0;     // nothing left: any valid address
#pragma unroll
            for (int k = 0; k < (TM + kStep - 1) / kStep; ++k)
                if ((uint32_t)(r0 + k * kStep) < j.M)
                    simt::cp_async16_n(dst + k * kStep * kWPitch, gd + k * gstep + o, bytes);
#pragma unroll
            for (int k = 0; k < (TN + kStep - 1) / kStep; ++k)
                if ((uint32_t)(r0 + k * kStep) < j.N)
                    simt::cp_async16_n(dst + (TM + k * kStep) * kWPitch, ga + k * gstep + o, bytes);
        }
        simt::cp_async_commit();
    };
    unsigned long long acc[RU][4];
#pragma unroll
    for (int u = 0; u < RU; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) acc[u][w] = 0ull;
#pragma unroll
    for (int s = 0; s < kWStages - 1; ++s) issue(s);
    for (uint32_t s = 0; s < stages; ++s) {
        simt::cp_async_wait<kWStages - 2>();
        __syncthreads();   // stage s has landed for everyone, and stage s - 1 is free
        issue(s + kWStages - 1);
        const float* D = sm + (s % kWStages) * kStage + ty * kWPitch;
        const float* X = sm + (s % kWStages) * kStage + (TM + tx) * kWPitch;
#pragma unroll 2
        for (int q = grp; q < kWS / 4; q += GROUPS) {
            ulonglong2 x[4];
#pragma unroll
            for (int w = 0; w < 4; ++w)
                x[w] = *reinterpret_cast<const ulonglong2*>(X + w * TX * kWPitch + 4 * q);
#pragma unroll
            for (int u = 0; u < RU; ++u) {
                const ulonglong2 d =
                    *reinterpret_cast<const ulonglong2*>(D + u * TY * kWPitch + 4 * q);
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    acc[u][w] = simt::fma2(d.y, x[w].y, simt::fma2(d.x, x[w].x, acc[u][w]));
            }
        }
    }
    simt::cp_async_wait<0>();
    __syncthreads();
    // group sums, then the chunk's partial in group order
#pragma unroll
    for (int u = 0; u < RU; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            float e, o;
            simt::unpack2f(acc[u][w], e, o);
            sm[grp * TM * TN + (ty + u * TY) * TN + tx + w * TX] = e + o;
        }
    __syncthreads();
    for (int e = tid; e < TM * TN; e += kWThr) {
        const uint32_t m = e / TN, k = e % TN;
        if (m >= j.M || k >= j.store_n) continue;
        float t = 0.f;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) t += sm[g * TM * TN + e];
        out[(size_t)m * j.ldw + k] = t;
    }
}

// the tile shapes: rows (delta) x columns (activation) of an output tile
struct WShape {
    uint32_t tm, tn;
};
constexpr WShape kWShapes[] = {{64, 64}, {32, 32}, {64, 16}, {32, 16}, {8, 64}, {8, 32}};

// Bound by the FP32 FMA pipe for the square tiles and by HBM for the narrow output layers (both
// operands are read once per output tile). 64 x 64 tiles of 8 x 4 outputs per thread read 12
// 16-byte words per 128 FMAs; two CTAs per SM. The tile follows the layer (32 x 32 for the shipped
// network, 8 rows for the output layers), so little work is done for padding. Measured: 64 x 2,
// 262,144 samples 251 us (272 with a stage's copy addresses formed by divisions each time),
// where 16 outputs per thread fed by scalar shared-memory reads, one stage deep, took 937 us;
// shipped network, 50,021 samples 38 us against 419 us (25 chunks of 2,048 left the chip idle).
// The tile loop alone, on resident shared memory, reaches 46 TFLOP/s (43 to 49 for 4 x 4 to 8 x 8
// outputs per thread, paired or not); the work here is 7.5 GFLOP.
__global__ void __launch_bounds__(kWThr, 2) k_wgrad(const __grid_constant__ WGradArgs a) {
    extern __shared__ float4 smem4[];
    float* sm = reinterpret_cast<float*>(smem4);
    wait_for_stream();
    const WJob& j = a.job[blockIdx.y];
    const uint32_t i0 = blockIdx.x * a.chunk;
    const uint32_t i1 = min(a.n, i0 + a.chunk);
    float* out = a.partial + (size_t)blockIdx.x * a.total + j.out;
    switch (j.shape) {
        case 0: wgrad_tile<8, 8, 16>(a, j, sm, i0, i1, out); break;
        case 1: wgrad_tile<4, 8, 8>(a, j, sm, i0, i1, out); break;
        case 2: wgrad_tile<8, 8, 4>(a, j, sm, i0, i1, out); break;
        case 3: wgrad_tile<4, 8, 4>(a, j, sm, i0, i1, out); break;
        case 4: wgrad_tile<4, 2, 16>(a, j, sm, i0, i1, out); break;
        default: wgrad_tile<4, 2, 8>(a, j, sm, i0, i1, out); break;
    }
}

// samples per weight-gradient chunk of an n-sample step: 256 chunks (times the layers: several
// waves of the grid, so that the last one costs little), and at least 256 samples to each, four
// stages, so that a chunk's start-up and its partial stay small beside it (2,048 in the compact
// layout, for fewer partials)
uint32_t wgrad_chunk(uint64_t n, bool compact) {
    const uint64_t least = compact ? 2048 : 256;
    uint64_t c = (n + 255) / 256;
    c = (c + kWS - 1) / kWS * kWS;
    return (uint32_t)(c < least ? least : c);
}
// chunk partials that steps of up to n samples need
uint64_t wgrad_chunks_max(uint64_t n, bool compact) {
    const uint64_t least = compact ? 2048 : 256, c = (n + least - 1) / least;
    return c < 256 ? c : 256;
}

// the output tiles of one layer (M outputs x N stored inputs of width ldw) as jobs
int add_layer_jobs(WJob* job, uint32_t d_row, uint32_t a_row, uint32_t M, uint32_t N,
                   uint32_t ldw, uint32_t out) {
    uint32_t shape = 0;
    if (M <= 8) shape = ldw >= 64 ? 4 : 5;
    else if (ldw <= 16) shape = M >= 64 ? 2 : 3;
    else shape = M >= 64 ? 0 : 1;
    const WShape t = kWShapes[shape];
    int k = 0;
    for (uint32_t m = 0; m < M; m += t.tm)
        for (uint32_t n = 0; n < ldw; n += t.tn) {
            const uint32_t mv = M - m < t.tm ? M - m : t.tm, nv = N - n < t.tn ? N - n : t.tn;
            const uint32_t sv = ldw - n < t.tn ? ldw - n : t.tn;
            job[k++] = WJob{d_row + m, a_row + n, mv, nv, sv, ldw, out + m * ldw + n, shape};
        }
    return k;
}

// gradients = sum of the chunk partials of [chunks][stride] for the first `count` entries, in a
// fixed order: eight slices of consecutive chunks, each in chunk order, then the slices in order.
// Latency-bound (a few MB from L2): one serial sum per entry over 128 partials of the 64 x 2
// networks took 11.0 us; eight slices over 256 partials take 5.2 us. 128 x 3 networks (90,000
// entries, 55 partials): 18.3 -> 12.6 us.
constexpr int kRedSlices = 8;
__global__ void __launch_bounds__(32 * kRedSlices) k_wreduce(const float* partial, uint32_t chunks,
                                                             uint32_t stride, uint32_t count,
                                                             float* grad, float scale) {
    __shared__ float red[kRedSlices][32];
    wait_for_stream();
    const uint32_t lane = threadIdx.x & 31u, sl = threadIdx.x >> 5;
    const uint32_t e = blockIdx.x * 32u + lane;
    const uint32_t per = (chunks + kRedSlices - 1) / kRedSlices;
    const uint32_t c0 = sl * per, c1 = min(chunks, c0 + per);
    float s = 0.f;
    if (e < count)
        for (uint32_t c = c0; c < c1; c += 8) {   // eight loads in flight, whatever the remainder
            float v[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
                v[k] = c + k < c1 ? partial[(size_t)(c + k) * stride + e] : 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) s += v[k];
        }
    red[sl][lane] = s;
    __syncthreads();
    if (sl == 0 && e < count) {
#pragma unroll
        for (int k = 1; k < kRedSlices; ++k) s += red[k][lane];
        grad[e] = s * scale;
    }
}

struct AdamArgs {
    float* p;
    const float* g;
    float gscale;
    float* m;
    float* v;
    __half* table_h;       // FP16 copy of [0, n_table) refreshed in the same pass (may be null)
    uint64_t n_table;
    uint64_t count;
    uint64_t rrs_first;    // parameters from here on (the RRSNet) use lr_rrs
    float lr, lr_rrs, b1, b2, eps, l2, inv_c1, inv_c2;
    // the moving average of all n_params (e = null: none)
    float* e;
    float* pi;             // the debiased average
    __half* table_hi;      // FP16 copy of pi over [0, n_table) (may be null)
    uint64_t n_params;
    float d, omd, inv;     // decay, 1 - decay, 1 / (1 - decay^t)
};

// Adam on one parameter. The bias corrections are multiplications by 1/c1 and 1/c2 computed on
// the host, and the step is one fast division: IEEE divisions made this streaming kernel
// instruction-bound (69 % issue-active at 50 % of HBM bandwidth).
__device__ __forceinline__ float adam_one(const AdamArgs& a, uint64_t k, float w, float g0,
                                          float& m, float& v) {
    const float g = g0 * a.gscale + a.l2 * w;
    m = a.b1 * m + (1.0f - a.b1) * g;
    v = a.b2 * v + (1.0f - a.b2) * g * g;
    const float lr = k < a.rrs_first ? a.lr : a.lr_rrs;
    return w - __fdividef(lr * (m * a.inv_c1), sqrtf(v * a.inv_c2) + a.eps);
}

// the moving average after an Adam step: e = d e + (1 - d) w, pi = e / (1 - d^t), each product
// and the sum rounded separately (no contraction), so a float32 restatement gives the same bits
__device__ __forceinline__ float ema_one(const AdamArgs& a, float w, float& e) {
    e = __fadd_rn(__fmul_rn(a.d, e), __fmul_rn(a.omd, w));
    return __fmul_rn(e, a.inv);
}

// four parameters from k on into an FP16 table of n
__device__ __forceinline__ void store_half4(__half* table, uint64_t n, uint64_t k, float4 x) {
    if (k + 4 <= n) {
        __half2 h0 = __floats2half2_rn(x.x, x.y), h1 = __floats2half2_rn(x.z, x.w);
        uint2 u;
        u.x = *reinterpret_cast<uint32_t*>(&h0);
        u.y = *reinterpret_cast<uint32_t*>(&h1);
        // 4-byte stores where the table's shift is an odd number of rows
        uint32_t* d = reinterpret_cast<uint32_t*>(table + k);
        if ((reinterpret_cast<uintptr_t>(d) & 7u) == 0) *reinterpret_cast<uint2*>(d) = u;
        else d[0] = u.x, d[1] = u.y;
    } else {
        const float nv[4] = {x.x, x.y, x.z, x.w};
        for (int j = 0; j < 4; ++j)
            if (k + j < n) table[k + j] = __float2half_rn(nv[j]);
    }
}

// HBM-bound (30 B per parameter, 42 with the moving average): four parameters per thread with
// 16-byte loads and stores; the FP16 copies of the table and the moving average, whose weight is
// at hand here, are written in the same pass. The arrays are 16-byte aligned; a scalar tail
// finishes, and the moving average goes on over the parameters that this step does not train. The
// shipped configuration: 38 us, and 24 + 22 with the average in a kernel of its own of 4-byte
// accesses.
template <bool EMA>
__global__ void k_adam(const __grid_constant__ AdamArgs a) {
    const uint64_t quads = a.count / 4;
    for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < quads;
         q += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = 4 * q;
        const float4 w = *reinterpret_cast<const float4*>(a.p + k);
        const float4 g = *reinterpret_cast<const float4*>(a.g + k);
        float4 m = *reinterpret_cast<const float4*>(a.m + k);
        float4 v = *reinterpret_cast<const float4*>(a.v + k);
        float4 e;
        if constexpr (EMA) e = *reinterpret_cast<const float4*>(a.e + k);
        float4 nw;
        nw.x = adam_one(a, k, w.x, g.x, m.x, v.x);
        nw.y = adam_one(a, k + 1, w.y, g.y, m.y, v.y);
        nw.z = adam_one(a, k + 2, w.z, g.z, m.z, v.z);
        nw.w = adam_one(a, k + 3, w.w, g.w, m.w, v.w);
        *reinterpret_cast<float4*>(a.m + k) = m;
        *reinterpret_cast<float4*>(a.v + k) = v;
        *reinterpret_cast<float4*>(a.p + k) = nw;
        if (a.table_h && k < a.n_table) store_half4(a.table_h, a.n_table, k, nw);
        if constexpr (EMA) {
            float4 pi;
            pi.x = ema_one(a, nw.x, e.x);
            pi.y = ema_one(a, nw.y, e.y);
            pi.z = ema_one(a, nw.z, e.z);
            pi.w = ema_one(a, nw.w, e.w);
            *reinterpret_cast<float4*>(a.e + k) = e;
            *reinterpret_cast<float4*>(a.pi + k) = pi;
            if (a.table_hi && k < a.n_table) store_half4(a.table_hi, a.n_table, k, pi);
        }
    }
    for (uint64_t k = 4 * quads + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
         k < (EMA ? a.n_params : a.count); k += (uint64_t)gridDim.x * blockDim.x) {
        float nw = a.p[k];
        if (k < a.count) {
            float m = a.m[k], v = a.v[k];
            nw = adam_one(a, k, nw, a.g[k], m, v);
            a.m[k] = m;
            a.v[k] = v;
            a.p[k] = nw;
            if (a.table_h && k < a.n_table) a.table_h[k] = __float2half_rn(nw);
        }
        if constexpr (EMA) {
            float e = a.e[k];
            const float pi = ema_one(a, nw, e);
            a.e[k] = e;
            a.pi[k] = pi;
            if (a.table_hi && k < a.n_table) a.table_hi[k] = __float2half_rn(pi);
        }
    }
}

// after_stat() is called once the StatNet kernel is launched (the step forks the table-gradient
// scatter there)
template <int WS, int HS, int WR, int HR, class AfterStat>
cudaError_t launch_train(nrrs_ctx* ctx, TrainArgs& a, cudaStream_t s, AfterStat after_stat) {
    constexpr int kThr = TrShape<WS>::kThr;
    const size_t smem = TrShape<WS>::kSmem;
    auto ks = k_train_stat<WS, HS, WR, HR>;
    auto kr = k_train_rrs<WR, HR>;
    cudaError_t e = cudaFuncSetAttribute(ks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const uint32_t tiles = (a.n + kTM - 1) / kTM;
    uint32_t grid = (uint32_t)(ctx->sm_count * resident_ctas((const void*)ks, kThr, smem, 16));
    if (grid > tiles) grid = tiles;
    a.part_n = grid;
    {
        ProfScope ps(ctx, NRRS_KERNEL_TRAIN_STAT, s);
        e = launch_early(ks, grid, kThr, smem, 0, s, a);
    }
    if (e != cudaSuccess || (e = after_stat()) != cudaSuccess) return e;
    ProfScope ps(ctx, NRRS_KERNEL_TRAIN_RRS, s);
    return launch_early(kr, grid, kThr, smem, 0, s, a);
}

struct Layout {
    uint32_t r_x0, r_hs, r_dhs, r_dx, r_dy, r_x1, r_hr, r_dhr, r_draw, rows;
};

Layout layout_of(const nrrs_config& c, bool compact) {
    Layout L{};
    uint32_t r = 0;
    const bool ref = c.network == NRRS_NET_REFERENCE;
    L.r_x0 = r; r += ref ? kRefStatIn : 56;
    L.r_hs = r; r += c.statnet_hidden * c.statnet_width;
    L.r_dhs = r; r += c.statnet_hidden * c.statnet_width;
    L.r_dx = r; r += compact ? 0 : 2 * c.n_levels;
    L.r_dy = r; r += ref ? 8 : 4;
    L.r_x1 = r; r += 16;
    L.r_hr = r; r += c.rrsnet_hidden * c.rrsnet_width;
    L.r_dhr = r; r += c.rrsnet_hidden * c.rrsnet_width;   // at least 2 * n_levels rows
    if (compact) L.r_dx = L.r_dhr;
    L.r_draw = r; r += 4;
    L.rows = r;
    return L;
}

uint32_t ld_of(uint32_t n) { return (n + 127) / 128 * 128; }

}  // namespace

cudaError_t launch_wreduce(const float* partial, uint32_t chunks, uint32_t stride, uint32_t count,
                           float* grad, float scale, cudaStream_t s) {
    return launch_early(k_wreduce, (count + 31) / 32, 32u * kRedSlices, 0, 0, s, partial, chunks,
                        stride, count, grad, scale);
}

// Adam over the trained parameters: table + StatNet (+ RRSNet at step 3); refreshes the FP16
// tables and the moving average of every parameter (the caller rebuilds the other derived images)
cudaError_t launch_adam_step(nrrs_ctx* ctx, bool train_rrs, cudaStream_t s, float scale) {
    const nrrs_config& c = ctx->cfg;
    ctx->adam_t += 1;
    AdamArgs ad{};
    ad.p = ctx->params;
    ad.g = ctx->grads;
    ad.gscale = scale;
    ad.m = ctx->adam_m;
    ad.v = ctx->adam_v;
    ad.table_h = ctx->table_h ? ctx->table_h + 2 * ctx->shift_h : nullptr;
    ad.n_table = ctx->n_table;
    ad.count = ctx->n_table + ctx->n_stat + (train_rrs ? ctx->n_rrs : 0);
    ad.lr = c.lr;
    ad.rrs_first = ctx->n_table + ctx->n_stat;
    ad.lr_rrs = c.lr_rrsnet > 0.f ? c.lr_rrsnet : c.lr;
    ad.b1 = c.beta1;
    ad.b2 = c.beta2;
    ad.eps = c.eps;
    ad.l2 = c.l2_reg;
    ad.inv_c1 = 1.0f / (1.0f - powf(c.beta1, (float)ctx->adam_t));
    ad.inv_c2 = 1.0f / (1.0f - powf(c.beta2, (float)ctx->adam_t));
    if (ctx->ema) {
        ctx->ema_t += 1;
        ad.e = ctx->ema;
        ad.pi = ctx->params_inf;
        ad.table_hi = ctx->table_h_inf ? ctx->table_h_inf + 2 * ctx->shift_h : nullptr;
        ad.n_params = ctx->n_params;
        ad.d = c.ema_decay;
        ad.omd = 1.0f - c.ema_decay;
        ad.inv = (float)(1.0 / (1.0 - std::pow((double)c.ema_decay, (double)ctx->ema_t)));
    }
    {
        ProfScope ps(ctx, NRRS_KERNEL_ADAM, s);
        const unsigned grid = (unsigned)ctx->sm_count * 8;
        if (ctx->ema) k_adam<true><<<grid, 256, 0, s>>>(ad);
        else k_adam<false><<<grid, 256, 0, s>>>(ad);
    }
    return cudaGetLastError();
}

bool train_tc_supported(const nrrs_config& c);
size_t train_tc_scratch_bytes(const nrrs_config& c, uint32_t n, int sm_count);
int train_step_tc(nrrs_ctx* ctx, const VertexPtrs& v, const float* target, uint32_t n,
                  double* loss_dev, cudaStream_t s, bool apply, const LossWeights* lw);

size_t train_scratch_bytes(const nrrs_config& c, uint32_t n, int sm_count, bool compact) {
    if (train_tc_supported(c)) return train_tc_scratch_bytes(c, n, sm_count);
    const Layout L = layout_of(c, compact);
    const uint64_t mlp = (uint64_t)64 * c.statnet_width + (uint64_t)(c.statnet_hidden - 1) *
                         c.statnet_width * c.statnet_width + 3ull * c.statnet_width +
                         16ull * c.rrsnet_width + (uint64_t)(c.rrsnet_hidden - 1) * c.rrsnet_width *
                         c.rrsnet_width + (uint64_t)c.rrsnet_width;
    const uint64_t chunks = wgrad_chunks_max(n, compact);
    return sizeof(float) * (uint64_t)L.rows * ld_of(n) + sizeof(double) * 4 * (uint64_t)sm_count * 16 +
           sizeof(float) * chunks * mlp + 1024;
}

int train_step_impl(nrrs_ctx* ctx, const VertexPtrs& v, const float* target, uint32_t n,
                    double* loss_dev, cudaStream_t s, bool apply, const LossWeights* lw) {
    if (train_tc_supported(ctx->cfg))
        return train_step_tc(ctx, v, target, n, loss_dev, s, apply, lw);
    const nrrs_config& c = ctx->cfg;
    const Layout L = layout_of(c, ctx->train_compact);
    const uint32_t ld = ld_of(c.max_train);
    const uint32_t chunk = wgrad_chunk(n, ctx->train_compact);
    const uint64_t chunks = (n + chunk - 1) / chunk;
    const uint64_t mlp = ctx->n_stat + ctx->n_rrs;
    uint8_t* base = reinterpret_cast<uint8_t*>(ctx->train_scratch);
    float* act = reinterpret_cast<float*>(base);
    double* part = reinterpret_cast<double*>(base + sizeof(float) * (size_t)L.rows * ld);
    float* partial = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(part) +
                                              sizeof(double) * 4 * (size_t)ctx->sm_count * 16);
    const bool train_rrs = c.step >= 3;
    cudaError_t e;

    // gradients of this step only: the scatter zeroes the table's, the weight gradients write
    // theirs, and an untrained RRSNet's are zero
    e = train_rrs ? cudaSuccess
                  : cudaMemsetAsync(ctx->grads + ctx->n_table + ctx->n_stat, 0,
                                    sizeof(float) * ctx->n_rrs, s);
    if (e != cudaSuccess) {
        ctx->last_error = std::string("train memset: ") + cudaGetErrorString(e);
        return NRRS_ERR_CUDA;
    }

    TrainArgs a{};
    a.v = v;
    a.target = target;
    a.n = n;
    a.ld = ld;
    a.fp.stat_eps = c.stat_eps;
    a.fp.ref_eps = c.ref_eps;
    a.loss_clamp = c.loss_clamp_max;
    a.cost_offset = c.cost_offset;
    a.train_rrs = train_rrs;
    a.wt_stat = ctx->wt;
    a.wt_rrs = ctx->wt + ctx->wt_rrs_offset;
    a.w_stat = ctx->wrow;
    a.w_rrs = ctx->wrow + ctx->n_stat;
    a.act = act;
    a.r_x0 = L.r_x0; a.r_hs = L.r_hs; a.r_dhs = L.r_dhs; a.r_dx = L.r_dx; a.r_dy = L.r_dy;
    a.r_x1 = L.r_x1; a.r_hr = L.r_hr; a.r_dhr = L.r_dhr; a.r_draw = L.r_draw;
    a.part = part;
    a.loss_out = loss_dev ? loss_dev : ctx->loss_dev;
    if (lw) a.lw = *lw;

    // the hash rows of x0, level-major
    EncodeF32Args ea{};
    ea.enc = ctx->enc;
    ea.segs.n = 1;
    ea.segs.s[0].count = n;
    ea.segs.total_tiles = (n + kTile - 1) / kTile;
    ea.pos = v.pos;
    ea.table = ctx->params;
    ea.out = act + (size_t)L.r_x0 * ld;
    ea.tile_stride = kTile;
    ea.lane_stride = ld;
    ea.tile_end = ea.segs.total_tiles;
    {
        ProfScope ps(ctx, NRRS_KERNEL_TRAIN_ENCODE, s);
        e = launch_encode_f32(ea, ctx->sm_count, s);
    }
    if (e != cudaSuccess) {
        ctx->last_error = std::string("training encoding launch: ") + cudaGetErrorString(e);
        return NRRS_ERR_CUDA;
    }
    // The scatter is bound by L2 reductions, the RRSNet kernel and the weight gradients by the
    // FP32 pipe: it runs beside them on the context's side stream, forked after the StatNet
    // kernel and joined before Adam (nothing in between reads the table gradient).
    // (In the compact layout the RRSNet kernel overwrites the lane gradients: the scatter stays on
    // the caller's stream.)
    bool forked = false;
    auto after_stat = [&]() -> cudaError_t {
        const LaneGrads g{act + (size_t)L.r_dx * ld, 2 * (size_t)ld, 1, ld, 1.0f};
        if (ctx->train_compact) return launch_scatter_table(ctx, v.pos, n, g, s);
        cudaError_t ef = cudaEventRecord(ctx->ev_fork, s);
        if (ef == cudaSuccess) ef = cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0);
        if (ef != cudaSuccess) return ef;
        forked = true;
        ef = launch_scatter_table(ctx, v.pos, n, g, ctx->side);
        const cudaError_t ej = cudaEventRecord(ctx->ev_join, ctx->side);
        return ef != cudaSuccess ? ef : ej;
    };
    auto join = [&]() {
        if (forked) cudaStreamWaitEvent(s, ctx->ev_join, 0);
        forked = false;
    };
    if (c.statnet_width == 64 && c.statnet_hidden == 2)
        e = launch_train<64, 2, 64, 2>(ctx, a, s, after_stat);
    else if (c.statnet_width == 64 && c.statnet_hidden == 3)
        e = launch_train<64, 3, 64, 3>(ctx, a, s, after_stat);
    else if (c.statnet_width == 32)   // the reference network
        e = launch_train<32, 3, 32, 3>(ctx, a, s, after_stat);
    else
        e = launch_train<128, 3, 128, 3>(ctx, a, s, after_stat);
    if (e != cudaSuccess) {
        join();
        ctx->last_error = std::string("train launch: ") + cudaGetErrorString(e);
        return NRRS_ERR_CUDA;
    }

    // weight-gradient jobs: (delta rows, activation rows, M, N, layer input width, offset)
    WGradArgs w{};
    w.act = act;
    w.ld = ld;
    w.n = n;
    w.chunk = chunk;
    w.partial = partial;
    w.total = (uint32_t)mlp;
    const uint32_t WS = c.statnet_width, HS = c.statnet_hidden;
    const uint32_t WR = c.rrsnet_width, HR = c.rrsnet_hidden;
    const bool ref = c.network == NRRS_NET_REFERENCE;
    const uint32_t sin = stat_in_of((int)WS), sout = stat_out_of((int)WS);
    int nj = 0;
    uint32_t off = 0;
    nj += add_layer_jobs(w.job + nj, L.r_dhs, L.r_x0, WS, ref ? (uint32_t)kRefStatIn : 56u, sin, off);
    off += WS * sin;
    for (uint32_t h = 1; h < HS; ++h) {
        nj += add_layer_jobs(w.job + nj, L.r_dhs + h * WS, L.r_hs + (h - 1) * WS, WS, WS, WS, off);
        off += WS * WS;
    }
    nj += add_layer_jobs(w.job + nj, L.r_dy, L.r_hs + (HS - 1) * WS, sout, WS, WS, off);
    off += sout * WS;
    if (train_rrs) {
        nj += add_layer_jobs(w.job + nj, L.r_dhr, L.r_x1, WR, ref ? (uint32_t)kRefRrsLanes : 10u,
                             kRrsIn, off);
        off += WR * kRrsIn;
        for (uint32_t h = 1; h < HR; ++h) {
            nj += add_layer_jobs(w.job + nj, L.r_dhr + h * WR, L.r_hr + (h - 1) * WR, WR, WR, WR, off);
            off += WR * WR;
        }
        nj += add_layer_jobs(w.job + nj, L.r_draw, L.r_hr + (HR - 1) * WR, 1, WR, WR, off);
        off += WR;
    }
    e = cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWSmem);
    if (e == cudaSuccess) {
        ProfScope ps(ctx, NRRS_KERNEL_TRAIN_WGRAD, s);
        e = launch_early(k_wgrad, dim3((unsigned)chunks, (unsigned)nj), kWThr, kWSmem, 0, s, w);
    }
    if (e == cudaSuccess) {
        // the first `off` entries have partials; gradients of untrained layers stay zero
        ProfScope ps(ctx, NRRS_KERNEL_TRAIN_REDUCE, s);
        e = launch_wreduce(partial, (uint32_t)chunks, (uint32_t)mlp, off, ctx->grads + ctx->n_table,
                           1.0f, s);
    }
    join();  // the table gradient is complete on s from here
    if (e != cudaSuccess) {
        ctx->last_error = std::string("wgrad launch: ") + cudaGetErrorString(e);
        return NRRS_ERR_CUDA;
    }

    if (!apply) return NRRS_OK;
    e = launch_adam_step(ctx, train_rrs, s);
    if (e != cudaSuccess) {
        ctx->last_error = std::string("adam launch: ") + cudaGetErrorString(e);
        return NRRS_ERR_CUDA;
    }
    return NRRS_OK;
}

}  // namespace nrrs
