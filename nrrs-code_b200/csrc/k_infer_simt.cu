// k_infer_simt.cu -- plain FP32 inference: hash grid + SH encoding, StatNet, glue, RRSNet,
// activation, clamp and the exact normalisation sum, on the FP32 SIMT pipes.
//
// This is the "plain FP32 per-depth path" the mixed-precision tcgen05 path is measured
// against. It fuses what the reference runs as nrrs_generate_inference_data (train.cu:269-287),
// tcnn inference_mixed_precision x2 (myNetworkLL2.cpp:206, network.cpp:346),
// nrrs_generate_inference_data_from_0to1 (train.cu:41-112) and the "Gen RRS Number" lambda
// (integrator.cpp:1184-1298), so the AoS round trips of the reference disappear.
//
// A CTA works on 64 vertices at a time (half of a 128-vertex tile of the segment table) with 64
// threads (128 for the 128-wide networks). Their activations live in one shared-memory tile;
// every hidden layer is a register-tiled FP32 GEMM in place on it (simt_gemm.cuh). The encoding,
// the narrow layers (3 and 1 outputs), the glue, the factor and the exact-sum term run one thread
// per vertex on that vertex's column of the tile (with 128 threads, two for the encoding).
// Every output is accumulated as fmaf(w_k, x_k, acc) over k ascending, the same sequence for any
// launch shape.
// The hash features come from the encoding kernel (k_encode.cu), in passes of at most 1,048,576
// vertices, through the context's feature scratch: for the steps, which use the context's scratch in
// any case (the sum, the decision). Calls that only infer keep nothing in the context, so that they
// may overlap on several streams and with a step: for them this kernel gathers for itself (GATHER),
// with 128 threads, whose two per vertex halve the rounds of loads. 64 x 2 networks, 65,536 vertices,
// us per step with the decision, inputs and table in L2 / evicted: 75 / 87 with the encoding kernel
// (24 us of it, and 47 for this one), 75 / 91 gathering; the FMA pipe's floor is 24 us. Inference
// alone, gathering: 67 us, and 107 when an 8-byte load per corner and plain FMAs made it up.
#include "simt_gemm.cuh"

namespace nrrs {

namespace {

using simt::at;
using simt::kTM;

template <int W, int NT>
struct FpShape {
    static constexpr int kActFloats = simt::imax(stat_in_of(W), W) * kTM;
    static constexpr int kChunkFloats = simt::kKC * W;
    static constexpr size_t kSmem = sizeof(float) * (kActFloats + 2 * kChunkFloats);
};

// out[n][m] = act(sum_k wt[k][n] act[k][m]) for k < k_eff, in place on the activation tile, with
// ReLU (the workload's network) or LeakyReLU (the reference network, W = 32); wt is [in][W] in
// global memory (input lanes from k_eff on are zero)
template <int W, int NT>
__device__ __forceinline__ void hidden_layer(const float* __restrict__ wt, int k_eff, float* act,
                                             float* wch, int tid) {
    simt::tile_gemm<W, NT>(
        wt, W, k_eff, act, wch, tid, [&](int, int n, int m0, const float* v) {
            float r[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = W == 32 ? leaky(v[i]) : fmaxf(v[i], 0.f);
            simt::tile_store8(act, n, m0, r);
        });
}

// resident CTAs per SM: 64 x 2 networks gathering with 128 threads, 65,536 vertices, 5 a SM 74.6 / 91.1
// us a step, 4 76.6 / 93.2, 6 74.1 / 93.2; the 128-wide ones spill at 5 (278 us, 261 at 4)
template <int WS, int NT, bool GATHER>
constexpr int min_ctas() {
    return NT == 64 ? 8 : (GATHER && WS == 64 ? 5 : 4);
}

template <int WS, int HS, int WR, int HR, int NT, bool GATHER>
__global__ void __launch_bounds__(NT, min_ctas<WS, NT, GATHER>())
    k_infer_fp32(const __grid_constant__ InferArgs a) {
    static_assert(WS == WR, "one tile shape for both networks");
    constexpr bool REF = WS == 32;             // the reference's shipped network
    constexpr int SIN = stat_in_of(WS), SOUT = stat_out_of(WS);
    constexpr int TPS = NT / kTM;         // threads per vertex of the encoding
    extern __shared__ float4 smem4[];
    float* act = reinterpret_cast<float*>(smem4);
    float* wch = act + FpShape<WS, NT>::kActFloats;
    wait_for_stream();
    const int tid = threadIdx.x;
    const int m = tid & (kTM - 1);
    const bool lead = tid < kTM;               // the thread that owns vertex column m
    const SegmentTable& ST = seg_table(a.segs);
    const uint32_t tile_end = min(a.tile_end, ST.total_tiles);
    const uint32_t items = tile_end > a.tile_begin ? 2u * (tile_end - a.tile_begin) : 0u;
    // transposed layer images: [in][out] (outputs padded to 4), StatNet then RRSNet
    const float* s0 = a.wt_stat;
    const float* s_out = s0 + (size_t)SIN * WS + (size_t)(HS - 1) * WS * WS;
    const float* r0 = a.wt_rrs;
    const float* r_out = r0 + (size_t)kRrsIn * WR + (size_t)(HR - 1) * WR * WR;

#pragma unroll 1
    for (uint32_t u = blockIdx.x; u < items; u += gridDim.x) {
        const uint32_t t = a.tile_begin + (u >> 1);
        const int si = find_segment(ST, t);
        const Segment& sg = ST.s[si];
        const uint32_t i = sg.offset + (t - sg.tile_start) * kTile + (u & 1u) * kTM + m;
        const bool valid = i < sg.offset + sg.count;
        __syncthreads();   // the previous item's column reads are over
        // the hash features, and the other input lanes (one thread per vertex, or two)
        const bool lo = TPS == 1 || lead, hi = TPS == 1 || !lead;
        constexpr int HL = 2 * (REF ? kRefLevels : kMaxLevels);
        if constexpr (GATHER) {
            constexpr int NL = HL / 2 / TPS;     // levels per thread
            const int l0 = lo ? 0 : NL;
            float p[3] = {0.f, 0.f, 0.f};
            if (valid) norm_pos(a.enc, a.v.pos, i, p);
#pragma unroll 2
            for (int l = l0; l < l0 + NL; ++l) {
                float2 f = make_float2(0.f, 0.f);
                if (valid) {
                    const LevelDev L = a.enc.lv[l];
                    f = simt::level_features_f(reinterpret_cast<const float2*>(a.table), L,
                                               a.enc.hash_mask, cell_of(p, L.res));
                }
                act[at(2 * l, m)] = f.x;
                act[at(2 * l + 1, m)] = f.y;
            }
        } else {
            simt::load_rows<HL, NT>(a.feat + (size_t)(t - a.tile_begin) * kF32TileFloats +
                                             (u & 1u) * kTM,
                                         kTile, act, tid);
            simt::cp_async_commit();
        }
        if (valid) {
            if (REF) {
                float blob[16];
                ref_blob_lanes(a.v, i, blob);
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    if (k < 8 ? lo : hi) act[at(HL + k, m)] = blob[k];
            } else {
                if (lo) {
                    float sh[16];
                    const size_t i3 = 3 * (size_t)i;
                    sh16(a.v.wi[i3], a.v.wi[i3 + 1], a.v.wi[i3 + 2], sh);
#pragma unroll
                    for (int k = 0; k < 16; ++k) act[at(32 + k, m)] = sh[k];
                }
                if (hi) {
                    float misc[16];
                    misc_lanes(a.v, i, misc);
#pragma unroll
                    for (int k = 0; k < 8; ++k) act[at(48 + k, m)] = misc[k];
                }
            }
        } else {
            constexpr int NO = REF ? 16 : 24;    // non-hash lanes; `hi` owns the last 8
            for (int k = lo ? 0 : NO - 8; k < (hi ? NO : NO - 8); ++k) act[at(HL + k, m)] = 0.f;
        }
        VertexAux aux{};
        if (lead && valid) aux = load_aux(a.v, i);
        // StatNet: 56 live input lanes (48..55 misc, 56..63 zero); the reference network's 32
        hidden_layer<WS, NT>(s0, REF ? 32 : 56, act, wch, tid);
#pragma unroll 1
        for (int h = 1; h < HS; ++h)
            hidden_layer<WS, NT>(s0 + (size_t)SIN * WS + (size_t)(h - 1) * WS * WS, WS, act, wch, tid);
        float y[SOUT];
#pragma unroll
        for (int k = 0; k < SOUT; ++k) y[k] = 0.f;
        if (lead) {
            simt::narrow_out<WS, SOUT>(s_out, act, m, y);
            // glue: the RRSNet input in this vertex's column (10 live lanes; the reference's 12)
            float x1[16];
            if (REF) glue16_ref_aux(y, aux, x1);
            else glue16_aux(a.fp, y, aux, x1);
#pragma unroll
            for (int k = 0; k < (REF ? kRefRrsLanes : 10); ++k) act[at(k, m)] = x1[k];
        }
        hidden_layer<WR, NT>(r0, REF ? kRefRrsLanes : 10, act, wch, tid);
#pragma unroll 1
        for (int h = 1; h < HR; ++h)
            hidden_layer<WR, NT>(r0 + (size_t)kRrsIn * WR + (size_t)(h - 1) * WR * WR, WR, act, wch, tid);
        long long term = 0;
        if (lead && valid) {
            float raw;
            simt::narrow_out<WR, 1>(r_out, act, m, &raw);
            const float rrs = rrs_factor_aux<REF>(a.fp, y, raw, aux);
            if (a.stats) {
#pragma unroll
                for (int k = 0; k < SOUT; ++k) a.stats[SOUT * (size_t)i + k] = y[k];
            }
            a.rrs[i] = rrs;
            if (a.scr || a.ext_acc)
                term = fixed_term(a.fp, rrs, a.scr ? &a.scr->status : &g_dummy_status);
        }
        if (a.scr || a.ext_acc) {
            term = warp_sum_ll(term);
            if ((tid & 31) == 0 && term != 0)
                atomicAdd(a.ext_acc ? a.ext_acc : &a.scr->sum_acc[si], (unsigned long long)term);
        }
    }
}

template <int WS, int HS, int WR, int HR, int NT, bool GATHER>
cudaError_t launch_shape(const InferArgs& a, int sm_count, int ctas_per_sm, cudaStream_t s) {
    using S = FpShape<WS, NT>;
    auto kern = k_infer_fp32<WS, HS, WR, HR, NT, GATHER>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)S::kSmem);
    if (e != cudaSuccess) return e;
    int per_sm = resident_ctas((const void*)kern, NT, S::kSmem, 32);
    if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
    const uint32_t items = 2u * (a.tile_end - a.tile_begin);
    unsigned grid = (unsigned)(sm_count * per_sm);
    if (grid > items) grid = items;
    if (grid == 0) return cudaSuccess;
    g_last_grid = (int)grid;
    return launch_early(kern, grid, NT, S::kSmem, 0, s, a);
}

template <int WS, int HS, int WR, int HR>
cudaError_t launch_cfg(const InferArgs& a, int sm_count, int ctas_per_sm, cudaStream_t s) {
    constexpr int NT = simt::threads_of(WS);
    if (a.feat) return launch_shape<WS, HS, WR, HR, NT, false>(a, sm_count, ctas_per_sm, s);
    // The 32-wide network's chain is short beside its 8 levels of gathers: past one wave of 4 CTAs of
    // 128 threads, more CTAs of 64 threads hide them better (65,536 vertices 36 us against 46, 20,000
    // the same; 3,071 17 against 13.5). The 64-wide networks are faster with 128 threads at every
    // size (1 vertex 17 us against 25, 65,536 69 against 82, 1,048,576 939 against 1,202).
    if constexpr (WS == 32)
        if (2u * (a.tile_end - a.tile_begin) > 4u * (uint32_t)sm_count)
            return launch_shape<WS, HS, WR, HR, 64, true>(a, sm_count, ctas_per_sm, s);
    return launch_shape<WS, HS, WR, HR, 128, true>(a, sm_count, ctas_per_sm, s);
}

}  // namespace

cudaError_t launch_infer_fp32(const InferArgs& a, int ws, int hs, int wr, int hr, int sm_count,
                              int ctas_per_sm, cudaStream_t s) {
    if (ws == 64 && hs == 2 && wr == 64 && hr == 2)
        return launch_cfg<64, 2, 64, 2>(a, sm_count, ctas_per_sm, s);
    if (ws == 128 && hs == 3 && wr == 128 && hr == 3)
        return launch_cfg<128, 3, 128, 3>(a, sm_count, ctas_per_sm, s);
    if (ws == 64 && hs == 3 && wr == 64 && hr == 3)
        return launch_cfg<64, 3, 64, 3>(a, sm_count, ctas_per_sm, s);
    if (ws == 32 && hs == 3 && wr == 32 && hr == 3)   // the reference network
        return launch_cfg<32, 3, 32, 3>(a, sm_count, ctas_per_sm, s);
    return cudaErrorInvalidValue;
}

template <int WS, int HS, int WR, int HR>
int max_ctas_fp32() {
    constexpr int NT = simt::threads_of(WS);
    using S = FpShape<WS, NT>;
    auto kern = k_infer_fp32<WS, HS, WR, HR, NT, false>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem) !=
        cudaSuccess)
        return 0;
    return resident_ctas((const void*)kern, NT, S::kSmem, 32);
}

int infer_max_ctas_fp32(int ws, int hs) {
    if (ws == 64 && hs == 2) return max_ctas_fp32<64, 2, 64, 2>();
    if (ws == 64 && hs == 3) return max_ctas_fp32<64, 3, 64, 3>();
    if (ws == 128 && hs == 3) return max_ctas_fp32<128, 3, 128, 3>();
    if (ws == 32 && hs == 3) return max_ctas_fp32<32, 3, 32, 3>();
    return 0;
}

}  // namespace nrrs
