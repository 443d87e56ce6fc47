// k_util.cu -- derived weight images and the FP16 table copy.
//
// The FP32 master weights are row-major W[out][in] per layer. Two derived images are rebuilt
// after every optimizer step or parameter upload:
//   * FP32 transposed Wt[in][out4] (out padded to a multiple of 4) for the SIMT path;
//   * FP16/BF16 UMMA image: per layer an [Npad][K] K-major operand in the canonical
//     no-swizzle core-matrix layout of tcgen05 (8 rows x 16 bytes per core matrix, adjacent
//     K core matrices 128 B apart (LBO), adjacent 8-row groups K*16 B apart (SBO)).
//     The output layers are padded to N = 16 rows with zeros.
#include "kernels.hpp"

namespace nrrs {

namespace {

struct LayerDesc {
    int in, out;
};

__host__ __device__ inline int pad4(int x) { return (x + 3) / 4 * 4; }
__host__ __device__ inline int npad16(int x) { return (x + 15) / 16 * 16; }

// layer list of a network: in -> w (hidden) -> out
__host__ __device__ inline LayerDesc layer_of(int in, int w, int hidden, int out, int l) {
    LayerDesc d;
    d.in = l == 0 ? in : w;
    d.out = l == hidden ? out : w;
    return d;
}

// element offset of (n, k) in a K-major core-matrix image with K columns
__host__ __device__ inline size_t umma_offset(int n, int k, int K) {
    return (size_t)(n >> 3) * (size_t)(K * 8) + (size_t)(k >> 3) * 64 + (size_t)(n & 7) * 8 +
           (size_t)(k & 7);
}

__device__ __forceinline__ uint16_t to_bits(float v, bool bf) {
    if (bf) {
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        return *reinterpret_cast<const uint16_t*>(&b);
    }
    const __half h = __float2half_rn(v);
    return *reinterpret_cast<const uint16_t*>(&h);
}

// The MLP images. The UMMA images hold per layer an [Npad][K] operand; in the training image
// StatNet is FP16 (its deltas are bounded) and RRSNet BF16 (its loss gradient r^2/q^2 can exceed
// FP16's range); its backward passes read the same bytes as MN-major operands, which is W^T, so no
// transposed copy is kept. One thread per (network, layer, n, k) of the padded images, grid-stride
// over the `threads` threads of which this is number `t0`.
__device__ __forceinline__ void pack_images(const PackArgs& a, size_t t0, size_t threads) {
    size_t mofs = 0, tofs = 0, pofs = 0;
    for (int net = 0; net < 2; ++net) {
        const int in = net == 0 ? stat_in_of(a.ws) : kRrsIn;
        const int w = net == 0 ? a.ws : a.wr;
        const int h = net == 0 ? a.hs : a.hr;
        const int out = net == 0 ? stat_out_of(a.ws) : 1;
        for (int l = 0; l <= h; ++l) {
            const LayerDesc d = layer_of(in, w, h, out, l);
            const int op4 = pad4(d.out);
            const int np = l == h ? npad16(d.out) : d.out;
            const size_t cells = (size_t)np * d.in;
            for (size_t e = t0; e < cells; e += threads) {
                const int n = (int)(e / d.in), k = (int)(e % d.in);
                const float v = n < d.out ? a.master[mofs + (size_t)n * d.in + k] : 0.f;
                if (n < op4) a.wt[tofs + (size_t)k * op4 + n] = v;
                if (n < d.out && a.wrow) a.wrow[mofs + (size_t)n * d.in + k] = v;
                const size_t o = pofs + umma_offset(n, k, d.in);
                if (a.wpack)
                    reinterpret_cast<uint16_t*>(a.wpack)[o] = to_bits(v, a.prec == NRRS_PREC_BF16);
                if (a.tpack) a.tpack[o] = to_bits(v, net == 1);
            }
            mofs += (size_t)d.out * d.in;
            tofs += (size_t)d.in * op4;
            pofs += cells;
        }
    }
}

// The cell image of the FP16 table's dense levels: cell (x, y, z) of level L gets its 8 corner
// entries (raw FP16 pairs) in corner order k = x-bit + 2 y-bit + 4 z-bit, the order in which
// the gathers sum them, so features from the image equal features from the table bit for bit.
// A warp takes whole (y, z) rows of cells, x over its lanes: contiguous reads, 32-byte stores.
__device__ __forceinline__ void cell_image(const uint32_t* __restrict__ rows, const EncodeParams& e,
                                           uint4* __restrict__ cells, uint32_t n_rows, uint32_t w0,
                                           uint32_t warps) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t l = 0, base = 0;
    for (uint32_t r = w0; r < n_rows; r += warps) {
        // the dense levels are a prefix of the levels (N_l grows with l)
        while (r - base >= e.lv[l].res * e.lv[l].res) {
            base += e.lv[l].res * e.lv[l].res;
            ++l;
        }
        const LevelDev L = e.lv[l];
        const uint32_t N = L.res, q = r - base, z = q / N, y = q - z * N;
        uint4* out = cells + 2 * ((size_t)L.cell + (size_t)N * q);
#pragma unroll 2
        for (uint32_t x = lane; x < N; x += 32) {
            uint32_t t[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                t[k] = rows[grid_row(L, e.hash_mask, x + (k & 1), y + ((k >> 1) & 1),
                                     z + ((k >> 2) & 1))];
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + 2 * x),
                         "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]),
                         "r"(t[6]), "r"(t[7])
                         : "memory");
        }
    }
}

constexpr unsigned kPackBlocks = 64;   // CTAs of one parameter vector's MLP images

// CTAs [0, 64 n_pack) pack, the rest build the cell images, side by side: the training step's three
// kernels after Adam (4.3 + 4.7 + 3.6 us at 64 x 2 and 2^19 entries, and the gaps between them) take
// 6.2 us as one; 24 + 7 + 4 us at 128 x 3 and 2^22 entries 23.7.
__global__ void __launch_bounds__(256) k_derive(const __grid_constant__ DeriveArgs a) {
    wait_for_stream();
    const unsigned nb = kPackBlocks * a.n_pack;
    if (blockIdx.x < nb) {
        pack_images(a.pack[blockIdx.x / kPackBlocks],
                    (blockIdx.x % kPackBlocks) * 256u + threadIdx.x, kPackBlocks * 256u);
        return;
    }
    const uint32_t warps = (gridDim.x - nb) * 8u, w0 = (blockIdx.x - nb) * 8u + (threadIdx.x >> 5);
    for (int k = 0; k < a.n_cell; ++k)
        cell_image(reinterpret_cast<const uint32_t*>(a.table_h[k]), a.enc, a.cells[k], a.cell_rows,
                   w0, warps);
}

__global__ void k_table_half(const float* t, __half* h, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        h[i] = __float2half_rn(t[i]);
}

}  // namespace

cudaError_t launch_derive(const DeriveArgs& a, int sm_count, cudaStream_t s) {
    const unsigned grid = kPackBlocks * a.n_pack + (a.n_cell ? (unsigned)sm_count * 8u : 0u);
    return grid ? launch_early(k_derive, grid, 256, 0, 0, s, a) : cudaSuccess;
}

thread_local int g_last_grid = 0;

int resident_ctas(const void* kern, int threads, size_t dyn_smem, int cap) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return 1;
    int dev = 0, smem_sm = 0, regs_sm = 0, thr_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    const size_t per_cta_smem = dyn_smem + fa.sharedSizeBytes + 1024;
    int by_smem = (int)((size_t)smem_sm / per_cta_smem);
    const int regs = (fa.numRegs + 7) / 8 * 8;  // allocation granularity per thread
    int by_regs = regs > 0 ? regs_sm / (regs * threads) : 32;
    int by_thr = thr_sm / threads;
    int n = by_smem < by_regs ? by_smem : by_regs;
    n = n < by_thr ? n : by_thr;
    n = n < cap ? n : cap;
    return n < 1 ? 1 : n;
}

size_t transposed_weight_floats(int ws, int hs, int wr, int hr) {
    size_t t = 0;
    for (int l = 0; l <= hs; ++l) {
        LayerDesc d = layer_of(stat_in_of(ws), ws, hs, stat_out_of(ws), l);
        t += (size_t)d.in * pad4(d.out);
    }
    for (int l = 0; l <= hr; ++l) {
        LayerDesc d = layer_of(kRrsIn, wr, hr, 1, l);
        t += (size_t)d.in * pad4(d.out);
    }
    return t;
}

size_t packed_weight_bytes(int ws, int hs, int wr, int hr) {
    size_t t = 0;
    for (int l = 0; l <= hs; ++l) {
        LayerDesc d = layer_of(stat_in_of(ws), ws, hs, stat_out_of(ws), l);
        t += (size_t)(l == hs ? npad16(d.out) : d.out) * d.in;
    }
    for (int l = 0; l <= hr; ++l) {
        LayerDesc d = layer_of(kRrsIn, wr, hr, 1, l);
        t += (size_t)(l == hr ? npad16(d.out) : d.out) * d.in;
    }
    return t * 2;
}

size_t train_pack_bytes(int ws, int hs, int wr, int hr) {
    size_t t = 0;
    for (int net = 0; net < 2; ++net) {
        const int in = net == 0 ? stat_in_of(ws) : kRrsIn;
        const int w = net == 0 ? ws : wr;
        const int h = net == 0 ? hs : hr;
        const int out = net == 0 ? stat_out_of(ws) : 1;
        for (int l = 0; l <= h; ++l) {
            const LayerDesc d = layer_of(in, w, h, out, l);
            t += (size_t)(l == h ? npad16(d.out) : d.out) * d.in;
        }
    }
    return t * 2;
}

cudaError_t launch_table_to_half(const float* t, __half* h, size_t n, cudaStream_t s) {
    k_table_half<<<148 * 4, 256, 0, s>>>(t, h, n);
    return cudaGetLastError();
}

}  // namespace nrrs
