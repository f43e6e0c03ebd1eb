// Weight pre-packing: the offline step before the GEMM (the reference's counterpart is the host-side format conversion
// mem_transfer<int8_t, float> of bfAintBGemm/mem_transfer.hpp:23-32, called once at bfAintBGemm.cc:96-97).
//
// Output layout AFB_LAYOUT_COL_PACKED: [N,K], K contiguous, same pitch rules as AFB_LAYOUT_COL; the stored integers are
// unchanged, only moved inside every 32-bit word to the places the kernels' cheap unpack reads as pairs:
//     int8: word bytes   [k0,k2,k1,k3]             int4: word nibbles [k0,k2,k4,k6,k1,k3,k5,k7]
// so that the unpack (dequant.cuh: bytes (0,2),(1,3) / nibbles (0,4),(1,5),(2,6),(3,7)) yields CONSECUTIVE k pairs and the
// activations can be used exactly as they lie in memory.  Input may be [N,K] (int8 or int4) or the reference's own
// [K,N] (int8), which is transposed on the way: that is how the reference's layout reaches the fast kernels.
#include "afb_internal.h"
#include "dequant.cuh"

namespace afb {
namespace {

__device__ __forceinline__ uint32_t pack_word8(uint32_t w) { return prmt(w, 0u, 0x3120u); }   // [b0,b2,b1,b3]
__device__ __forceinline__ uint32_t pack_word4(uint32_t w) {
    uint32_t e = w & 0x0f0f0f0fu, o = (w >> 4) & 0x0f0f0f0fu;     // even / odd nibbles, one per byte
    e = (e | (e >> 4)) & 0x00ff00ffu; e = (e | (e >> 8)) & 0xffffu;   // n0,n2,n4,n6 in 16 bits
    o = (o | (o >> 4)) & 0x00ff00ffu; o = (o | (o >> 8)) & 0xffffu;
    // wanted: nibble i of the output = weight perm[i], perm = [0,2,4,6,1,3,5,7]
    return e | (o << 16);
}

// [N,K] -> packed [N,K]: one 32-bit word per thread step
__global__ void __launch_bounds__(256) prepack_col_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t n, uint32_t row_bytes,
                                                          uint32_t in_pitch, uint32_t out_pitch, uint32_t bits) {
    const uint32_t words = row_bytes / 4;
    const size_t total = (size_t)n * words;
    for (size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x; id < total; id += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(id / words), wi = (uint32_t)(id % words);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(in + (size_t)r * in_pitch + wi * 4);
        *reinterpret_cast<uint32_t*>(out + (size_t)r * out_pitch + wi * 4) = bits == 8 ? pack_word8(w) : pack_word4(w);
    }
}

// [K,N] int8 -> packed [N,K]: a 32 (k) x 32 (n) tile through shared memory, so that both sides are coalesced
__global__ void __launch_bounds__(256) prepack_row_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t n, uint32_t k,
                                                          uint32_t in_pitch, uint32_t out_pitch) {
    __shared__ uint8_t tile[32][33];
    const uint32_t n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
    for (uint32_t r = ty; r < 32; r += 8)
        tile[r][tx] = (k0 + r < k && n0 + tx < n) ? in[(size_t)(k0 + r) * in_pitch + n0 + tx] : (uint8_t)0;
    __syncthreads();
    // 32 channels x 8 words of 4 k
    const uint32_t ch = threadIdx.x >> 3, wi = threadIdx.x & 7;
    if (n0 + ch < n && k0 + wi * 4 < k) {
        const uint32_t w = (uint32_t)tile[wi * 4][ch] | ((uint32_t)tile[wi * 4 + 1][ch] << 8) | ((uint32_t)tile[wi * 4 + 2][ch] << 16) |
                           ((uint32_t)tile[wi * 4 + 3][ch] << 24);
        *reinterpret_cast<uint32_t*>(out + (size_t)(n0 + ch) * out_pitch + k0 + wi * 4) = pack_word8(w);
    }
}

// The same for 16-byte aligned rows: a 128 (k) x 128 (n) tile per CTA.  A thread loads 16 channels of 4 consecutive k (four 16-byte
// loads in flight), transposes 4 x 4 byte blocks in registers straight into packed words, and the tile crosses shared memory once in
// words: both sides move whole 128-byte lines.  Word q of channel c lies at q ^ 4 * (c / 16 % 8), so that the transposing stores (8
// channel groups x 4 words per warp) and the 16-byte loads that follow are free of bank conflicts.  Bound by HBM (one read and one write
// of B): 4096 x 11008 18.4 us = 4.9 TB/s, the byte-wise kernel above 94 us.
__global__ void __launch_bounds__(256) prepack_row_wide_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t n, uint32_t k,
                                                               uint32_t in_pitch, uint32_t out_pitch) {
    __shared__ __align__(16) uint32_t tile[128][32];
    const uint32_t n0 = blockIdx.x * 128, k0 = blockIdx.y * 128;
    {
        const uint32_t cg = threadIdx.x & 7, q = threadIdx.x >> 3;   // 16 channels from n0 + 16 cg, k from k0 + 4 q
        const uint32_t nn = n0 + cg * 16, kk = k0 + q * 4;
        uint32_t v[4][4] = {};   // [k][four channels]
        if (kk < k && nn < n) {   // k is a multiple of 4: all four rows exist
            const uint8_t* src = in + (size_t)kk * in_pitch + nn;
            if (nn + 16 <= n) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 x = __ldcs(reinterpret_cast<const uint4*>(src + (size_t)i * in_pitch));
                    v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int b = 0; b < 16; ++b)
                        if (nn + b < n) v[i][b >> 2] |= (uint32_t)src[(size_t)i * in_pitch + b] << (8 * (b & 3));
            }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {   // packed word of a channel: bytes of k [0,2,1,3]
            const uint32_t lo02 = prmt(v[0][b], v[2][b], 0x5140u), hi02 = prmt(v[0][b], v[2][b], 0x7362u);   // {k0,k2} of channels 0,1 / 2,3
            const uint32_t lo13 = prmt(v[1][b], v[3][b], 0x5140u), hi13 = prmt(v[1][b], v[3][b], 0x7362u);
            const uint32_t w[4] = {prmt(lo02, lo13, 0x5410u), prmt(lo02, lo13, 0x7632u), prmt(hi02, hi13, 0x5410u), prmt(hi02, hi13, 0x7632u)};
#pragma unroll
            for (int e = 0; e < 4; ++e) tile[cg * 16 + b * 4 + e][q ^ (cg * 4)] = w[e];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t c = i * 32 + (threadIdx.x >> 3), piece = threadIdx.x & 7;
        const uint32_t nn = n0 + c, kk = k0 + piece * 16;
        if (nn >= n || kk >= k) continue;
        const uint4 x = *reinterpret_cast<const uint4*>(&tile[c][(piece ^ ((c >> 4) & 7u)) * 4]);
        uint8_t* dst = out + (size_t)nn * out_pitch + kk;
        if (kk + 16 <= k) {
            *reinterpret_cast<uint4*>(dst) = x;
        } else {   // the last words of a row
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (kk + e * 4 < k) *reinterpret_cast<uint32_t*>(dst + e * 4) = w[e];
        }
    }
}

// rows of two equally shaped byte matrices interleaved: dst row 2i = g row i, dst row 2i+1 = u row i
__global__ void __launch_bounds__(256) interleave_rows_kernel(const uint8_t* __restrict__ g, const uint8_t* __restrict__ u, uint8_t* __restrict__ dst,
                                                              uint32_t rows, uint32_t row_bytes) {
    const size_t total = (size_t)rows * row_bytes;
    for (size_t id = blockIdx.x * (size_t)blockDim.x + threadIdx.x; id < total; id += (size_t)gridDim.x * blockDim.x) {
        const size_t r = id / row_bytes, c = id % row_bytes;
        dst[(2 * r) * row_bytes + c] = g[id];
        dst[(2 * r + 1) * row_bytes + c] = u[id];
    }
}

}  // namespace
}  // namespace afb

using namespace afb;

extern "C" int afb_prepack(const afb_gemm_args* a, void* out_b, uint32_t out_ldb, void* stream) {
    if (!a || !a->ptr_b || !out_b || a->n == 0 || a->k == 0) return AFB_ERR_BAD_ARG;
    if (a->b_bits != 8 && a->b_bits != 4) return AFB_ERR_BAD_ARG;
    if (a->b_layout != AFB_LAYOUT_ROW && a->b_layout != AFB_LAYOUT_COL) return AFB_ERR_BAD_ARG;   // already packed input is refused
    if (a->b_bits == 4 && a->b_layout != AFB_LAYOUT_COL) return AFB_ERR_UNSUPPORTED;
    if (out_ldb < a->k || (a->b_layout == AFB_LAYOUT_COL ? a->ldb < a->k : a->ldb < a->n)) return AFB_ERR_BAD_ARG;
    const uint32_t per_word = a->b_bits == 8 ? 4u : 8u;
    if (a->k % per_word) return AFB_ERR_UNSUPPORTED;                      // whole 32-bit words of weights per row
    const uint32_t out_pitch = out_ldb * a->b_bits / 8, row_bytes = a->k * a->b_bits / 8;
    if (out_pitch % 4 || (uintptr_t)out_b % 4) return AFB_ERR_BAD_ARG;
    if ((const void*)a->ptr_b == (const void*)out_b && a->b_layout == AFB_LAYOUT_ROW) return AFB_ERR_BAD_ARG;   // the transpose cannot run in place
    if (!current_ctx()) return AFB_ERR_NOT_INIT;
    cudaStream_t s = (cudaStream_t)stream;
    if (a->b_layout == AFB_LAYOUT_COL) {
        const uint32_t in_pitch = a->ldb * a->b_bits / 8;
        if (in_pitch % 4 || (uintptr_t)a->ptr_b % 4) return AFB_ERR_BAD_ARG;
        prepack_col_kernel<<<592, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(a->ptr_b), reinterpret_cast<uint8_t*>(out_b), a->n, row_bytes,
                                               in_pitch, out_pitch, a->b_bits);
    } else {
        dim3 grid((a->n + 31) / 32, (a->k + 31) / 32);
        if (grid.y > 65535) return AFB_ERR_UNSUPPORTED;
        // rows of whole 16-byte pieces on both sides; other pitches and pointers take the byte-wise kernel (five times slower)
        const bool wide = a->ldb % 16 == 0 && out_pitch % 16 == 0 && (uintptr_t)a->ptr_b % 16 == 0 && (uintptr_t)out_b % 16 == 0;
        if (wide) prepack_row_wide_kernel<<<dim3((a->n + 127) / 128, (a->k + 127) / 128), 256, 0, s>>>(reinterpret_cast<const uint8_t*>(a->ptr_b), reinterpret_cast<uint8_t*>(out_b), a->n, a->k, a->ldb, out_pitch);
        else
        prepack_row_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(a->ptr_b), reinterpret_cast<uint8_t*>(out_b), a->n, a->k, a->ldb, out_pitch);
    }
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AFB_OK : cuda_fail(e);
}

extern "C" int afb_prepack_gated(const afb_gemm_args* gate, const void* b_up, const void* scale_up, const void* zero_up, void* out_b,
                                 uint32_t out_ldb, void* out_scale, void* out_zero, void* stream) {
    if (!gate || !gate->ptr_b || !gate->ptr_scale || !b_up || !scale_up || !out_b || !out_scale || gate->n == 0 || gate->k == 0) return AFB_ERR_BAD_ARG;
    if (gate->b_bits != 8 && gate->b_bits != 4) return AFB_ERR_BAD_ARG;
    if (gate->b_layout != AFB_LAYOUT_COL) return AFB_ERR_UNSUPPORTED;
    if ((gate->ptr_zero != nullptr) != (zero_up != nullptr) || (gate->ptr_zero && !out_zero)) return AFB_ERR_BAD_ARG;
    if (gate->group_size && gate->k % gate->group_size) return AFB_ERR_BAD_ARG;
    const uint32_t per_word = gate->b_bits == 8 ? 4u : 8u;
    if (gate->k % per_word || out_ldb < gate->k || gate->ldb < gate->k) return AFB_ERR_BAD_ARG;
    const uint32_t out_pitch = out_ldb * gate->b_bits / 8, in_pitch = gate->ldb * gate->b_bits / 8, row_bytes = gate->k * gate->b_bits / 8;
    if (out_pitch % 4 || in_pitch % 4 || (uintptr_t)out_b % 4 || (uintptr_t)gate->ptr_b % 4 || (uintptr_t)b_up % 4) return AFB_ERR_BAD_ARG;
    if (!current_ctx()) return AFB_ERR_NOT_INIT;
    cudaStream_t s = (cudaStream_t)stream;
    uint8_t* ob = reinterpret_cast<uint8_t*>(out_b);
    // the packing kernel with a doubled output pitch writes every other row: gate rows at 2i, up rows at 2i + 1
    prepack_col_kernel<<<592, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(gate->ptr_b), ob, gate->n, row_bytes, in_pitch, 2 * out_pitch, gate->b_bits);
    prepack_col_kernel<<<592, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(b_up), ob + out_pitch, gate->n, row_bytes, in_pitch, 2 * out_pitch, gate->b_bits);
    const uint32_t groups = gate->group_size ? gate->k / gate->group_size : 1;
    const uint32_t sbytes = groups * (gate->scale_dtype == AFB_SCALE_BF16 ? 2u : 4u);
    interleave_rows_kernel<<<148, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(gate->ptr_scale), reinterpret_cast<const uint8_t*>(scale_up),
                                               reinterpret_cast<uint8_t*>(out_scale), gate->n, sbytes);
    unsigned launches = 3;
    if (gate->ptr_zero) {
        interleave_rows_kernel<<<148, 256, 0, s>>>(reinterpret_cast<const uint8_t*>(gate->ptr_zero), reinterpret_cast<const uint8_t*>(zero_up),
                                                   reinterpret_cast<uint8_t*>(out_zero), gate->n, groups);
        ++launches;
    }
    count_launch(launches);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AFB_OK : cuda_fail(e);
}
