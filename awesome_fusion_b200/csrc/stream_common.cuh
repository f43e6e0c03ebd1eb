// Shared by the streaming form (stream.cu) and the pair form (pair.cu): sizes, bounded waits, ring positions, tensor maps.
#pragma once
#include "afb_internal.h"
#include "ptx_sm100.cuh"
#include "stream_deal.h"

namespace afb {

namespace {

constexpr int kCh = 128;              // output channels of a CTA's tile = TMEM lanes
constexpr int kSlab = 64;             // k of one activation box (128 bytes, one swizzle span)
constexpr int kRawBytes = kCh * 128;  // one raw block of weights: 128 channels x 128 bytes
constexpr int kGroups = 4;            // converter groups

__device__ __forceinline__ void report_timeout(int32_t* status, int where, int a, int b) {
    if (atomicCAS(status, 0, AFB_ERR_TIMEOUT) == 0) { status[1] = where; status[2] = a; status[3] = b; }
}
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    unsigned long long t0 = 0;
    for (uint32_t tries = 0; !ptx::mbar_try_wait(bar, parity);) {
        if ((++tries & 0x3fu) == 0) {   // the clock is read only here: reading %globaltimer takes longer than most waits
            if (*abort_flag) return false;
            const unsigned long long t = ptx::globaltimer();
            if (t0 == 0) t0 = t;
            else if (t - t0 > ptx::kWaitLimitNs) return false;
        }
    }
    return true;
}
// The same for a converged warp: every lane gets the same answer, so that none is missing from the warp-wide instructions that follow.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag) {
    return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag));
}
// A position in a ring of runtime length.
struct Ring {
    uint32_t i, phase;
    __device__ __forceinline__ void step(uint32_t by, uint32_t len) { i += by; if (i >= len) { i -= len; phase ^= 1u; } }   // by <= len
    __device__ __forceinline__ void set(uint32_t count, uint32_t len) { const uint32_t w = count / len; i = count - w * len; phase = w & 1u; }
};

inline int tmap_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
            uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swz) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return AFB_ERR_CUDA;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_stride_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? AFB_OK : AFB_ERR_CUDA;
}

}  // namespace

}  // namespace afb
