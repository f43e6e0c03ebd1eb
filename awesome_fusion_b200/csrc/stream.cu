// Streaming form of the decode and prefill variants (B in [N,K] layout): weights flow HBM -> shared memory -> registers -> tensor
// memory -> tcgen05.mma in one pipeline that is deep enough to run at memory speed when M is small and at tensor-core speed when
// M is large (reference counterpart of the whole kernel: bf16gemm_kernel_gfx90a.s:184-636).
//
// D[n, m] = sum_k W[n,k] * A[m,k]: a tile has 128 output channels (the TMEM lanes) and `rows` activation rows (a multiple of 16,
// fitted to M).  One CTA per SM:
//
//   warp 0                TMA: raw weight blocks, 128 channels x 128 bytes (128 k of int8, 256 k of int4), 128-byte swizzle
//   warp 1                TMA: activation slabs [rows x 64] bf16, 128-byte swizzle
//   warp 2 (and 3)        tcgen05.mma 128 x rows x 16, weights from TMEM, activations from shared memory; up to 16 rows two warps, one for
//                         each part of a step (warps 0 to 3 run as whole warps and elect a lane for the asynchronous instructions)
//   warps 4-7             epilogue, one lane quarter each: accumulator -> scale -> bf16 -> C, or fp32 partial sums -> workspace
//   warps 8-23            converters: four groups of four warps (one per lane quarter); group g takes every fourth part of k,
//                         64 or 128 wide, so that four parts are being unpacked at any time.  A warp's chain wait -> load ->
//                         unpack -> tcgen05.st -> arrive takes about 800 cycles; what bounds a form in which all converters
//                         share ONE step is that chain, whatever M is.
//
// k goes by in parts (one converter group's work: 64 or 128 k) and steps (one hand-off to and from the issuing warp: one part, or
// two where few rows make the hand-off the larger cost).  Weights and activations have rings of their own.
// Work is dealt in units of one raw block: first every CTA takes the same number of units of the tiles that do not fill whole
// waves (contiguous, so at most two of its tiles are shared with neighbours), then whole tiles, one wave after the other.
// A shared tile is finished by the last CTA to arrive, which adds the fp32 partial sums in CTA order (= ascending K): the bits do
// not depend on who that is, and no CTA waits for another.  Up to 16 rows the group scales multiply the fp32 sum of each group, in the
// epilogue warps, while the next groups are being computed (per-channel sums are handed over every 1024 k); above that they are folded
// into the bf16 weights.
//
// What bounds it: for few rows int8 the weight stream (28672 x 8192, 16 rows: 44.7 us = 5.3 TB/s of weights, 63.8 with decode.cu), int4
// the converters, which take 2400 cycles for a part of 128 k next to each other, and the issuing warps (5 rows with zero-points, caches cold: 53.6 us
// with one issuing warp, 49.2 with two; 16 rows int8 47.0 and 45.9); for 65 to 128 rows the activations through L2 (28672 x 8192 int4
// group-128, 128 rows: 66 us, 82 with prefill.cu); for many rows the pace of the issuing warp next to the unpack.
#include <cstdlib>
#include "afb_internal.h"
#include "dequant.cuh"
#include "ptx_sm100.cuh"
#include "stream_common.cuh"

namespace afb {

namespace {

constexpr int kFirstEpi = 4, kFirstConv = 8;
constexpr int kThreads = 32 * (kFirstConv + 4 * kGroups);
constexpr int kMaxRaw = 12, kMaxSlots = 8, kMaxAcc = 8;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kSet = 4;            // kSums, kParts: sums handed to the epilogue at a time (5 x 28672 x 8192 int4: 51.5 us with 2, 49.7 with 4)
// kParts: k that one accumulator adds up before the sum goes on in fp32 registers.  The tensor cores cut off what an addition shifts out,
// so a sum over all of K drifts: of 16 x 28672 x 8192 int8 results 15 in 10000 were not the correctly rounded ones (8 rows: 14), with
// decode.cu, whose warps and CTAs each add a stretch of K, 10 (5), with sums over 1024 k 3 (3).
constexpr uint32_t kPartSum = 1024;
constexpr int kBars = 2 * (kMaxRaw + 2 * kMaxSlots + kMaxAcc) + kMaxSlots + 3;
constexpr int kOffMisc = kBars * 8, kOffOut = 1024;
constexpr int kOutBytes = 16 * 32 * 2;                    // one block of the result: 16 rows x 32 channels
constexpr int kOffRaw = kOffOut + 4 * 2 * kOutBytes;      // two blocks per epilogue warp
constexpr int kRingBudget = 232448 - 1024 - kOffRaw;      // bytes for the two rings (1 KiB for the alignment of the base)
static_assert(kOffMisc + 32 <= kOffOut && kOffRaw % 1024 == 0, "shared memory layout");

enum Mode { kChannel = 0,   // per-channel scale on the finished sum
            kFold = 1,      // group scale folded into the bf16 weight (more than 16 activation rows)
            kSums = 2,      // group scale on the fp32 sum of each group (up to 16 rows)
            kParts = 3 };   // as kChannel, for up to 16 rows: the tensor cores' sums over kPartSum of k are added in fp32
__host__ __device__ constexpr bool channel_scaled(int mode) { return mode == kChannel || mode == kParts; }
__host__ __device__ constexpr bool summed(int mode) { return mode == kSums || mode == kParts; }

struct StreamParams {
    uint16_t* c;
    const void* scale;
    const uint8_t* zero;
    uint32_t m, n, k, ldc;
    uint32_t enc, scale_dtype, packed;
    uint32_t group_shift;     // log2(group / k of a part)
    uint32_t flush;           // kSums, kParts: parts per sum
    uint32_t acc_cols;        // TMEM columns handed to the epilogue at a time (kSums, kParts: kSet sums)
    uint32_t rows, m_tiles, n_tiles, group_m;
    uint32_t parts;           // parts along K
    StreamDeal deal;          // who does what, in units of one raw block
    uint32_t raw_stages, slots, accs;
    uint32_t slot_first;      // converters wait for their slot before they wait for their raw block
    uint32_t c_tma, c_vec;    // tile stores; 8-byte stores of finished shared tiles
    uint32_t finish_late;     // shared tiles are finished by all warps at the CTA's end, not by the epilogue warps on the way
    float* ws;                // [2 * CTA + (not the CTA's first shared tile)][row][channel]
    uint32_t* counters;       // one per shared tile, zero on entry and on exit
    int32_t* status;
};

// Groups of group_m row tiles; inside a group the channel tiles advance, row tile fastest.
__device__ __forceinline__ void tile_origin(const StreamParams& p, uint32_t t, uint32_t& m0, uint32_t& n0) {
    const uint32_t per_group = p.group_m * p.n_tiles;
    const uint32_t g = t / per_group, r = t - g * per_group;
    const uint32_t gsz = min(p.group_m, p.m_tiles - g * p.group_m);
    const uint32_t nt = r / gsz;
    n0 = nt * kCh;
    m0 = (g * p.group_m + (r - nt * gsz)) * p.rows;
}

template <int BITS, int MODE, int KS, int PAIR>
__global__ void __launch_bounds__(kThreads, 1)
stream_kernel(const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_w,
              const __grid_constant__ CUtensorMap tmap_c, const StreamParams p) {
    constexpr uint32_t SPB = (BITS == 8 ? 128 : 256) / KS;   // parts per raw block
    constexpr uint32_t kPartCols = KS / 2, kSlotCols = PAIR * kPartCols;   // TMEM columns of the converted weights of a part, of a step
    extern __shared__ uint8_t smem_raw_base[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw_base) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw_base + (smem_base - ptx::smem_u32(smem_raw_base));
    auto bar = [&](uint32_t i) { return smem_base + 8u * i; };
    auto raw_full = [&](uint32_t s) { return bar(s); };
    auto raw_empty = [&](uint32_t s) { return bar(kMaxRaw + s); };
    // Up to 16 rows a step's two parts are issued by two warps, each into sums of its own (`h`: which part): one warp, next to busy
    // converters on its scheduler, needs 46 cycles per tcgen05.mma and 450 besides per step, the tensor cores 9 for 16 rows (5 x 28672 x
    // 8192 int4 group-128: 1500 cycles per step of 256 k with one).
    // A free slot then tells a converter group about one part of a step only, so the raw block that had its place in the raw ring before
    // must have been this group's own: the ring is a multiple of the groups' turn, and a step takes the places of two int8 blocks even if
    // it lacks the second (kPadded).
    constexpr bool kDual = summed(MODE) && PAIR == 2, kPadded = kDual && SPB == 1;
    auto step_full = [&](uint32_t s, uint32_t h = 0) { return bar(2 * kMaxRaw + h * kMaxSlots + s); };          // converted weights in TMEM, activations in shared memory
    auto step_empty = [&](uint32_t s, uint32_t h = 0) { return bar(2 * kMaxRaw + (2 + h) * kMaxSlots + s); };   // the MMAs of the step are done with both
    // The arrival of a step's activations.  Where a step is two parts (few rows) a converter warp waits for it before it reports its part,
    // so that the issuing warp, whose own instructions set the pace there, has one thing to wait for that is usually complete (28672 x
    // 8192, 1 row: 43.3 -> 41.9 us int8); with more rows it counts into step_full (39 against 38 us on 333 x 11008 x 4096 otherwise).
    constexpr bool kActApart = PAIR == 2;
    auto act_full = [&](uint32_t s) { return kActApart ? bar(2 * (kMaxRaw + 2 * kMaxSlots + kMaxAcc) + s) : step_full(s); };
    auto acc_full = [&](uint32_t s) { return bar(2 * (kMaxRaw + 2 * kMaxSlots) + s); };
    auto acc_empty = [&](uint32_t s) { return bar(2 * (kMaxRaw + 2 * kMaxSlots) + kMaxAcc + s); };
    // a shared tile: every epilogue warp has published its part; the count has been taken.  The end: the epilogue is through
    const uint32_t bar_stored = bar(kBars - 3), bar_verdict = bar(kBars - 2), bar_finish = bar(kBars - 1);
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_gen + kOffMisc);   // TMEM base, abort flag, "arrived last", tiles to finish, their number
    volatile uint32_t* abort_flag = misc + 1;
    const uint32_t slab_bytes = p.rows * 128u, part_bytes = slab_bytes * (KS / kSlab), act_bytes = PAIR * part_bytes, off_act = kOffRaw + p.raw_stages * kRawBytes;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // see decode.cu: no-op without AFB_FLAG_PDL

    // Warp 0 needs only its own barriers: it starts the weight stream while the others are still setting up.
    if (warp == 0) {
        if (lane == 0) {
            for (uint32_t s = 0; s < p.raw_stages; ++s) { ptx::mbar_init(raw_full(s), 1); ptx::mbar_init(raw_empty(s), 4 * SPB); }
            *abort_flag = 0;
            ptx::fence_mbar_init();
        }
        __syncwarp();
        asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
    } else {
        if (warp == 1 && lane == 0) {
            for (uint32_t s = 0; s < p.slots; ++s) { ptx::mbar_init(step_full(s), kDual ? 4 : kActApart ? 4 * PAIR : 4 * PAIR + 1); ptx::mbar_init(step_empty(s), 1); if (kActApart) ptx::mbar_init(act_full(s), 1); }
            for (uint32_t s = 0; kDual && s < p.slots; ++s) { ptx::mbar_init(step_full(s, 1), 4); ptx::mbar_init(step_empty(s, 1), 1); }
            for (uint32_t s = 0; s < p.accs; ++s) { ptx::mbar_init(acc_full(s), kDual ? 2 : 1); ptx::mbar_init(acc_empty(s), 4); }
            ptx::mbar_init(bar_stored, 4);
            ptx::mbar_init(bar_verdict, 1);
            ptx::mbar_init(bar_finish, 4);
            ptx::fence_mbar_init();
            ptx::prefetch_tmap(&tmap_act);
            if (p.c_tma) ptx::prefetch_tmap(&tmap_c);
        }
        if (warp == 2) {
            ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(misc)), kTmemCols);
            ptx::tmem_relinquish();
        }
        __syncwarp();
        ptx::tc_fence_before_sync();
        asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
        ptx::tc_fence_after_sync();
    }
    constexpr uint32_t tmem_base = 0;   // all 512 columns are this CTA's: the allocation starts at column 0
    const uint32_t slot_base = tmem_base + kTmemCols - p.slots * kSlotCols;   // accumulators from column 0, slots at the end

    auto give_up = [&](int where, uint32_t a, uint32_t b) {
        if (!*abort_flag) { report_timeout(p.status, where, (int)a, (int)b); *abort_flag = 1; }
    };
    Walk walk;
    walk.start(p.deal, blockIdx.x);   // every role walks the same list of pieces
    Piece x;
    auto parts_of = [&](const Piece& q) { return min(q.kb1 * SPB, p.parts) - q.kb0 * SPB; };

    auto channel_scale = [&](uint32_t nn) {
        if (!channel_scaled(MODE) || nn >= p.n) return 0.f;
        return p.scale_dtype == AFB_SCALE_BF16 ? __uint_as_float((uint32_t)reinterpret_cast<const uint16_t*>(p.scale)[nn] << 16)
                                               : reinterpret_cast<const float*>(p.scale)[nn];
    };
    auto finished = [&](float sum, float scale) {
        return channel_scaled(MODE) ? unscaled(sum, scale) : sum * (MODE == kSums ? kUnpackInverse : kGroupInverse);
    };

    // Adds the partial sums of shared tile t in CTA order, scales, rounds and stores it; `tid` of `threads` threads, four channels of
    // one row at a time, up to eight 16-byte loads in flight per thread.
    auto finish_tile = [&](uint32_t t, uint32_t tid, uint32_t threads) {
        uint32_t m0, n0;
        tile_origin(p, t, m0, n0);
        const uint32_t first = p.deal.first_cta(t), last = p.deal.last_cta(t);
        const uint32_t valid = min(p.rows, p.m - m0), vecs = valid * (kCh / 4);
        const uint32_t nn = n0 + (tid & 31u) * 4;   // threads is a multiple of 32: the same four channels in every turn
        float sc[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
            sc[e] = channel_scale(nn + e);
        const uint32_t first_slot = p.deal.slot(first, t);   // the others' runs begin in this tile: slot 2c
        const size_t stride = (size_t)p.rows * kCh;
        for (uint32_t v = tid; v < vecs; v += 2 * threads) {
            float4 sum[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
            for (uint32_t c = first; c <= last; c += 4) {
                float4 y[2][4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        y[h][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (c + i <= last && v + h * threads < vecs)
                            y[h][i] = __ldcg(reinterpret_cast<const float4*>(p.ws + (size_t)(c + i == first ? first_slot : 2 * (c + i)) * stride) + v + h * threads);
                    }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) { sum[h].x += y[h][i].x; sum[h].y += y[h][i].y; sum[h].z += y[h][i].z; sum[h].w += y[h][i].w; }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (v + h * threads >= vecs) break;
                const __nv_bfloat162 lo = __floats2bfloat162_rn(finished(sum[h].x, sc[0]), finished(sum[h].y, sc[1])),
                                     hi = __floats2bfloat162_rn(finished(sum[h].z, sc[2]), finished(sum[h].w, sc[3]));
                uint16_t* dst = p.c + (size_t)(m0 + (v + h * threads) / (kCh / 4)) * p.ldc + nn;
                if (p.c_vec && nn + 4 <= p.n) {
                    *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                } else {
                    const uint16_t o[4] = {__bfloat16_as_ushort(lo.x), __bfloat16_as_ushort(lo.y), __bfloat16_as_ushort(hi.x), __bfloat16_as_ushort(hi.y)};
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (nn + e < p.n) dst[e] = o[e];
                }
            }
        }
    };

    // Warps 0 to 2 run their loops as whole warps and elect a lane for the asynchronous instructions only: the operands are then
    // warp-uniform values.  (With the loops under `if (lane == 0)` the issuing warp needed 900 cycles per 64-wide step, whatever M.)
    if (warp == 0) {
        // ======================= TMA: raw weights =======================
        Ring r{0, 0};
        uint32_t issued = 0, parity = 0;
        bool ok = true;
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            uint32_t m0, n0;
            tile_origin(p, x.t, m0, n0);
            for (uint32_t kb = x.kb0; kb < x.kb1; ++kb) {
                if (!warp_wait(raw_empty(r.i), r.phase ^ 1u, abort_flag)) { give_up(31, x.t, kb); ok = false; break; }
                if (ptx::elect_one()) {
                    ptx::mbar_arrive_expect_tx(raw_full(r.i), kRawBytes);
                    ptx::tma_load_2d(smem_base + kOffRaw + r.i * kRawBytes, &tmap_w, (int)(kb * 128u), (int)n0, raw_full(r.i));
                }
                issued |= 1u << r.i; parity = (parity & ~(1u << r.i)) | (r.phase << r.i);
                r.step(1, p.raw_stages);
            }
            if (kPadded && ok && ((x.kb1 - x.kb0) & 1u)) {
                if (!warp_wait(raw_empty(r.i), r.phase ^ 1u, abort_flag)) { give_up(31, x.t, x.kb1); break; }
                if (ptx::elect_one()) ptx::mbar_arrive(raw_full(r.i));
                issued |= 1u << r.i; parity = (parity & ~(1u << r.i)) | (r.phase << r.i);
                r.step(1, p.raw_stages);
            }
        }
        for (uint32_t s = 0; s < p.raw_stages; ++s)   // never leave with a bulk copy still writing this CTA's shared memory
            if (issued & (1u << s)) ptx::mbar_wait(raw_full(s), (parity >> s) & 1u);
    } else if (warp == 1) {
        // ======================= TMA: activations =======================
        asm volatile("griddepcontrol.wait;" ::: "memory");   // everything before this line reads weights only
        Ring r{0, 0};
        uint32_t issued = 0, parity = 0;
        bool ok = true;
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            uint32_t m0, n0;
            tile_origin(p, x.t, m0, n0);
            const uint32_t k0 = x.kb0 * SPB, ns = parts_of(x);
            for (uint32_t l = 0; l < ns; l += PAIR) {
                if (!warp_wait(step_empty(r.i), r.phase ^ 1u, abort_flag) || (kDual && !warp_wait(step_empty(r.i, 1), r.phase ^ 1u, abort_flag))) { give_up(32, x.t, l); ok = false; break; }
                if (ptx::elect_one()) {
                    ptx::mbar_arrive_expect_tx(act_full(r.i), l + PAIR <= ns ? act_bytes : part_bytes);
#pragma unroll
                    for (int h = 0; h < PAIR * KS / kSlab; ++h)
                        if (PAIR == 1 || h < KS / kSlab || l + 1 < ns)
                            ptx::tma_load_2d(smem_base + off_act + r.i * act_bytes + h * slab_bytes, &tmap_act, (int)((k0 + l) * KS + h * kSlab), (int)m0, act_full(r.i));
                }
                issued |= 1u << r.i; parity = (parity & ~(1u << r.i)) | (r.phase << r.i);
                r.step(1, p.slots);
            }
        }
        for (uint32_t s = 0; s < p.slots; ++s)
            if (issued & (1u << s)) ptx::mbar_wait(act_full(s), (parity >> s) & 1u);   // after an abort the converters' part may be missing: then the limit of the wait, far above the time of a copy
    } else if (kDual && warp < kFirstEpi) {
        // ======================= MMA issuers, one for each part of a step =======================
        const uint32_t h = (uint32_t)warp - 2, idesc = ptx::umma_idesc_bf16_f32(kCh, p.rows);
        const uint64_t desc0 = ptx::umma_desc_kmajor_sw128(smem_base + off_act) + h * (part_bytes >> 4);
        const uint32_t slab_d = slab_bytes >> 4, act_d = act_bytes >> 4;   // in units of the descriptor's address field
        Ring rs{0, 0}, rc{0, 0};
        bool ok = true, ready = false;
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            const uint32_t ns = parts_of(x);
            uint32_t in_sum = 0, sum = h;   // parts in this warp's current sum; which of the accumulator's sums (this warp's are h and h + 2)
            for (uint32_t l = 0; l < ns; l += 2) {
                if (in_sum == 0 && sum == h && !warp_wait(acc_empty(rc.i), rc.phase ^ 1u, abort_flag)) { give_up(33, x.t, l); ok = false; break; }
                if (!__all_sync(0xffffffffu, ready) && !warp_wait(step_full(rs.i, h), rs.phase, abort_flag)) { give_up(34, x.t, l); ok = false; break; }
                ptx::tc_fence_after_sync();
                const uint64_t db = desc0 + rs.i * act_d;
                const uint32_t ta = slot_base + rs.i * kSlotCols + h * kPartCols, td = tmem_base + rc.i * p.acc_cols + sum * 16, done = step_empty(rs.i, h), acc_done = acc_full(rc.i);
                rs.step(1, p.slots);
                ready = ptx::mbar_test_wait(step_full(rs.i, h), rs.phase);   // of the next step: the answer is back when this one has been issued
                const bool there = l + h < ns, first = in_sum == 0;   // the last step of a piece may lack its second part
                if (++in_sum == p.flush) { in_sum = 0; sum += 2; }
                const bool last = l + 2 >= ns || sum >= kSet;
                if (ptx::elect_one()) {
                    if (there) {
#pragma unroll
                        for (int j = 0; j < KS / 16; ++j)
                            ptx::umma_bf16_ts(td, ta + 8 * j, db + (uint32_t)(j / 4) * slab_d + 2u * (j % 4), idesc, !first || j > 0 ? 1u : 0u);
                    }
                    ptx::umma_commit(done);
                    if (last) ptx::umma_commit(acc_done);
                }
                if (last) { rc.step(1, p.accs); in_sum = 0; sum = h; }
            }
        }
    } else if (warp == 2) {
        // ======================= MMA issuer =======================
        const uint32_t idesc = ptx::umma_idesc_bf16_f32(kCh, p.rows);
        const uint64_t desc0 = ptx::umma_desc_kmajor_sw128(smem_base + off_act);
        const uint32_t slab_d = slab_bytes >> 4, act_d = act_bytes >> 4;   // in units of the descriptor's address field
        Ring rs{0, 0}, rc{0, 0};
        bool ok = true, ready = false;
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            const uint32_t ns = parts_of(x);
            uint32_t in_sum = 0, sum = 0;   // parts in the current sum; sums in the current accumulator (kSums, kParts)
            for (uint32_t l = 0; l < ns; l += PAIR) {
                if (in_sum == 0 && sum == 0 && !warp_wait(acc_empty(rc.i), rc.phase ^ 1u, abort_flag)) { give_up(33, x.t, l); ok = false; break; }
                if (!__all_sync(0xffffffffu, ready) && !warp_wait(step_full(rs.i), rs.phase, abort_flag)) { give_up(34, x.t, l); ok = false; break; }
                ptx::tc_fence_after_sync();
                const uint64_t db = desc0 + rs.i * act_d;
                const uint32_t ta = slot_base + rs.i * kSlotCols, td = tmem_base + rc.i * p.acc_cols, done = step_empty(rs.i), acc_done = acc_full(rc.i);
                rs.step(1, p.slots);
                ready = ptx::mbar_test_wait(step_full(rs.i), rs.phase);   // of the next step: the answer is back when this one has been issued
                bool last = false;
#pragma unroll
                for (int h = 0; h < PAIR; ++h) {
                    if (PAIR > 1 && h > 0 && l + h >= ns) break;
                    if (ptx::elect_one()) {
#pragma unroll
                        for (int j = 0; j < KS / 16; ++j)
                            ptx::umma_bf16_ts(td + sum * 16, ta + h * kPartCols + 8 * j, db + (uint32_t)(h * (KS / kSlab) + j / 4) * slab_d + 2u * (j % 4), idesc, (in_sum | (uint32_t)j) ? 1u : 0u);
                    }
                    ++in_sum;
                    if (summed(MODE) && in_sum == p.flush) { in_sum = 0; ++sum; }
                    last = l + h + 1 == ns || (summed(MODE) && sum == kSet);
                }
                if (ptx::elect_one()) {
                    ptx::umma_commit(done);
                    if (last) ptx::umma_commit(acc_done);
                }
                if (last) { rc.step(1, p.accs); in_sum = sum = 0; }
            }
        }
    } else if (warp >= kFirstConv) {
        // ======================= converters =======================
        const uint32_t g = (uint32_t)(warp - kFirstConv) >> 2, quarter = (uint32_t)warp & 3u;
        const uint32_t ch = quarter * 32 + lane;
        const uint32_t flip = BITS == 8 ? flip8(p.enc) : flip4(p.enc);
        const uint32_t sel0 = p.packed ? kSel8Strided02 : kSel8Natural01, sel1 = p.packed ? kSel8Strided13 : kSel8Natural23;
        const Nibbles nib = nibbles(p.packed != 0);
        const bool has_zero = p.zero != nullptr;
        const uint32_t groups_per_row = channel_scaled(MODE) ? 0 : (p.parts >> p.group_shift);
        auto zero_of = [&](uint32_t zb) { return !has_zero ? 0 : (BITS == 8 ? decode_zero8(zb, p.enc) : decode_zero4(zb, p.enc)); };
        GroupUnpack up;
        up.mul0 = BITS == 8 ? kMulByte : nib.mul[0]; up.mul1 = nib.mul[1]; up.add = unpack_add(BITS, 0); up.scale = 0;
        uint32_t steps_before = 0, blocks_before = 0;   // of the pieces walked so far (a step is PAIR parts, the last of a piece may lack one)
        bool ok = true;
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            uint32_t m0, n0;
            tile_origin(p, x.t, m0, n0);
            const uint32_t nn = n0 + ch, ns = parts_of(x), k0 = x.kb0 * SPB;
            const size_t g0 = (size_t)nn * groups_per_row;
            uint32_t sc = 0, zb = 0, sc_nxt = 0, zb_nxt = 0;
            auto load_group = [&](uint32_t l, uint32_t& s, uint32_t& z) {
                if (channel_scaled(MODE) || nn >= p.n || l >= ns) return;
                const size_t i = g0 + ((k0 + l) >> p.group_shift);
                if (MODE == kFold) s = reinterpret_cast<const uint16_t*>(p.scale)[i];
                if (has_zero) z = p.zero[i];
            };
            if (channel_scaled(MODE) && has_zero) up.add = unpack_add(BITS, zero_of(nn < p.n ? p.zero[nn] : 0u));
            uint32_t l = (g - steps_before * PAIR) & (kGroups - 1);
            Ring rr, rs;
            rr.set((kPadded ? 2 * steps_before : blocks_before) + l / SPB, p.raw_stages);
            rs.set(steps_before + l / PAIR, p.slots);
            load_group(l, sc_nxt, zb_nxt);
            const uint32_t nv = (ns + PAIR - 1) / PAIR * PAIR;
            for (; l < nv; l += kGroups) {
                if (PAIR > 1 && l == ns) {
                    // The part that the last step of this piece lacks: waited for and reported like the others.  A group that passed
                    // over it would next look at a slot two uses later, where the parity of the barrier no longer tells it anything.
                    if (!warp_wait(step_empty(rs.i, kDual), rs.phase ^ 1u, abort_flag)) { give_up(36, x.t, l); ok = false; break; }
                    if (kPadded && !warp_wait(raw_full(rr.i), rr.phase, abort_flag)) { give_up(35, x.t, l); ok = false; break; }
                    // (with two issuing warps also for its activations: or their loader could find this barrier a phase ahead)
                    if (kDual && quarter == 0 && !warp_wait(act_full(rs.i), rs.phase, abort_flag)) { give_up(39, x.t, l); ok = false; break; }
                    if (lane == 0) ptx::mbar_arrive(step_full(rs.i, kDual));
                    if (kPadded && lane == 0) ptx::mbar_arrive(raw_empty(rr.i));
                    continue;
                }
                const uint32_t which = kDual ? g & 1u : 0u;   // a group's parts are all first or all second ones
                const uint32_t sub = l % SPB, left = ns - (l - sub);   // `left`: parts of this block and all after it
                if (!channel_scaled(MODE)) { sc = sc_nxt; zb = zb_nxt; load_group(l + kGroups, sc_nxt, zb_nxt); }
                if (p.slot_first && !warp_wait(step_empty(rs.i, which), rs.phase ^ 1u, abort_flag)) { give_up(36, x.t, l); ok = false; break; }
                if (!warp_wait(raw_full(rr.i), rr.phase, abort_flag)) { give_up(35, x.t, l); ok = false; break; }
                const uint8_t* raw = smem_gen + kOffRaw + rr.i * kRawBytes + ch * 128;
                constexpr int kWords = BITS == 8 ? 16 : 8;   // of 64 weights
                bool folded = true;
                if (MODE == kFold) {
                    folded = __all_sync(0xffffffffu, group_folds((uint16_t)sc, has_zero));
                    up = group_unpack(BITS, (uint16_t)sc, zero_of(zb), folded, nib);
                } else if (MODE == kSums && has_zero) {
                    up.add = unpack_add(BITS, zero_of(zb));
                }
#pragma unroll
                for (int h = 0; h < KS / 64; ++h) {
                    uint32_t w[kWords], o[32];
#pragma unroll
                    for (int i = 0; i < kWords / 4; ++i) {
                        const uint4 v = *reinterpret_cast<const uint4*>(raw + ((((sub * (KS / 64) + h) * (kWords / 4) + i) ^ (ch & 7u)) << 4));
                        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
                    }
#pragma unroll
                    for (int j = 0; j < kWords; ++j) {
                        if (BITS == 8) {
                            s8x4_to_bf16(w[j], flip, sel0, sel1, up.mul0, up.add, o[2 * j], o[2 * j + 1]);
                        } else {
                            uint32_t qv[4];
                            s4x8_to_bf16(w[j], flip, nib, up.mul0, up.mul1, up.add, qv);
                            o[4 * j] = qv[0]; o[4 * j + 1] = qv[1]; o[4 * j + 2] = qv[2]; o[4 * j + 3] = qv[3];
                        }
                    }
                    if (MODE == kFold && !folded) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = bf16x2_mul(o[j], up.scale);
                    }
                    if (h == 0) {
                        if (!p.slot_first && !warp_wait(step_empty(rs.i, which), rs.phase ^ 1u, abort_flag)) { give_up(36, x.t, l); ok = false; break; }
                        ptx::tc_fence_after_sync();
                    }
                    ptx::tmem_st_32x32(slot_base + ((quarter * 32u) << 16) + rs.i * kSlotCols + (l % PAIR) * kPartCols + h * 32, o);
                }
                if (!ok) break;
                if (kActApart && quarter == 0 && !warp_wait(act_full(rs.i), rs.phase, abort_flag)) { give_up(39, x.t, l); ok = false; break; }
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();   // every lane's weights are in tensor memory
                if (lane == 0) {
                    ptx::mbar_arrive(step_full(rs.i, which));
                    ptx::mbar_arrive_count(raw_empty(rr.i), left < SPB && sub + 1 == left ? 1 + SPB - left : 1u);   // a short last block: for its missing parts, too
                }
                rr.step(kGroups / SPB, p.raw_stages);   // four parts on
                rs.step(kGroups / PAIR, p.slots);
            }
            steps_before += (ns + PAIR - 1) / PAIR;
            blocks_before += x.kb1 - x.kb0;
        }
    } else if (warp >= kFirstEpi) {
        // ======================= epilogue =======================
        const uint32_t quarter = (uint32_t)warp & 3u, ch = quarter * 32 + lane;
        const uint32_t lane_base = tmem_base + ((quarter * 32u) << 16);
        const uint32_t groups_per_row = channel_scaled(MODE) ? 0 : (p.parts >> p.group_shift);
        Ring rc{0, 0};
        uint32_t meeting = 0, to_finish = 0;
        uint32_t block = 0;   // staging block of the next tile store
        bool ok = true;
        asm volatile("griddepcontrol.wait;" ::: "memory");   // workspace, counters and C belong to the predecessor until it has ended
        while (ok && walk.next(p.deal, blockIdx.x, x)) {
            uint32_t m0, n0;
            tile_origin(p, x.t, m0, n0);
            const uint32_t nn = n0 + ch, ns = parts_of(x);
            const uint32_t valid = min(p.rows, p.m - m0);
            const bool whole = x.kb0 == 0 && x.kb1 == p.deal.blocks;
            const float scale = channel_scale(nn);
            // 16 rows of this lane's channel, finished
            auto store = [&](uint32_t c0, const float (&v)[16]) {
                if (p.c_tma) {
                    // through shared memory as a tile store (clipped at the edges of C); two blocks per warp take turns
                    const uint32_t out = smem_base + kOffOut + (quarter * 2 + block) * kOutBytes;
                    if (lane == 0) ptx::bulk_wait_group_read1();
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(out + (uint32_t)j * 64u + (uint32_t)lane * 2u),
                                     "h"(__bfloat16_as_ushort(__float2bfloat16_rn(finished(v[j], scale)))) : "memory");
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        ptx::tma_store_2d(&tmap_c, out, (int)(n0 + quarter * 32u), (int)(m0 + c0));
                        ptx::bulk_commit_group();
                    }
                    block ^= 1u;
                } else if (nn < p.n) {
                    uint16_t* dst = p.c + (size_t)(m0 + c0) * p.ldc + nn;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c0 + j < valid) dst[(size_t)j * p.ldc] = __bfloat16_as_ushort(__float2bfloat16_rn(finished(v[j], scale)));
                }
            };
            float* part = p.ws + (size_t)(whole ? 0 : p.deal.slot(blockIdx.x, x.t)) * p.rows * kCh + ch;
            auto emit = [&](uint32_t c0, const float (&v)[16]) {
                if (whole) { store(c0, v); return; }
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c0 + j < valid) __stcg(part + (size_t)(c0 + j) * kCh, v[j]);
            };
            if (summed(MODE)) {
                // Added up in two levels, every kInner sums to a part of their own, as decode.cu's warps do: one chain over all groups left
                // more results wrongly rounded than decode.cu (5 x 28672 x 8192 int4 group-128: 97 of 860160 against 65, in two levels
                // 67; 16 x 8192 x 28672: 149 of 786432 against 109, 76), in the same time (49.7 us).  Eight columns at a time: 16 spill.
                constexpr uint32_t kInner = 8;
                float sum[16], inner[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[j] = inner[j] = 0.f;
                uint32_t held = 0;   // sums in `inner`
                const size_t g0 = (size_t)nn * groups_per_row;
                auto group_scale = [&](uint32_t l) {
                    if (nn >= p.n || l >= ns) return 0.f;
                    if (MODE == kParts) return 1.f;
                    const size_t i = g0 + ((x.kb0 * SPB + l) >> p.group_shift);
                    return p.scale_dtype == AFB_SCALE_BF16 ? __uint_as_float((uint32_t)reinterpret_cast<const uint16_t*>(p.scale)[i] << 16)
                                                           : reinterpret_cast<const float*>(p.scale)[i];
                };
                // the part that sum i of a set begins with: with two issuing warps 0 and 1, and the next two 2 * flush parts on
                auto begins = [&](uint32_t i) { return kDual ? (i >> 1) * 2 * p.flush + (i & 1u) : i * p.flush; };
                float sc[kSet];
#pragma unroll
                for (uint32_t i = 0; i < kSet; ++i) sc[i] = group_scale(begins(i));
                for (uint32_t l = 0; l < ns; l += kSet * p.flush) {
                    float sc_nxt[kSet];
#pragma unroll
                    for (uint32_t i = 0; i < kSet; ++i) sc_nxt[i] = group_scale(l + kSet * p.flush + begins(i));
                    if (!warp_wait(acc_full(rc.i), rc.phase, abort_flag)) { give_up(37, x.t, l); ok = false; break; }
                    ptx::tc_fence_after_sync();
#pragma unroll
                    for (uint32_t i = 0; i < kSet; ++i) {
                        if (l + begins(i) >= ns) break;
#pragma unroll
                        for (int h = 0; h < 16; h += 8) {
                            uint32_t r[8];
                            ptx::tmem_ld_32x8(lane_base + rc.i * p.acc_cols + i * 16 + h, r);
                            ptx::tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 8; ++j) inner[h + j] = fmaf(sc[i], __uint_as_float(r[j]), inner[h + j]);
                        }
                    }
                    held += kSet;
                    if (held == kInner || l + kSet * p.flush >= ns) {
                        held = 0;
#pragma unroll
                        for (int j = 0; j < 16; ++j) { sum[j] += inner[j]; inner[j] = 0.f; }
                    }
                    ptx::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(acc_empty(rc.i));
                    rc.step(1, p.accs);
#pragma unroll
                    for (uint32_t i = 0; i < kSet; ++i) sc[i] = sc_nxt[i];
                }
                if (!ok) break;
                emit(0, sum);
            } else {
                if (!warp_wait(acc_full(rc.i), rc.phase, abort_flag)) { give_up(37, x.t, 0); break; }
                ptx::tc_fence_after_sync();
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < p.rows; c0 += 32) {
                    uint32_t r[2][16];
                    ptx::tmem_ld_32x16(lane_base + rc.i * p.acc_cols + c0, r[0]);
                    if (c0 + 16 < p.rows) ptx::tmem_ld_32x16(lane_base + rc.i * p.acc_cols + c0 + 16, r[1]);
                    ptx::tmem_ld_wait();
                    if (c0 + 32 >= p.rows) {   // everything is in registers: the accumulator is free
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(acc_empty(rc.i));
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (c0 + 16 * h >= p.rows) break;
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[h][j]);
                        emit(c0 + 16 * h, v);
                    }
                }
                rc.step(1, p.accs);
            }
            if (!whole) {
                // the CTAs holding units of this tile meet at its counter
                const uint32_t first = p.deal.first_cta(x.t), last = p.deal.last_cta(x.t);
                __threadfence();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive(bar_stored);
                    if (quarter == 0) {
                        misc[2] = wait_or_abort(bar_stored, meeting, abort_flag) && atomicAdd(p.counters + x.t, 1u) == last - first ? 1u : 0u;
                        ptx::mbar_arrive(bar_verdict);
                    }
                }
                if (!warp_wait(bar_verdict, meeting, abort_flag)) { give_up(38, x.t, 0); break; }
                meeting ^= 1u;   // misc[2] is written again only after all four warps have arrived at the next meeting
                if (misc[2]) {
                    __threadfence();
                    if (p.finish_late) {   // all the warps together, when this CTA's work is done (at most two tiles are shared)
                        if (quarter == 0 && lane == 0) misc[4 + to_finish] = x.t;
                        ++to_finish;
                    } else {
                        finish_tile(x.t, threadIdx.x - 32 * kFirstEpi, 128);
                    }
                    if (quarter == 0 && lane == 0) p.counters[x.t] = 0u;
                }
            }
        }
        if (p.finish_late) {
            if (quarter == 0 && lane == 0) misc[3] = ok ? to_finish : 0u;
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar_finish);
        }
        if (p.c_tma && lane == 0) ptx::bulk_wait_group0();   // this warp's tile stores are complete
    }

    if (p.finish_late && warp >= kFirstEpi && warp_wait(bar_finish, 0u, abort_flag)) {
        __threadfence();
        for (uint32_t i = 0; i < misc[3]; ++i) finish_tile(misc[4 + i], threadIdx.x - 32 * kFirstEpi, kThreads - 32 * kFirstEpi);
    }

    // ---- teardown: every thread gets here, also after an abort ----
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <int BITS, int MODE, int KS, int PAIR>
int launch_cfg(const CUtensorMap& ta, const CUtensorMap& tw, const CUtensorMap& tc, const StreamParams& p, uint32_t grid, bool pdl,
               DeviceCtx* ctx, cudaStream_t s) {
    auto kern = stream_kernel<BITS, MODE, KS, PAIR>;
    static DeviceOnce attr_set;  // per template instance
    if (!attr_set.done(ctx->device)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e != cudaSuccess) return cuda_fail(e);
        attr_set.mark(ctx->device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(kThreads); cfg.stream = s;
    cfg.dynamicSmemBytes = 1024 + kOffRaw + p.raw_stages * kRawBytes + p.slots * p.rows * 128 * (PAIR * KS / kSlab);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tw, tc, p);
    count_launch();
    count_stream_launch();
    return e == cudaSuccess ? AFB_OK : cuda_fail(e);
}

}  // namespace

namespace {

bool stream_supports(const afb_gemm_args& a) {
    if (a.b_layout != AFB_LAYOUT_COL && a.b_layout != AFB_LAYOUT_COL_PACKED) return false;
    if (a.k % kSlab || a.lda % 8) return false;
    if (((uint64_t)a.ldb * a.b_bits / 8) % 16) return false;
    if ((uintptr_t)a.ptr_a % 16 || (uintptr_t)a.ptr_b % 16) return false;
    // forced forms, fp32 results (their order of addition is that of the exchange forms) and the two-term mode stay where they are
    // (an explicit decode or prefill variant does not: this is a form of both)
    if (a.flags & (AFB_FLAG_C_F32 | AFB_FLAG_PREFILL_SMEM_B | AFB_FLAG_PREFILL_TMEM_A)) return false;
    if ((a.flags & AFB_FLAG_GROUP_EXACT) && a.group_size) return false;
    if (a.group_size) {
        if (a.group_size % kSlab || (a.group_size & (a.group_size - 1)) || a.k % a.group_size) return false;
        if (a.m > 16 && a.scale_dtype != AFB_SCALE_BF16) return false;
    }
    return true;
}

// Rows per tile for M rows.  Up to 192 (two accumulators next to four weight slots in tensor memory), or up to 128 where steps of
// 128 k are possible and the tiles are few enough that the finer grain pays for the weights being unpacked once more per 128 rows
// instead of 192 (28672 x 8192 int4 group-128: 222 against 236 us at M = 512, 449 against 496 at 1024, 944 against 915 at 2048).
uint32_t tile_rows(const afb_gemm_args& a) {
    const bool wide_steps = a.k % 128 == 0 && a.group_size % 128 == 0;
    const uint32_t most = wide_steps && a.m > 192 && a.m <= 1024 ? 128 : 192;
    const uint32_t tiles = (a.m + most - 1) / most;
    return ((a.m + tiles - 1) / tiles + 15) / 16 * 16;
}

// Where this form is the faster one (of the forms with one SM per tile: pair.cu is asked before), from times of both forms on one B200 (us, the
// other form / this one): 23 matrices from 1024 x 1024 to 28672 x 8192, 35 row counts from 4 to 4096, int8, int4, int4 in groups of 128 and 64,
// int8 in groups of 128.  At none of those that it takes is this form more than 4 % the slower one (20 matrices again up to 16 rows, caches cold,
// with two issuing warps; of int4 in groups of 256 at one: 8 x 8192 x 8192, 25 / 27).
bool is_faster(const afb_gemm_args& a, uint32_t sms) {
    const double weights = (double)a.n * a.k, mbytes = weights * a.b_bits / 8 / 1e6;
    const uint32_t n_tiles = (a.n + kCh - 1) / kCh;
    if (a.m <= 16) {
        // The decode kernel has about 9 us less to set up and finish, and its arithmetic grows with M; this form's does not.
        //   28672 x 8192 int8   M = 2: 49 / 47   4: 56 / 46    8: 72 / 46   16: 69 / 47
        //   28672 x 8192 int4   M = 4: 60 / 49   5: 66 / 50    8: 68 / 50   16: 69 / 51    (group 128; without groups 4: 43 / 43   5: 45 / 43)
        //   12288 x 4096 int8   M = 4: 23 / 23   9: 29 / 23   16: 32 / 24;   4096 x 4096   M = 4: 12 / 19   16: 16 / 19
        // The lines date from when one warp issued both parts of a step; with two this form is the faster one below some of them, too (12288 x
        // 4096 int8 M = 8: 28 / 24;  4096 x 11008 int8 M = 5: 23 / 23;  1024 x 11008 int8 M = 9: 43 / 19).
        if (mbytes >= 100) return a.m >= (a.b_bits == 8 ? 4u : 5u);
        // Long rows: the decode kernel stages the activations in several passes.  Without groups its int4 arithmetic is so much
        // cheaper that this must cost it more, more than 192 KiB of activations:
        //   4096 x 11008 int4   M = 8: 43 / 24 (group 128)   8: 31 / 23   9: 49 / 23 (no groups);   8192 x 8192 int4   M = 8: 21 / 25   12: 39 / 25
        if (a.k >= 8192 && mbytes >= 20) return a.m >= 8 && (a.b_bits == 8 || a.group_size || a.m * a.k >= 98304);
        return mbytes >= 40 && a.m >= 9;
    }
    if (a.m <= 128) {
        // Both other forms unpack at the pace of one step's hand-off chain (79 to 88 us on 28672 x 8192 whatever M is: 45 to 69 here);
        // what remains here is the cost of sharing tiles between CTAs, which grows with M.
        if (weights >= 40e6) {
            // group-scaled:  8192 x 8192 int4: 41 / 23 to 31;  int4 in short rows of more than a wave of tiles, 28672 x 2048: 26 / 22 at M = 17,
            // 26 / 23 at 40, 27 / 31 at 128 (groups of 64: 0.98 at 32, 1.11 at 40)
            if (a.group_size) return a.b_bits == 8 || n_tiles <= sms || a.k >= 4096 || a.m <= (a.group_size % 128 ? 32u : 64u);
            // int8:  8192 x 8192: 29 to 31 / 24 to 31;  12288 x 4096: 25 / 23 at M = 64, 25 / 27 at 128;  4096 x 11008: 24 / 24 and 25 / 29
            return a.m <= 64 || weights >= 55e6;
        }
        if (a.b_bits == 8 || a.m > 40) return false;   // 4096 x 4096 int8: 16 / 17 to 22
        // Small int4 matrices, up to 40 rows.  Tiles that fill half a wave to a whole one keep the other forms busy, too:
        // 12288 x 1024: 13 / 16 group-scaled, 10 / 16 without; 16384 x 2048: 18 / 15 and 16 / 14 to 18
        if (n_tiles > sms / 2 && n_tiles <= sms) return a.k >= 2048 && (a.group_size || a.m <= 24);
        if (n_tiles > sms && a.group_size && a.k < 1536) return a.m <= 32;   // 28672 x 1024: 16 / 16 at 32, 16 / 17 at 40 (groups of 64: 1.13)
        if (a.group_size) return true;                 // 1024 x 1024 ... 8192 x 2560: this form 0.8 to 0.95 of the other; 1024 x 11008 0.3
        // 4096 x 4096: 15 / 15 at M = 20, 15 / 17 at 40;  3072 x 3072: 13 / 13 and 13 / 14;  5120 x 5120 and 1024 x 11008: 0.85 and 0.7 throughout
        return a.m <= 24 || n_tiles > sms || a.k >= 8192 || weights >= 25e6 || weights <= 5e6;
    }
    // Many rows: the tensor-memory form with 256-row tiles has the higher rate, this one fits its tiles to M and shares the last
    // ones evenly.  Group-scaled int4 is bound by the unpack there and faster here (28672 x 8192 group 128: 138 / 114 at
    // M = 256, 261 / 223 at 512, 971 / 915 at 2048, 1904 / 1819 at 4096; 4096 x 4096: 29 / 30 at 512, 72 / 68 at 2048), but for
    // next to no channels and very many rows (1024 x 11008: 91 / 77 at 3000, 94 / 110 at 4096; groups of 64 0.86).
    if (a.b_bits == 4 && a.group_size) return weights >= 40e6 || (weights * a.m >= 30e9 && (n_tiles >= 16 || a.m <= 3072 || a.group_size % 128));
    // Otherwise compared in rows per SM, with 1.2 for the difference in rate.  Without group scales the other form has little to unpack
    // besides, and the comparison holds only where its 256-row tiles are mostly padding: one tile and a little more (28672 x 8192 int8:
    // 102 / 86 at M = 129, 106 / 109 at 200; 8192 x 8192: 37 / 35 and 38 / 41; 12288 x 4096: 28 / 31 at 129), or two, with enough channels
    // (11008 x 4096: 47 / 40 at 333; 8192 x 8192: 50 / 52; at 640 and 777 rows 12288 x 4096: 56 / 63 and 78 / 80, 28672 x 8192: 353 / 392).
    // Between 193 and 256 rows it would also add up longer stretches of K in one accumulator than the other form, which cuts them
    // (8192 x 8192, 200 rows: 13057 of 9830400 results wrongly rounded, 9665 there).
    if (weights < 40e6) return false;
    if (!a.group_size && !(a.m <= 192 ? weights >= 60e6 : a.m > 256 && a.m <= 384 && n_tiles >= 80)) return false;
    const uint32_t rows = tile_rows(a);
    const uint32_t others = (a.m + 255) / 256 * n_tiles, waves = others / sms, rest = others % sms;
    const uint32_t parts = rest == 0 || rest > sms / 2 ? 1 : sms / rest < 4 ? sms / rest : 4;
    const double there = 256.0 * (waves + (rest ? 1.0 / parts : 0.0)), here = (double)((a.m + rows - 1) / rows) * n_tiles * rows / sms;
    return 1.2 * here < there;
}

}  // namespace

bool stream_is_faster(const afb_gemm_args& a, uint32_t sms) { return stream_supports(a) && is_faster(a, sms); }

// A tuning variable that asks for one of the variant's other forms, or for a shape of theirs.
static bool other_form_asked(uint32_t variant) {
    if (variant == AFB_VARIANT_PREFILL) return getenv("AFB_PREFILL_IMPL") != nullptr;
    for (const char* name : {"AFB_DECODE_BALANCED", "AFB_DECODE_WR", "AFB_DECODE_SLICES", "AFB_DECODE_DEEP_RING", "AFB_DECODE_SINGLE_PASS"})
        if (getenv(name)) return true;
    return false;
}

int stream_if_faster(const afb_gemm_args& a, uint32_t variant, DeviceCtx* ctx, cudaStream_t s, bool* done) {
    *done = false;
    const char* env = getenv("AFB_STREAM");   // tuning aid: 1 wherever possible, 0 never
    const int forced = env ? atoi(env) : -1;
    if (forced == 0 || !stream_supports(a) || (forced < 0 && (!is_faster(a, (uint32_t)ctx->sm_count) || other_form_asked(variant)))) return AFB_OK;
    const uint32_t sms = (uint32_t)ctx->sm_count;
    StreamParams p{};
    p.c = reinterpret_cast<uint16_t*>(a.ptr_c);
    p.scale = a.ptr_scale;
    p.zero = reinterpret_cast<const uint8_t*>(a.ptr_zero);
    p.m = a.m; p.n = a.n; p.k = a.k; p.ldc = a.ldc;
    p.enc = a.b_encoding; p.scale_dtype = a.scale_dtype;
    p.packed = a.b_layout == AFB_LAYOUT_COL_PACKED ? 1u : 0u;
    const int mode = a.m > 16 ? (a.group_size ? kFold : kChannel) : (a.group_size ? kSums : kParts);
    p.rows = tile_rows(a);
    p.m_tiles = (a.m + p.rows - 1) / p.rows;
    p.n_tiles = (a.n + kCh - 1) / kCh;
    p.group_m = pick_group_m(a, p.m_tiles, p.n_tiles, p.rows, ctx->sm_count);
    // k per step: 128 halves the number of hand-offs per weight, which is what bounds few rows; more rows need the tensor memory
    // for their accumulators, and steps of 64 keep the tensor cores busy for longer than a hand-off takes
    const uint32_t ks = p.rows <= 128 && a.k % 128 == 0 && a.group_size % 128 == 0 ? 128 : 64;
    const uint32_t spb = (a.b_bits == 8 ? 128 : 256) / ks;
    p.parts = a.k / ks;
    while (a.group_size && ks << p.group_shift < a.group_size) ++p.group_shift;
    const uint32_t pair = ks == 128 && p.rows <= 64 ? 2 : 1;
    const bool dual = pair == 2 && summed(mode);   // parts per sum are then those of one issuing warp, and two parts are never in one group's sum
    p.flush = mode == kParts ? kPartSum / ks : mode == kSums ? (dual ? 1 : 1u << p.group_shift < spb ? 1u << p.group_shift : spb) : 0;
    p.acc_cols = summed(mode) ? kSet * 16 : p.rows;
    p.accs = p.rows <= 192 ? 2 : 1;
    p.slots = (kTmemCols - p.accs * p.acc_cols) / (pair * ks / 2);
    if (p.slots > (uint32_t)kMaxSlots) p.slots = kMaxSlots;
    const uint32_t act_bytes = p.rows * ks * 2 * pair;
    while (p.slots * pair > (uint32_t)kGroups && (kRingBudget - p.slots * act_bytes) / kRawBytes < p.slots * pair) --p.slots;
    p.raw_stages = (kRingBudget - p.slots * act_bytes) / kRawBytes;
    if (p.raw_stages > (uint32_t)kMaxRaw) p.raw_stages = kMaxRaw;

    if (dual)   // see kDual in the kernel
        p.raw_stages -= p.raw_stages % (kGroups / spb);
    // A converter warp sees only every fourth part, and a wait for phase n of a raw stage means something only once phase n - 1 has
    // completed.  What tells it that is the MMA order: a free slot means that everything up to `slots` steps earlier has been
    // consumed.  With the slot wait of the PREVIOUS part behind it, up to 3 + slots * pair earlier parts may still be under way,
    // with that of its own part up to slots * pair - 1; a raw block has at least one part, so the ring must be longer than that.
    p.slot_first = p.raw_stages >= kGroups + p.slots * pair ? 0u : 1u;
    if (p.raw_stages < p.slots * pair || p.slots * pair < (uint32_t)kGroups) return AFB_OK;

    p.deal = deal_tiles(p.m_tiles * p.n_tiles, (p.parts + spb - 1) / spb, sms);
    if (!p.deal.fits()) return AFB_OK;
    const uint32_t grid = p.deal.grid;
    if (p.deal.shared_tiles) {
        if (p.deal.shared_tiles > ctx->stream_counter_count) return AFB_OK;
        if (!stream_workspace(ctx, s, (size_t)2 * grid * p.rows * kCh * sizeof(float), &p.ws, &p.counters)) return AFB_OK;   // the caller's other forms
    }
    p.status = ctx->status;

    *done = true;
    CUtensorMap ta, tw;
    int rc = tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.ptr_a, a.k, a.m, (uint64_t)a.lda * 2, kSlab, p.rows, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.ptr_b, (uint64_t)a.k * a.b_bits / 8, a.n, (uint64_t)a.ldb * a.b_bits / 8, 128, kCh,
                 CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    CUtensorMap tc = ta;
    p.c_tma = a.ldc % 8 == 0 && (uintptr_t)a.ptr_c % 16 == 0 && a.n % 8 == 0 &&
              tmap_2d(&tc, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.ptr_c, a.n, a.m, (uint64_t)a.ldc * 2, 32, 16, CU_TENSOR_MAP_SWIZZLE_NONE) == AFB_OK;
    p.c_vec = a.ldc % 4 == 0 && (uintptr_t)a.ptr_c % 8 == 0;
    p.finish_late = p.deal.whole_waves == 0 || (p.deal.whole_waves == 1 && p.rows > 32);
    const bool pdl = (a.flags & AFB_FLAG_PDL) != 0 && a.m <= 16;   // of the decode variant only
#define AFB_STREAM_LAUNCH(B, M) (pair == 2 ? launch_cfg<B, M, 128, 2>(ta, tw, tc, p, grid, pdl, ctx, s) : ks == 128 ? launch_cfg<B, M, 128, 1>(ta, tw, tc, p, grid, pdl, ctx, s) : launch_cfg<B, M, 64, 1>(ta, tw, tc, p, grid, pdl, ctx, s))
    switch (mode) {
        case kChannel: return a.b_bits == 8 ? AFB_STREAM_LAUNCH(8, kChannel) : AFB_STREAM_LAUNCH(4, kChannel);
        case kFold:    return a.b_bits == 8 ? AFB_STREAM_LAUNCH(8, kFold) : AFB_STREAM_LAUNCH(4, kFold);
        case kSums:    return a.b_bits == 8 ? AFB_STREAM_LAUNCH(8, kSums) : AFB_STREAM_LAUNCH(4, kSums);
        default:       return a.b_bits == 8 ? AFB_STREAM_LAUNCH(8, kParts) : AFB_STREAM_LAUNCH(4, kParts);
    }
#undef AFB_STREAM_LAUNCH
}

}  // namespace afb
