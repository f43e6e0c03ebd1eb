// Pair form of the prefill variant (more than 64 activation rows, B in [N,K] layout), also with the fused epilogue: two SMs on one tile
// (reference counterpart of the whole kernel: bf16gemm_kernel_gfx90a.s:184-636).
//
// As in the streaming form, D[n, m] = sum_k W[n,k] * A[m,k] with the unpacked weights as the tensor-memory operand.  A cluster of two CTAs
// owns 256 output channels x `rows` (up to 256) activation rows: each unpacks its own 128 channels into its own tensor memory, each loads
// half of the activation rows, and one tcgen05.mma.cta_group::2 reads both halves.
//
//   warp 0        TMA: raw weight blocks, 128 channels x 128 bytes, 128-byte swizzle
//   warp 1        TMA: this CTA's half of the activation rows, [rows / 2 x 64] bf16 slabs, 128-byte swizzle
//   warp 2        rank 0: tcgen05.mma 256 x rows x 16;  rank 1: reports to rank 0 that its half of a step is complete
//   warps 4-11    epilogue, two per lane quarter: accumulator -> registers or shared memory -> (accumulator free) -> C, or fp32 partial
//                 sums -> workspace
//   warps 12-27   converters: four groups of four warps; group g takes every fourth step of k (KS = 128 or 64 wide)
//
// Work is dealt over the pairs as the streaming form deals it over CTAs (stream_deal.h); the two CTAs of a pair finish their channels of
// a shared tile by themselves.
//
// What bounded the forms with one SM per tile: 256 rows of activations and 128 channels of weights per 64 k are 40 KiB against 512 cycles of
// tensor work, 80 bytes a cycle where an SM takes in 64 (2048 x 11008 x 4096 int8: 1.80 GB, 55 bytes a cycle in the full waves, tensor
// pipe 66 %).  Here it is 24 KiB.  What set the pace next:
//   the issuing warp: 700 cycles per hand-off of 64 k (a wait 80, four MMAs 240, a commit to both CTAs 180, the loop), so a step is 128 k
//     wherever K and the groups allow it: 820 against 1024 cycles of tensor work;
//   one accumulator of 256 columns next to four weight slots: it is drained in one go (packed bf16 in registers; of gate * up into shared
//     memory) and stored from there: 1500 cycles a tile; storing as it was drained held it for 5800;
//   the converters' own instructions: a whole step per group, its words loaded first (64 k at a time took 15 % longer on 128 rows);
//   the hand-off between the SMs: see mbar_arrive_remote.
// Measured (one B200, caches cold between passes, the forms before / this one): 4096 x 28672 x 8192 int4 group-128 1909 / 1380 us, 2048 x
// 11008 x 4096 int8 165 / 150, 128 x 28672 x 8192 int4 79 / 71, gated 1000 x 2*11008 x 4096 int8 224 / 179.  The tensor pipe is now fed as fast as
// it goes in the main loop of 256-row tiles (1036 cycles per 128 k); the clock (1.5 to 1.6 GHz under the power limit) and the last wave set the rest.
// ptxas spills 96 to 140 bytes in the instances without fused epilogue, whose epilogue holds 64 registers of results once per tile, and 24 to
// 132 in the others.
#include <cstdlib>
#include "dequant.cuh"
#include "stream_common.cuh"

namespace afb {

namespace {

constexpr int kFirstEpi = 4, kEpiWarps = 8, kFirstConv = kFirstEpi + kEpiWarps;
constexpr int kThreads = 32 * (kFirstConv + 4 * kGroups);   // 896: launched with 72 registers a thread
// Registers of the three kinds of warps.
constexpr uint32_t kRegsCtrl = 56;
__host__ __device__ constexpr uint32_t regs_epi(bool fused) { return fused ? 112 : 96; }
__host__ __device__ constexpr uint32_t regs_conv(bool fused) { return fused ? 56 : 64; }
constexpr bool regs_fit(bool fused) { return 128 * kRegsCtrl + 32 * kEpiWarps * regs_epi(fused) + 128 * kGroups * regs_conv(fused) <= 72 * kThreads; }
static_assert(regs_fit(false) && regs_fit(true), "shares of the registers");
constexpr uint32_t kFinishWarps = kEpiWarps + 4 * kGroups;   // of each CTA that shares a tile
constexpr uint32_t kTileWords = 3;                      // counters of a shared tile and rank
constexpr int kMaxRaw = 12, kMaxSlots = 8, kMaxAcc = 2;
__host__ __device__ constexpr uint32_t slots(int ks) { return ks == 128 ? 4 : 6; }   // steps under way, in 256 columns at most
constexpr uint32_t kTmemCols = 512;
constexpr int kBars = 2 * (kMaxRaw + kMaxSlots + kMaxAcc) + 2;
constexpr int kOffMisc = kBars * 8, kOffOut = 1024;
constexpr int kOutBytes = 16 * 32 * 2;   // one block of the result: 16 rows x 32 channels
// Staging of one epilogue warp: two blocks, or a warp's whole part of a gated tile (128 rows x 16 channels).
__host__ __device__ constexpr int out_bytes(bool fused) { return fused ? 128 * 16 * 2 : 2 * kOutBytes; }
__host__ __device__ constexpr int off_raw(bool fused) { return kOffOut + kEpiWarps * out_bytes(fused); }
__host__ __device__ constexpr int ring_budget(bool fused) { return 232448 - 1024 - off_raw(fused); }   // bytes for the two rings (1 KiB for the alignment of the base)
static_assert(kOffMisc + 32 <= kOffOut && off_raw(false) % 1024 == 0 && off_raw(true) % 1024 == 0, "shared memory layout");

struct PairParams {
    uint16_t* c;
    const void* scale;
    const uint8_t* zero;
    uint32_t m, n, k, ldc;
    uint32_t enc, scale_dtype, packed;
    uint32_t group_shift;     // log2(group / KS)
    uint32_t rows, m_tiles, n_tiles, group_m;
    uint32_t steps;           // steps along K
    StreamDeal deal;          // who does what, in units of one raw block
    uint32_t raw_stages, accs;
    uint32_t stretches;       // of K, each in columns of its own and added up in fp32 at the end (1, or where a pair has one whole tile: 2, 4)
    uint32_t slot_first;      // converters wait for their slot before they wait for their raw block
    float* ws;                // [(2 * pair + (not the pair's first shared tile)) * 2 + rank][row][channel]
    uint32_t* counters;       // kTileWords for each rank of a shared tile, zero on entry and on exit
    int32_t* status;
    // fused epilogue: v = sum * scale + bias[channel]; gated: channels 2i / 2i + 1 are gate and up of output channel i, C = act(gate) * up,
    // else C = act(v); then + residual; one rounding
    const float* bias;
    const uint16_t* residual;
    uint32_t ld_res, gated, act;
};

// Groups of group_m row tiles; inside a group the channel tiles advance, row tile fastest.  n0: of this CTA's 128 channels.
__device__ __forceinline__ void tile_origin(const PairParams& p, uint32_t rank, uint32_t t, uint32_t& m0, uint32_t& n0) {
    const uint32_t per_group = p.group_m * p.n_tiles;
    const uint32_t g = t / per_group, r = t - g * per_group;
    const uint32_t gsz = min(p.group_m, p.m_tiles - g * p.group_m);
    const uint32_t nt = r / gsz;
    n0 = (2 * nt + rank) * kCh;
    m0 = (g * p.group_m + (r - nt * gsz)) * p.rows;
}

__device__ __forceinline__ float bf16_value(uint32_t bits) { return __uint_as_float(bits << 16); }
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// 1 / (1 + 2^t), t = -v log2(e), without a branch.  The rounding error of the product t comes back as a first-order factor (TwoProduct by
// fused multiply-add, Ogita, Rump and Oishi 2005): without it, as in exp(), it grows with |v|.  Beyond the clamp the result is 0 or 1 in fp32;
// NaN and infinities come back with the v that the caller multiplies by.
__device__ __forceinline__ float sigmoid(float v) {
    const float x = fminf(fmaxf(v, -128.f), 128.f);
    constexpr float kLog2e = 1.44269504f, kLn2 = 0.69314718f, kLog2eLow = 1.92596299e-8f;   // log2(e) = kLog2e + kLog2eLow
    const float t = x * -kLog2e, low = fmaf(x, -kLog2eLow, fmaf(x, -kLog2e, -t));
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
    const float better = fmaf(e, low * kLn2, e);
    e = t < 128.f ? better : e;   // infinite from there on
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    return r;
}

template <int N> struct Rows { static constexpr int value = N; };

template <int BITS, bool GROUPED, int KS, bool FUSED>
__global__ void __launch_bounds__(kThreads, 1)
pair_kernel(const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_w, const PairParams p) {
    constexpr uint32_t SPB = (BITS == 8 ? 128 : 256) / KS;   // steps per raw block
    constexpr uint32_t kSlotCols = KS / 2;                   // TMEM columns of a step's weights
    constexpr uint32_t kSlots = slots(KS);
    constexpr int kOffRaw = off_raw(FUSED);
    extern __shared__ uint8_t smem_raw_base[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw_base) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw_base + (smem_base - ptx::smem_u32(smem_raw_base));
    auto bar = [&](uint32_t i) { return smem_base + 8u * i; };
    auto raw_full = [&](uint32_t s) { return bar(s); };
    auto raw_empty = [&](uint32_t s) { return bar(kMaxRaw + s); };
    auto step_full = [&](uint32_t s) { return bar(2 * kMaxRaw + s); };                // weights in TMEM, activations in shared memory; rank 0: of both CTAs
    auto step_empty = [&](uint32_t s) { return bar(2 * kMaxRaw + kMaxSlots + s); };   // the MMAs of the step are done with both
    auto acc_full = [&](uint32_t s) { return bar(2 * (kMaxRaw + kMaxSlots) + s); };
    auto acc_empty = [&](uint32_t s) { return bar(2 * (kMaxRaw + kMaxSlots) + kMaxAcc + s); };   // rank 0: of both CTAs
    // a shared tile: every epilogue warp has published its part.  All shared tiles of this CTA have been
    const uint32_t bar_stored = bar(kBars - 2), bar_finish = bar(kBars - 1);
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_gen + kOffMisc);   // TMEM base, abort flag, -, number of shared tiles, which
    volatile uint32_t* abort_flag = misc + 1;
    const uint32_t act_rows = p.rows / 2, slab_bytes = act_rows * 128u, act_bytes = slab_bytes * (KS / kSlab), off_act = kOffRaw + p.raw_stages * kRawBytes;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_rank(), worker = blockIdx.x >> 1;

    // Warp 0 needs only its own barriers: it starts the weight stream while the others are still setting up.
    if (warp == 0) {
        if (lane == 0) {
            for (uint32_t s = 0; s < p.raw_stages; ++s) { ptx::mbar_init(raw_full(s), 1); ptx::mbar_init(raw_empty(s), 4 * SPB); }
            *abort_flag = 0;
            ptx::fence_mbar_init();
        }
        __syncwarp();
        ptx::cluster_arrive();
    } else {
        if (warp == 1 && lane == 0) {
            for (uint32_t s = 0; s < kSlots; ++s) { ptx::mbar_init(step_full(s), 4 + 1 + (rank == 0 ? 1 : 0)); ptx::mbar_init(step_empty(s), 1); }
            for (uint32_t s = 0; s < p.accs; ++s) { ptx::mbar_init(acc_full(s), 1); ptx::mbar_init(acc_empty(s), 2 * kEpiWarps); }
            ptx::mbar_init(bar_stored, kEpiWarps);
            ptx::mbar_init(bar_finish, 1);
            ptx::fence_mbar_init();
            ptx::prefetch_tmap(&tmap_act);
        }
        if (warp == 2) {
            ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(misc)), kTmemCols);
            ptx::tmem_relinquish_pair();
        }
        __syncwarp();
        ptx::tc_fence_before_sync();
        ptx::cluster_arrive();
        ptx::cluster_wait();   // both CTAs' barriers are there
        ptx::tc_fence_after_sync();
    }
    constexpr uint32_t tmem_base = 0;   // all 512 columns are this CTA's: the allocation starts at column 0
    const uint32_t slot_base = tmem_base + kTmemCols - kSlots * kSlotCols;   // accumulators from column 0, slots at the end

    auto give_up = [&](int where, uint32_t a, uint32_t b) {
        if (!*abort_flag) { report_timeout(p.status, where, (int)a, (int)b); *abort_flag = 1; }
    };
    Walk walk;
    walk.start(p.deal, worker);   // every role of both CTAs walks the same list of pieces
    Piece x;
    auto steps_of = [&](const Piece& q) { return min(q.kb1 * SPB, p.steps) - q.kb0 * SPB; };

    auto channel_scale = [&](uint32_t nn) {
        if (GROUPED || nn >= p.n) return 0.f;
        return p.scale_dtype == AFB_SCALE_BF16 ? bf16_value(reinterpret_cast<const uint16_t*>(p.scale)[nn]) : reinterpret_cast<const float*>(p.scale)[nn];
    };
    // the sum of products as the user's weights give it, with the channel's scale and bias
    auto finished = [&](float sum, float scale, float bias) {
        if (!FUSED) return GROUPED ? sum * kGroupInverse : unscaled(sum, scale);
        return GROUPED ? fmaf(sum, kGroupInverse, bias) : fmaf(sum * kUnpackInverse, scale, bias);
    };
    const bool silu = p.act == AFB_ACT_SILU;
    auto activated = [&](float v) { return v * (silu ? sigmoid(v) : 1.f); };

    // Adds the partial sums of kChunkRows rows of shared tile t in pair order, finishes and stores them; one warp, four channels of a row per
    // lane, `rows_at_once` rows at a time (loads in flight).
    constexpr uint32_t kChunkRows = 4;
    auto finish_rows = [&](uint32_t t, uint32_t row_begin, auto rows_at_once) {
        uint32_t m0, n0;
        tile_origin(p, rank, t, m0, n0);
        const uint32_t first = p.deal.first_cta(t), last = p.deal.last_cta(t);
        const uint32_t valid = min(p.rows, p.m - m0);
        const uint32_t nn = n0 + (uint32_t)lane * 4;
        if (nn >= p.n) return;   // n is a multiple of 8
        const uint32_t first_slot = p.deal.slot(first, t);   // the others' runs begin in this tile: slot 2c
        const size_t stride = (size_t)p.rows * (kCh / 4);
        constexpr int kRows = decltype(rows_at_once)::value;
#pragma unroll 1
        for (uint32_t r0 = row_begin; r0 < row_begin + kChunkRows; r0 += kRows) {
            if (r0 >= valid) break;
            float4 sum[kRows];
#pragma unroll
            for (int h = 0; h < kRows; ++h) sum[h] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (uint32_t c = first; c <= last; ++c) {
                // rows beyond the last valid one hold whatever was there before; they are not stored
                const float4* src = reinterpret_cast<const float4*>(p.ws) + (size_t)((c == first ? first_slot : 2 * c) * 2 + rank) * stride + r0 * (kCh / 4) + lane;
                float4 y[kRows];
#pragma unroll
                for (int h = 0; h < kRows; ++h) y[h] = __ldcg(src + h * (kCh / 4));
#pragma unroll
                for (int h = 0; h < kRows; ++h) { sum[h].x += y[h].x; sum[h].y += y[h].y; sum[h].z += y[h].z; sum[h].w += y[h].w; }
            }
#pragma unroll
            for (int h = 0; h < kRows; ++h) {
                if (r0 + h >= valid) break;
                const size_t row = m0 + r0 + h;
                float o[4] = {sum[h].x, sum[h].y, sum[h].z, sum[h].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) o[e] = finished(o[e], channel_scale(nn + e), FUSED && p.bias ? p.bias[nn + e] : 0.f);
                if (FUSED && p.gated) {
                    o[0] = activated(o[0]) * o[1];
                    o[1] = activated(o[2]) * o[3];
                    if (p.residual) {
                        const uint16_t* res = p.residual + row * p.ld_res + (nn >> 1);
                        o[0] += bf16_value(res[0]); o[1] += bf16_value(res[1]);
                    }
                    *reinterpret_cast<uint32_t*>(p.c + row * p.ldc + (nn >> 1)) = bf16_pair(o[0], o[1]);
                } else {
                    if (FUSED) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            o[e] = activated(o[e]);
                            if (p.residual) o[e] += bf16_value(p.residual[row * p.ld_res + nn + e]);
                        }
                    }
                    *reinterpret_cast<uint2*>(p.c + row * p.ldc + nn) = make_uint2(bf16_pair(o[0], o[1]), bf16_pair(o[2], o[3]));
                }
            }
        }
    };
    // The end of a CTA's work: what it shared with others is finished by the warps of all of them, kChunkRows rows at a time, as they come
    // free.  A warp that comes before the last contribution leaves the tile to the others; the CTA that makes it comes after it.
    auto finish_shared = [&](auto rows_at_once) {
        if (!p.deal.shared_tiles || !warp_wait(bar_finish, 0u, abort_flag)) return;
        const uint32_t n = misc[3];
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i) {
            const uint32_t t = misc[4 + i], parts = p.deal.last_cta(t) - p.deal.first_cta(t) + 1;
            uint32_t* word = p.counters + (2 * t + rank) * kTileWords;   // contributions, chunks taken, warps that have left
            uint32_t seen = 0;
            if (lane == 0) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(word) : "memory");
            const bool complete = __shfl_sync(0xffffffffu, seen, 0) == parts;
            __syncwarp();   // the other lanes' loads of the partial sums are ordered after lane 0's acquire
            if (complete) {
                for (;;) {
                    uint32_t chunk = 0;
                    if (lane == 0) chunk = atomicAdd(word + 1, 1u);
                    chunk = __shfl_sync(0xffffffffu, chunk, 0);
                    if (chunk >= p.rows / kChunkRows) break;
                    finish_rows(t, chunk * kChunkRows, rows_at_once);
                }
            }
            if (lane == 0 && atomicAdd(word + 2, 1u) == parts * kFinishWarps - 1) { word[0] = 0u; word[1] = 0u; word[2] = 0u; }
        }
    };

    // Warps 0 to 2 run their loops as whole warps and elect a lane for the asynchronous instructions only (stream.cu).
    if (warp < kFirstEpi) {
        ptx::regs_down<kRegsCtrl>();
        Ring r{0, 0};
        uint32_t issued = 0, parity = 0;
        bool ok = true;
        if (warp == 0) {
            // ======================= TMA: raw weights =======================
            while (ok && walk.next<true>(p.deal, worker, x)) {
                uint32_t m0, n0;
                tile_origin(p, rank, x.t, m0, n0);
                for (uint32_t kb = x.kb0; kb < x.kb1; ++kb) {
                    if (!warp_wait(raw_empty(r.i), r.phase ^ 1u, abort_flag)) { give_up(51, x.t, kb); ok = false; break; }
                    if (ptx::elect_one()) {
                        ptx::mbar_arrive_expect_tx(raw_full(r.i), kRawBytes);
                        ptx::tma_load_2d(smem_base + kOffRaw + r.i * kRawBytes, &tmap_w, (int)(kb * 128u), (int)n0, raw_full(r.i));
                    }
                    issued |= 1u << r.i; parity = (parity & ~(1u << r.i)) | (r.phase << r.i);
                    r.step(1, p.raw_stages);
                }
            }
            for (uint32_t s = 0; s < p.raw_stages; ++s)   // never leave with a bulk copy still writing this CTA's shared memory
                if (issued & (1u << s)) ptx::mbar_wait(raw_full(s), (parity >> s) & 1u);
        } else if (warp == 1) {
            // ======================= TMA: activations =======================
            while (ok && walk.next<true>(p.deal, worker, x)) {
                uint32_t m0, n0;
                tile_origin(p, rank, x.t, m0, n0);
                const uint32_t k0 = x.kb0 * SPB, ns = steps_of(x);
                for (uint32_t l = 0; l < ns; ++l) {
                    if (!warp_wait(step_empty(r.i), r.phase ^ 1u, abort_flag)) { give_up(52, x.t, l); ok = false; break; }
                    if (ptx::elect_one()) {
                        ptx::mbar_arrive_expect_tx(step_full(r.i), act_bytes);
#pragma unroll
                        for (int h = 0; h < KS / kSlab; ++h)
                            ptx::tma_load_2d(smem_base + off_act + r.i * act_bytes + h * slab_bytes, &tmap_act, (int)((k0 + l) * KS + h * kSlab), (int)(m0 + rank * act_rows), step_full(r.i));
                    }
                    issued |= 1u << r.i; parity = (parity & ~(1u << r.i)) | (r.phase << r.i);
                    r.step(1, kSlots);
                }
            }
            // nor with a copy on its way, nor while a commit of rank 0 may still arrive here
            for (uint32_t s = 0; s < kSlots; ++s)
                if (issued & (1u << s)) (void)warp_wait(step_empty(s), (parity >> s) & 1u, abort_flag);
            for (uint32_t s = 0; s < kSlots; ++s)
                if (issued & (1u << s)) ptx::mbar_wait(step_full(s), (parity >> s) & 1u);   // after an abort the converters' part may be missing: then the limit of the wait, far above the time of a copy
        } else if (warp == 2 && rank == 0) {
            // ======================= MMA issuer =======================
            const uint32_t idesc = ptx::umma_idesc_bf16_f32(2 * kCh, p.rows);
            const uint64_t desc0 = ptx::umma_desc_kmajor_sw128(smem_base + off_act);
            const uint32_t slab_d = slab_bytes >> 4, act_d = act_bytes >> 4;   // in units of the descriptor's address field
            Ring rc{0, 0};
            bool ready = false, more = true;
            uint32_t l = 0, ns = 0, td = tmem_base, acc_done = 0, phase = 0, stretch = 0, from = 0, to = 0;
            while (more) {
#pragma unroll
                for (uint32_t s = 0; s < kSlots; ++s) {   // the slots in turn, so that what belongs to one is a constant of the loop
                    if (l == ns) {
                        if (!walk.next<true>(p.deal, worker, x)) { more = false; break; }
                        l = 0; ns = steps_of(x);
                        td = tmem_base + rc.i * p.rows; acc_done = acc_full(rc.i);
                        stretch = 0; from = 0; to = ns / p.stretches;
                        if (!warp_wait(acc_empty(rc.i), rc.phase ^ 1u, abort_flag)) { give_up(53, x.t, 0); more = false; break; }
                        rc.step(1, p.accs);
                    }
                    if (!__all_sync(0xffffffffu, ready) && !warp_wait(step_full(s), phase, abort_flag)) { give_up(54, x.t, l); more = false; break; }
                    ptx::tc_fence_after_sync();
                    ready = ptx::mbar_test_wait(step_full((s + 1) % kSlots), s + 1 == kSlots ? phase ^ 1u : phase);   // of the next step: the answer is back when this one has been issued
                    if (l == to && p.stretches > 1) { td += p.rows; from = l; to = ++stretch + 1 < p.stretches ? to + ns / p.stretches : ns; }
                    if (ptx::elect_one()) {
#pragma unroll
                        for (int j = 0; j < KS / 16; ++j)
                            ptx::umma_bf16_ts_pair(td, slot_base + s * kSlotCols + 8 * j, desc0 + s * act_d + (uint32_t)(j / 4) * slab_d + 2u * (j % 4), idesc, ((l - from) | (uint32_t)j) ? 1u : 0u);
                        ptx::umma_commit_pair(step_empty(s));
                        if (l + 1 == ns) ptx::umma_commit_pair(acc_done);
                    }
                    ++l;
                }
                phase ^= 1u;
            }
        } else if (warp == 2) {
            // ======================= rank 1: reports its half of each step =======================
            // One warp with nothing else under way, behind the barrier of its own CTA; rank 0 waits for one arrival more.
            while (ok && walk.next<true>(p.deal, worker, x)) {
                const uint32_t ns = steps_of(x);
                for (uint32_t l = 0; l < ns; ++l) {
                    if (!warp_wait(step_full(r.i), r.phase, abort_flag)) { give_up(55, x.t, l); ok = false; break; }
                    ptx::tc_fence_after_sync();
                    ptx::tc_fence_before_sync();
                    if (ptx::elect_one()) ptx::mbar_arrive_remote(step_full(r.i), 0);
                    r.step(1, kSlots);
                }
            }
        }
    } else if (warp >= kFirstConv) {
        // ======================= converters =======================
        ptx::regs_down<regs_conv(FUSED)>();
        const uint32_t g = (uint32_t)(warp - kFirstConv) >> 2, quarter = (uint32_t)warp & 3u;
        const uint32_t ch = quarter * 32 + lane;
        const uint32_t flip = BITS == 8 ? flip8(p.enc) : flip4(p.enc);
        const uint32_t sel0 = p.packed ? kSel8Strided02 : kSel8Natural01, sel1 = p.packed ? kSel8Strided13 : kSel8Natural23;
        const Nibbles nib = nibbles(p.packed != 0);
        const bool has_zero = p.zero != nullptr;
        const uint32_t groups_per_row = GROUPED ? p.steps >> p.group_shift : 0;
        auto zero_of = [&](uint32_t zb) { return !has_zero ? 0 : (BITS == 8 ? decode_zero8(zb, p.enc) : decode_zero4(zb, p.enc)); };
        GroupUnpack up;
        up.mul0 = BITS == 8 ? kMulByte : nib.mul[0]; up.mul1 = nib.mul[1]; up.add = unpack_add(BITS, 0); up.scale = 0;
        const GroupFold fold = group_fold(BITS, nib);
        const uint32_t row = kOffRaw + ch * 128, swz = (ch & 7u) << 4, lanes = (quarter * 32u) << 16;
        uint32_t steps_before = 0, blocks_before = 0;   // of the pieces walked so far
        bool ok = true;
        while (ok && walk.next<true>(p.deal, worker, x)) {
            uint32_t m0, n0;
            tile_origin(p, rank, x.t, m0, n0);
            const uint32_t nn = n0 + ch, ns = steps_of(x), k0 = x.kb0 * SPB;
            const size_t g0 = (size_t)nn * groups_per_row;
            uint32_t sc_nxt = 0, zb_nxt = 0;
            auto load_group = [&](uint32_t l, uint32_t& s, uint32_t& z) {
                if (!GROUPED || nn >= p.n || l >= ns) return;
                const size_t i = g0 + ((k0 + l) >> p.group_shift);
                s = reinterpret_cast<const uint16_t*>(p.scale)[i];
                if (has_zero) z = p.zero[i];
            };
            if (!GROUPED && has_zero) up.add = unpack_add(BITS, zero_of(nn < p.n ? p.zero[nn] : 0u));
            uint32_t l = (g - steps_before) & (kGroups - 1);
            Ring rr, rs;
            rr.set(blocks_before + l / SPB, p.raw_stages);
            rs.set(steps_before + l, kSlots);
            load_group(l, sc_nxt, zb_nxt);
            for (; l < ns; l += kGroups) {
                const uint32_t sub = l % SPB;
                bool folded = true;
                if (GROUPED) {
                    const uint32_t sc = sc_nxt, zb = zb_nxt;
                    load_group(l + kGroups, sc_nxt, zb_nxt);
                    folded = __all_sync(0xffffffffu, group_folds((uint16_t)sc, has_zero));
                    if (folded) group_folded(fold, (uint16_t)sc, up);
                    else up = group_unpack(BITS, (uint16_t)sc, zero_of(zb), false, nib);
                }
                if (p.slot_first && !warp_wait(step_empty(rs.i), rs.phase ^ 1u, abort_flag)) { give_up(56, x.t, l); ok = false; break; }
                if (!warp_wait(raw_full(rr.i), rr.phase, abort_flag)) { give_up(57, x.t, l); ok = false; break; }
                const uint32_t raw = smem_base + row + rr.i * kRawBytes, slot = slot_base + lanes + rs.i * kSlotCols;
                // KS / 64 times: the raw words of 64 k (of int4 the whole step's) first, then 32 k at a time
                constexpr int kWords = BITS == 8 ? 16 : KS / 8, kPieces = BITS == 8 ? KS / 64 : 1, kPerStore = BITS == 8 ? 8 : 4;
#pragma unroll
                for (int h = 0; h < kPieces; ++h) {
                    uint32_t w[kWords];
#pragma unroll
                    for (int i = 0; i < kWords / 4; ++i) {
                        const uint32_t at = raw + ((((sub * kPieces + h) * (kWords / 4) + i) << 4) ^ swz);
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4 * i]), "=r"(w[4 * i + 1]), "=r"(w[4 * i + 2]), "=r"(w[4 * i + 3]) : "r"(at));
                    }
#pragma unroll
                    for (int q = 0; q < kWords / kPerStore; ++q) {
                        uint32_t o[16];
#pragma unroll
                        for (int j = 0; j < kPerStore; ++j) {
                            const uint32_t v = w[q * kPerStore + j];
                            if (BITS == 8) {
                                s8x4_to_bf16(v, flip, sel0, sel1, up.mul0, up.add, o[2 * j], o[2 * j + 1]);
                            } else {
                                uint32_t qv[4];
                                s4x8_to_bf16(v, flip, nib, up.mul0, up.mul1, up.add, qv);
                                o[4 * j] = qv[0]; o[4 * j + 1] = qv[1]; o[4 * j + 2] = qv[2]; o[4 * j + 3] = qv[3];
                            }
                        }
                        if (GROUPED && !folded) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) o[j] = bf16x2_mul(o[j], up.scale);
                        }
                        if (h == 0 && q == 0) {
                            if (!p.slot_first && !warp_wait(step_empty(rs.i), rs.phase ^ 1u, abort_flag)) { give_up(56, x.t, l); ok = false; break; }
                            ptx::tc_fence_after_sync();
                        }
                        ptx::tmem_st_32x16(slot + (h * (kWords / kPerStore) + q) * 16, o);
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                ptx::tmem_st_wait();
                ptx::tc_fence_before_sync();
                __syncwarp();   // every lane's weights are in tensor memory
                if (lane == 0) {
                    ptx::mbar_arrive(step_full(rs.i));
                    const uint32_t left = ns - (l - sub);   // steps of this block and all after it
                    ptx::mbar_arrive_count(raw_empty(rr.i), left < SPB && sub + 1 == left ? 1 + SPB - left : 1u);   // a short last block: for its missing steps, too
                }
                rr.step(kGroups / SPB, p.raw_stages);   // four steps on
                rs.step(kGroups, kSlots);
            }
            steps_before += ns;
            blocks_before += x.kb1 - x.kb0;
        }
        finish_shared(Rows<2>());
    } else {
        // ======================= epilogue =======================
        ptx::regs_up<regs_epi(FUSED)>();
        const uint32_t quarter = (uint32_t)warp & 3u, half = (uint32_t)(warp - kFirstEpi) >> 2, ch = quarter * 32 + lane;
        const uint32_t cols = p.rows / 2;   // accumulator columns of this warp
        const bool odd = lane & 1;
        Ring rc{0, 0};
        uint32_t shared = 0;   // pieces of shared tiles so far
        bool told = false;
        uint32_t block = 0;    // staging block that comes next
        bool ok = true;
        auto drained = [&] {   // everything of the accumulator is in registers
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) { if (rank == 0) ptx::mbar_arrive(acc_empty(rc.i)); else ptx::mbar_arrive_remote(acc_empty(rc.i), 0); }
        };
        // A block of 16 rows x 32 channels turns round in shared memory and leaves in 16-byte pieces, 64 contiguous bytes a row; two blocks
        // take turns.
        const uint32_t stage = smem_base + kOffOut + (uint32_t)(warp - kFirstEpi) * out_bytes(FUSED);
        auto block_begin = [&]() -> uint32_t { return stage + block * kOutBytes; };
        // 16 columns of this warp's channels: the sums over all stretches of K
        auto load_sums = [&](uint32_t at, float (&v)[16]) {
            uint32_t r[16];
            ptx::tmem_ld_32x16(at, r);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
#pragma unroll 1
            for (uint32_t i = 1; i < p.stretches; ++i) {
                ptx::tmem_ld_32x16(at + i * p.rows, r);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
            }
        };
        auto put = [&](uint32_t at, uint32_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"((uint16_t)v) : "memory"); };
        auto block_end = [&](uint32_t out, uint32_t col0, uint32_t row0) {
            __syncwarp();
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint32_t piece = i * 32 + lane, row = row0 + piece / 4, col = col0 + piece % 4 * 8;
                uint4 v;
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(out + piece * 16));
                if (row < p.m && col < p.n) *reinterpret_cast<uint4*>(p.c + (size_t)row * p.ldc + col) = v;   // n is a multiple of 8
            }
            block ^= 1u;   // the next but one use of this block comes after the next block's __syncwarp
        };
        while (ok && walk.next<true>(p.deal, worker, x)) {
            uint32_t m0, n0;
            tile_origin(p, rank, x.t, m0, n0);
            const uint32_t nn = n0 + ch, row0 = m0 + half * cols;
            const bool whole = x.kb0 == 0 && x.kb1 == p.deal.blocks;
            const bool inside = n0 + quarter * 32u < p.n;   // some of this warp's channels are
            const float scale = channel_scale(nn), bias = FUSED && p.bias && nn < p.n ? p.bias[nn] : 0.f;
            if (FUSED && p.residual && whole && inside) {   // what will be added comes into L2 meanwhile: a lane takes every 32nd row
                for (uint32_t r = lane; r < cols; r += 32)
                    if (row0 + r < p.m) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.residual + (size_t)(row0 + r) * p.ld_res + ((n0 + quarter * 32u) >> p.gated)));
            }
            if (!warp_wait(acc_full(rc.i), rc.phase, abort_flag)) { give_up(58, x.t, 0); break; }
            ptx::tc_fence_after_sync();
            const uint32_t acc = tmem_base + ((quarter * 32u) << 16) + rc.i * p.rows + half * cols;
            if (!whole) {
                float* part = p.ws + (size_t)(p.deal.slot(worker, x.t) * 2 + rank) * p.rows * kCh + ch;
                const uint32_t valid = min(p.rows, p.m - m0);
                for (uint32_t c0 = 0; c0 < cols; c0 += 16) {
                    uint32_t r[16];
                    ptx::tmem_ld_32x16(acc + c0, r);
                    ptx::tmem_ld_wait();
                    if (c0 + 16 >= cols) drained();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (half * cols + c0 + j < valid) __stcg(part + (size_t)(half * cols + c0 + j) * kCh, __uint_as_float(r[j]));
                }
            } else if (!FUSED && walk.more(p.deal, worker)) {   // another tile waits for the accumulator
                uint32_t o[8][8];   // two rows each
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (16u * i >= cols) break;
                    float v[16];
                    load_sums(acc + 16 * i, v);
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[i][j] = bf16_pair(finished(v[2 * j], scale, 0.f), finished(v[2 * j + 1], scale, 0.f));
                }
                drained();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (16u * i >= cols || !inside || row0 + 16 * i >= p.m) break;
                    const uint32_t out = block_begin();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        put(out + (uint32_t)j * 128u + (uint32_t)lane * 2u, o[i][j]);
                        put(out + (uint32_t)j * 128u + 64u + (uint32_t)lane * 2u, o[i][j] >> 16);
                    }
                    block_end(out, n0 + quarter * 32u, row0 + 16 * i);
                }
            } else if (FUSED && p.gated) {
                // The lanes of a pair hold gate (even) and up (odd) of one output channel.  Of each 16 rows they exchange half: the even lane
                // finishes rows 0 to 7, the odd lane 8 to 15.  The warp's results wait in shared memory until the accumulator has been
                // given back.  A loop, not unrolled: with cold caches its instructions come from memory, too (1024 x 2*2048 x 2048: 53 us
                // with all of it in line, results in registers).
                const uint32_t nout = nn >> 1, my_row = odd ? 8u : 0u, n_out = p.n / 2;
                const uint16_t* res = p.residual + (size_t)(row0 + my_row) * p.ld_res + nout;
                uint32_t next[8];
                auto load_residual = [&](uint32_t c0) {   // -0 adds nothing, to zeros of either sign
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        next[j] = p.residual && nn < p.n && c0 < cols && row0 + c0 + my_row + j < p.m ? res[(size_t)(c0 + j) * p.ld_res] : 0x8000u;
                };
                load_residual(0);
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < cols; c0 += 16) {
                    float v[16], add[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) add[j] = bf16_value(next[j]);
                    load_residual(c0 + 16);
                    load_sums(acc + c0, v);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float lo = finished(v[j], scale, bias), hi = finished(v[j + 8], scale, bias);
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
                        const float o = activated(odd ? other : lo) * (odd ? hi : other) + add[j];
                        put(stage + (c0 + my_row + j) * 32u + ((uint32_t)lane >> 1) * 2u, __bfloat16_as_ushort(__float2bfloat16_rn(o)));
                    }
                }
                drained();
                const uint32_t col = ((n0 + quarter * 32u) >> 1) + (lane & 1u) * 8u;   // 16 bytes a lane, 16 rows a turn
#pragma unroll 1
                for (uint32_t r = (uint32_t)lane >> 1; r < cols; r += 16) {
                    uint4 v;
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(stage + r * 32u + (lane & 1u) * 16u));
                    if (row0 + r >= p.m || col >= n_out) continue;
                    uint16_t* dst = p.c + (size_t)(row0 + r) * p.ldc + col;
                    if (col + 8 <= n_out) *reinterpret_cast<uint4*>(dst) = v;
                    else *reinterpret_cast<uint2*>(dst) = make_uint2(v.x, v.y);   // n_out is a multiple of 4
                }
                __syncwarp();
            } else {
                // The residual of 16 rows is fetched as one, while the 16 before them are finished: a load between two stores into the staging
                // block waits for its answer each time (4096 x 2048 x 2048 int8, not gated: 121 us so).
                const uint16_t* res = p.residual + (size_t)row0 * p.ld_res + nn;
                uint32_t next[16];
                auto load_residual = [&](uint32_t c0) {   // -0 adds nothing, to zeros of either sign
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) next[j] = p.residual && nn < p.n && c0 < cols && row0 + c0 + j < p.m ? res[(size_t)(c0 + j) * p.ld_res] : 0x8000u;
                };
                if (FUSED) load_residual(0);
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < cols; c0 += 16) {
                    float sums[16], add[16];
                    if (FUSED) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) add[j] = bf16_value(next[j]);
                        load_residual(c0 + 16);
                    }
                    load_sums(acc + c0, sums);
                    if (c0 + 16 >= cols) drained();
                    if (!inside || row0 + c0 >= p.m) continue;
                    const uint32_t out = block_begin();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float v = finished(sums[j], scale, bias);
                        if (FUSED) v = activated(v) + add[j];
                        put(out + (uint32_t)j * 64u + (uint32_t)lane * 2u, __bfloat16_as_ushort(__float2bfloat16_rn(v)));
                    }
                    block_end(out, n0 + quarter * 32u, row0 + c0);
                }
            }
            rc.step(1, p.accs);
            if (!whole) {
                // published; the tile is finished at the end, see finish_shared
                __threadfence();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive(bar_stored);
                    if (warp == kFirstEpi) {
                        if (wait_or_abort(bar_stored, shared & 1u, abort_flag)) {
                            __threadfence();
                            atomicAdd(p.counters + (2 * x.t + rank) * kTileWords, 1u);
                            misc[4 + shared] = x.t;   // a pair holds parts of two tiles at most
                        } else {
                            give_up(59, x.t, 0);
                        }
                    }
                }
                ++shared;
            }
            // nothing shared comes after this piece: the converters may finish what is
            if (warp == kFirstEpi && lane == 0 && !told && walk.u == walk.u_end) { misc[3] = shared; ptx::mbar_arrive(bar_finish); }
            told |= walk.u == walk.u_end;
        }
        if (!told && warp == kFirstEpi && lane == 0) { misc[3] = 0u; ptx::mbar_arrive(bar_finish); }   // after an abort
        finish_shared(Rows<4>());
    }

    // ---- teardown: every thread gets here, also after an abort; neither CTA leaves while the other may read its shared memory or arrive there ----
    ptx::tc_fence_before_sync();
    __syncwarp();
    if (warp == 0) ptx::cluster_wait();   // of the arrival at the start
    ptx::cluster_arrive();
    ptx::cluster_wait();
    if (warp == 2) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

template <int BITS, bool GROUPED, int KS, bool FUSED>
int launch_cfg(const CUtensorMap& ta, const CUtensorMap& tw, const PairParams& p, DeviceCtx* ctx, cudaStream_t s) {
    auto kern = pair_kernel<BITS, GROUPED, KS, FUSED>;
    static DeviceOnce attr_set;  // per template instance
    if (!attr_set.done(ctx->device)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e != cudaSuccess) return cuda_fail(e);
        attr_set.mark(ctx->device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * p.deal.grid); cfg.blockDim = dim3(kThreads); cfg.stream = s;
    cfg.dynamicSmemBytes = 1024 + off_raw(FUSED) + p.raw_stages * kRawBytes + slots(KS) * p.rows * KS;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tw, p);
    count_launch();
    count_pair_launch();
    return e == cudaSuccess ? AFB_OK : cuda_fail(e);
}

// Rows per tile, and whether the tiles that do not fill whole waves are shared: the cheapest by a count of cycles.  Per step of 128 k
// 4 per activation row (the tensor cores) or 820 (the issuing warp; of 64 k 700); per tile 3300 until its only accumulator has been drained
// (up to 128 rows there are two); for sharing, that is partial sums written, read and added, 120 per row (2048 x 11008 x 4096 int8 with
// 256 rows: 131 us shared, 119 not; 128 x 28672 x 8192 int4 group-128 with 128 rows: 62 and 70) and 1200 per pair that shares a tile: a
// warp adds their sums one after the other (K = 8192 int8, 65 rows: 1 tile over a wave, 64 pairs on it, 116 us shared and 71 not; 3 tiles
// 78 and 72; 10 tiles 65 and 71).
// useful: the share of the pairs' cycles that goes into steps.
struct Plan { uint32_t rows, waves; bool shared; double cycles, useful; };
Plan plan(const afb_gemm_args& a, uint32_t ks, uint32_t pairs) {
    Plan best{};
    const uint32_t n_tiles = (a.n + 2 * kCh - 1) / (2 * kCh), steps = a.k / ks, blocks = (uint32_t)(((uint64_t)a.k * a.b_bits / 8 + 127) / 128);
    const uint32_t fewest = (a.m + 255) / 256, most = fewest + 8 < (a.m + 63) / 64 ? fewest + 8 : (a.m + 63) / 64;
    for (uint32_t row_tiles = fewest; row_tiles <= most; ++row_tiles) {
        const uint32_t rows = ((a.m + row_tiles - 1) / row_tiles + 31) / 32 * 32;   // for two SMs in steps of 32
        const uint32_t tiles = (a.m + rows - 1) / rows * n_tiles, waves = tiles / pairs, rest = tiles % pairs;
        const double hand_off = ks == 128 ? 820. : 700., mma = rows * (ks / 32.);
        const double work = steps * (mma > hand_off ? mma : hand_off), tile = work + (rows > 128 ? 3300. : 0.);
        // (Short of a wave, whole tiles of more than 128 rows add up all of K in one accumulator; there sharing stays as cheap as its rows.)
        const double sharers = !rest || (!waves && rows > 128) ? 0. : (double)pairs / rest < blocks ? (double)pairs / rest : blocks;
        const double whole = (waves + (rest ? 1 : 0)) * tile, split = waves * tile + work * rest / pairs + 120. * rows + 1200. * sharers;
        const bool shared = rest && split < whole;
        const double cycles = (shared ? split : whole) + 25. * rows;   // ... and the last tile's way out
        if (!best.rows || cycles < best.cycles) best = Plan{rows, waves, shared, cycles, tiles * work / pairs / cycles};
    }
    return best;
}

// Where this form is the faster one.  The lines are drawn through the times of this form and of the one that would take the call otherwise, on
// one B200, caches cold: 21700 sizes, K from 512 to 28672, N from 1024 to 40960, 65 to 4096 rows, int8 and int4 per channel and in groups of
// 128 and 64.  Of the 13400 that this form takes it is the slower one by more than 6 % at 6 (by 10 % at most) and 1.23 times as fast on
// average (with nothing to write back in L2 before: at 1 in 200, by 13 % at most, and 1.20).  Each line names sizes on its two sides (us, the other form / this one).
// Fused (9 matrices and 15 more with K of 512, K = 64 modulo 128 or few channels; 1 to 4096 rows):
//   1000 x 2*11008 x 4096 int8: 213 / 156;  1024 x 2*2048 x 2048: 37 / 31;  16 x 2*4096 x 11008 int4 group-128: 2.5 times;  but
//   64 x 2*2048 x 2048 int8: 28 / 33 (65 rows: 30 / 27);  128 x 2*4096 x 4160 int8, in steps of 64 k: 40 / 49, 2*5504 x 2112: 0.92
bool is_faster(const afb_gemm_args& a, const Plan& x, uint32_t ks, uint32_t sms, const afb_fused_args* fused) {
    const double weights = (double)a.n * a.k;
    const uint32_t pairs = sms / 2, n_tiles = (a.n + 2 * kCh - 1) / (2 * kCh), tiles = (a.m + x.rows - 1) / x.rows * n_tiles;
    if (fused) {
        if (a.group_size) return true;
        if (fused->gated && ks == 64 && a.m > 64 && a.m <= 128 && a.k >= 2048 && n_tiles * 2 <= pairs) return false;
        return a.m > 64 || weights >= 16e6;
    }
    if (a.m <= 64) return false;
    // All tiles shared: the other forms cut the same work into smaller pieces (128 x 8192 x 8192 int8: 36 / 49; 333 x 4096 x 11008: 51 / 57).
    if (x.shared && tiles < pairs) return false;
    if (a.group_size && a.b_bits == 8 && a.m <= 128) return false;   // 65 x 19200 x 8192 in groups of 64: 1.81; 72 x 20000 x 2048: 27 / 35
    // The streaming form shares whatever is left over a wave evenly and has less to hand off per row; what decides is how much of this form's
    // time is steps: 128 x 22528 x 8192 int8 (0.72) 60 / 66, 24576 (0.75) 69 / 67;  192 x 19200 x 8192 (0.46) 1.20, 160 x 20736 x 8192 (0.59) 74 / 72.
    if (a.m <= 256 && stream_is_faster(a, sms)) {
        if (x.shared && a.b_bits == 8 && a.m <= 96) return false;   // 65 x 28672 x 8192: 66 / 68, 40960: 96 / 100
        const double least = ks == 64 ? (a.m <= 128 ? 0.8 : 0.7) : (a.m <= 128 ? 0.74 : 0.5);
        return !x.waves || x.useful >= least;   // 128 x 14336 x 3072 int4 group-128, one wave: 0.80
    }
    // Short rows leave too little to gain for the longer start and way out: K = 512: 1024 x 4096 int8: 15 / 20; 2048 x 28672: 1.33; K = 896: 1.03 on
    // average from 513 rows on; groups of 64: 1.02 and 0.87.  With steps of 64 k and without groups up to K = 2047: 1088: 1.03, 1856: 0.98.
    // Up to 128 rows the others need two waves from 19200 channels on: 0.65 to 0.8.
    if (a.k < (a.group_size % 128 ? 768u : 1024u) || (ks == 64 && !a.group_size && a.k < 2048)) return !a.group_size && a.m <= 128 && n_tiles > pairs;
    if (ks == 64) {   // twice the hand-offs
        if (a.m > 256 && a.m <= 384) return weights < 40e6;   // 300 x 28672 x 4160 int8: 86 / 94; 28672 x 4096 in groups of 64: 1.03; 8192 x 4096: 0.68
        if (a.m <= 128) {
            // 128 x 8192 x 2112 int8: 1.12, 19200: 44 / 37;  groups of 64: 65 x 28672 x 2304: 1.12, 11008 x 2048: 0.82, 4096 x 2048 (32 tiles): 20 / 27
            if (!a.group_size) return n_tiles > pairs;
            return a.k > 1536 && tiles * 2 > pairs && (n_tiles <= pairs || a.k >= 4096);
        }
    }
    if (a.m <= 128 && a.k >= 3072 && tiles * 8 <= pairs) return false;         // 65 x 1024 x 3072 int4: 1.10
    if (a.m <= 256 && a.k <= 1536 && x.rows >= 224) return false;              // 256 x 11008 x 1280: 1.10
    if (!a.group_size && a.m > 192 && a.m <= 256 && a.k >= 3072 && x.useful < 0.5) return false;   // 256 x 19200 x 8192: 89 / 101
    if (a.group_size % 128) return true;
    // The form with tiles of 256 x 128 (prefill_ts.cu) starts and ends sooner.  Where those fill one or two waves well, that decides for short K.
    const uint32_t there = (a.m + 255) / 256 * ((a.n + kCh - 1) / kCh);
    if (there <= sms / 2 || there > 2 * sms) return true;
    const double full = (double)a.m * a.n / (256. * kCh * sms);   // waves of it, without padding
    if (there > sms) return a.k >= 1536 || full < 1.5;            // 2048 x 4096 x 1024 int8 (1.73): 27 / 29, 512 x 14336 (1.51): 27 / 30;  1280 x 5504 (1.45): 0.86
    if (a.k < 1536) return full <= 0.5 && (a.group_size || a.m > 256);   // 1024 x 4096 x 1024 (0.86): 18 / 22, 384 x 7168 (0.57): 1.0, 512 x 4096 (0.43): 0.76; 128 x 14336 int4: 1.08, 192 x 11008: 1.0
    if (a.group_size || a.m <= 128 || a.k > 4096) return true;
    if (x.rows == 256 || (a.m <= 256 && x.rows >= 224)) return false;   // 1024 x 4096 x 4096: 35 / 37, 512 x 8192 x 3072: 1.02;  224 x 14336 x 2048: 1.01
    // K = 1536: 1280 x 3072 (0.81) 1.08, 384 x 7168 (0.57) 0.97;  K = 2048: 450 x 7168 (0.67) 1.06, 777 x 4096 (0.66) 0.99, K = 2112: 450 (0.38) 1.03, 640 (0.54) 0.99
    return a.k >= 3072 || full <= (a.k < 2048 ? 0.58 : ks == 64 ? 0.6 : 0.66);
}

// A tuning variable that asks for one of the variant's other forms, or for a shape of theirs.
bool other_form_asked() {
    for (const char* name : {"AFB_STREAM", "AFB_PREFILL_IMPL", "AFB_PREFILL_TILE_STORE", "AFB_PREFILL_SPLIT_TAIL", "AFB_PREFILL_GROUP_M"})
        if (getenv(name)) return true;
    return false;
}

}  // namespace

int pair_if_faster(const afb_gemm_args& a, DeviceCtx* ctx, cudaStream_t s, const afb_fused_args* fused, bool* done) {
    *done = false;
    const char* env = getenv("AFB_PAIR");
    const int forced = env ? atoi(env) : -1;
    if (forced == 0 || a.flags & (AFB_FLAG_C_F32 | AFB_FLAG_PREFILL_SMEM_B | AFB_FLAG_PREFILL_TMEM_A)) return AFB_OK;
    if (forced < 0 && !fused && a.m <= 64) return AFB_OK;   // is_faster says so, too: without the plan
    if (a.group_size && ((a.flags & AFB_FLAG_GROUP_EXACT) || a.group_size % kSlab || (a.group_size & (a.group_size - 1)))) return AFB_OK;
    const uint32_t pairs = (uint32_t)ctx->sm_count / 2;
    const uint32_t ks = a.k % 128 == 0 && a.group_size % 128 == 0 ? 128 : 64, spb = (a.b_bits == 8 ? 128 : 256) / ks;
    Plan chosen = plan(a, ks, pairs);
    if (forced < 0 && (!is_faster(a, chosen, ks, (uint32_t)ctx->sm_count, fused) || other_form_asked())) return AFB_OK;
    if (const char* e = getenv("AFB_PAIR_ROWS")) {   // tuning aids: the most rows per tile, shared tiles or none
        const uint32_t most = (uint32_t)atoi(e), t = most >= 32 && most <= 256 ? (a.m + most - 1) / most : 0;
        if (t) chosen.rows = ((a.m + t - 1) / t + 31) / 32 * 32;
        if (chosen.rows > 256) chosen.rows = 256;
    }
    if (const char* e = getenv("AFB_PAIR_SHARE")) chosen.shared = atoi(e) != 0;
    PairParams p{};
    p.c = reinterpret_cast<uint16_t*>(a.ptr_c);
    p.scale = a.ptr_scale;
    p.zero = reinterpret_cast<const uint8_t*>(a.ptr_zero);
    p.m = a.m; p.n = a.n; p.k = a.k; p.ldc = a.ldc;
    p.enc = a.b_encoding; p.scale_dtype = a.scale_dtype;
    p.packed = a.b_layout == AFB_LAYOUT_COL_PACKED ? 1u : 0u;
    p.rows = chosen.rows;
    p.m_tiles = (a.m + p.rows - 1) / p.rows;
    p.n_tiles = (a.n + 2 * kCh - 1) / (2 * kCh);
    p.group_m = pick_group_m(a, p.m_tiles, p.n_tiles, p.rows, pairs, 2 * kCh);
    p.steps = a.k / ks;
    while (a.group_size && ks << p.group_shift < a.group_size) ++p.group_shift;
    const bool one_each = !chosen.shared && p.m_tiles * p.n_tiles <= pairs;
    p.stretches = one_each && p.steps >= 8 ? (p.rows <= 64 ? 4 : p.rows <= 128 ? 2 : 1) : 1;
    p.accs = p.rows <= 128 && p.stretches == 1 ? 2 : 1;
    const uint32_t act_bytes = p.rows * ks, kSlots = slots(ks);   // of one CTA and step
    p.raw_stages = (ring_budget(fused != nullptr) - kSlots * act_bytes) / kRawBytes;
    if (p.raw_stages > (uint32_t)kMaxRaw) p.raw_stages = kMaxRaw;
    // the parity waits of the converters: see stream.cu
    p.slot_first = p.raw_stages >= kGroups + kSlots ? 0u : 1u;
    if (p.raw_stages < kSlots) return AFB_OK;
    p.deal = chosen.shared ? deal_tiles(p.m_tiles * p.n_tiles, (p.steps + spb - 1) / spb, pairs, 0) : deal_whole(p.m_tiles * p.n_tiles, (p.steps + spb - 1) / spb, pairs);
    if (!p.deal.fits()) return AFB_OK;
    if (p.deal.shared_tiles) {
        if (p.deal.shared_tiles * 2 * kTileWords > ctx->stream_counter_count) return AFB_OK;
        if (!stream_workspace(ctx, s, (size_t)4 * p.deal.grid * p.rows * kCh * sizeof(float), &p.ws, &p.counters)) return AFB_OK;   // the caller's other forms
    }
    p.status = ctx->status;
    if (fused) {
        p.bias = reinterpret_cast<const float*>(fused->ptr_bias);
        p.residual = reinterpret_cast<const uint16_t*>(fused->ptr_residual);
        p.ld_res = fused->ld_residual;
        p.gated = fused->gated;
        p.act = fused->activation;
    }
    *done = true;
    CUtensorMap ta, tw;
    int rc = tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.ptr_a, a.k, a.m, (uint64_t)a.lda * 2, kSlab, p.rows / 2, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.ptr_b, (uint64_t)a.k * a.b_bits / 8, a.n, (uint64_t)a.ldb * a.b_bits / 8, 128, kCh,
                 CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
#define AFB_PAIR_KS(B, G, F) (ks == 128 ? launch_cfg<B, G, 128, F>(ta, tw, p, ctx, s) : launch_cfg<B, G, 64, F>(ta, tw, p, ctx, s))
#define AFB_PAIR_LAUNCH(B, G) (fused ? AFB_PAIR_KS(B, G, true) : AFB_PAIR_KS(B, G, false))
    if (a.b_bits == 8) return a.group_size ? AFB_PAIR_LAUNCH(8, true) : AFB_PAIR_LAUNCH(8, false);
    return a.group_size ? AFB_PAIR_LAUNCH(4, true) : AFB_PAIR_LAUNCH(4, false);
#undef AFB_PAIR_LAUNCH
#undef AFB_PAIR_KS
}

}  // namespace afb
