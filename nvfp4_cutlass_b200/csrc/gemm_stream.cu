// Grouped dual-NVFP4 GEMM for a few tokens per expert over activations that are already quantised: the decode orientation
// (128 weight rows on the MMA M axis, a token tile with its two passes stacked on the N axis, see gemm_swap.cu) with
// nothing in the main loop but loads and MMAs.
//
// gemm_swap.cu runs Algorithm 1 on the token tile once per 128 weight rows; on a layer with many weight rows that is the
// same arithmetic dozens of times, and its BF16 tiles take the shared memory that weights in flight need.  Here the codes
// come from a pass of their own (stream_quantize_kernel) or, in the expert-parallel layer, from the dispatch.  The scale
// factors stay in rows, (rows, passes, K / 16) bytes: the scale warps need one row per lane, so that a box of them is read
// back the way it landed and no layout of tensor-memory atoms is needed.
//
// Bound by HBM: every active expert's weights once, 36 KB per K block of 512 and CTA.  One ring carries weights, codes and
// scales of a K block, five positions deep for 16 tokens (four in gemm_swap.cu), four for 32.
// Decode of 64 tokens over 256 experts, N = 4096, K = 7168 (3.67 GB of live weights): 582 us = 6.3 TB/s, gemm_swap.cu 675; an
// expert layer of 256 tokens (128 experts, 4096 / 1536): 328 us, 443 with the 128-row kernels of gemm_split.cu.
#include <cuda_bf16.h>

#include "gemm_common.cuh"
#include "host_common.hpp"
#include "launchers.hpp"
#include "transform.cuh"

namespace nvfp4 {
namespace {

using gemm::Ring;

constexpr uint32_t BW = 128;                         // weight rows per tile
constexpr uint32_t kWarpTma = 0, kWarpMma = 1, kWarpEpi0 = 4, kNumEpiWarps = 4, kWarpSf0 = 8, kNumSfWarps = 4;
constexpr uint32_t kThreads = (kWarpSf0 + kNumSfWarps) * 32;                 // 384
constexpr uint32_t kSmemBudget = 232448 - 1024;
constexpr uint32_t kStageRow = 272;                  // a token's 64 gate and 64 up values, padded against bank conflicts

template <uint32_t T, uint32_t BK, bool kResidual, bool kSwigluOut>
struct Cfg {
    static_assert(BK == 256 || BK == 512, "K block: one or two 128-byte-swizzled sub-tiles");
    static constexpr uint32_t kPass = kResidual ? 2 : 1, kAtoms = BK / 64, kSubs = BK / 256;
    static constexpr uint32_t kRowsP = kPass * T;
    static constexpr uint32_t kSubW = BW * 128, kSubP = kRowsP * 128;
    static constexpr uint32_t kSlotW = kSubs * kSubW, kSlotP = kSubs * kSubP, kSlotSFW = kAtoms * 512, kSlotSFT = kRowsP * kAtoms * 4;
    static constexpr uint32_t kSlot = kSlotW + kSlotP + kSlotSFW + kSlotSFT;
    static constexpr uint32_t kStage = kSwigluOut ? T * kStageRow : 0;
    static constexpr uint32_t kDepthRaw = (kSmemBudget - kStage - 512) / kSlot, kDepth = kDepthRaw > 10 ? 10 : kDepthRaw;
    static_assert(kDepth >= 3, "ring too shallow");
    static constexpr uint32_t kOffW = 0, kOffP = kOffW + kDepth * kSlotW, kOffSFW = kOffP + kDepth * kSlotP;
    static constexpr uint32_t kOffSFT = kOffSFW + kDepth * kSlotSFW, kOffStage = kOffSFT + kDepth * kSlotSFT;
    static constexpr uint32_t kOffBars = kOffStage + kStage;
    static constexpr uint32_t kSmemAlloc = kOffBars + (2 * kDepth + 6) * 8 + 16 + 1024;
    static_assert(kSlotP % 1024 == 0 && kSubP % 1024 == 0 && kSlotSFT % 128 == 0 && kOffStage % 16 == 0 && kOffBars % 8 == 0, "alignment");
    static_assert(kSmemAlloc <= 232448, "shared memory budget");
    static constexpr uint32_t kAccStride = kRowsP < 32 ? 32 : kRowsP;
    static constexpr uint32_t kColSF = 2 * kAccStride, kSfBufCols = 8 * kAtoms, kSfW = 0, kSfT = 4 * kAtoms;
    static constexpr uint32_t kColsUsed = kColSF + 2 * kSfBufCols;
    static constexpr uint32_t kTmemCols = kColsUsed <= 128 ? 128 : (kColsUsed <= 256 ? 256 : 512);
    static constexpr uint32_t kSBO = 8 * 128;
};

struct Params {
    const float* gw;
    const int32_t* layout;     // contiguous: expert of every row; masked: real rows of every group
    __nv_bfloat16* d;
    int64_t ldd;
    uint32_t m, n, k, groups, max_m;
    gemm::Family family;       // masked
    // SwiGLU-quantised output (gate/up-interleaved weight rows): the next GEMM's codes (rows, n / 4) and scale rows
    uint8_t* out_a0;
    uint8_t* out_a1;
    uint8_t* out_sf;
    int32_t* status;
};

template <uint32_t T, uint32_t BK, bool kResidual, bool kMasked, bool kSwigluOut>
__global__ void __launch_bounds__(kThreads, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tm_a0, const __grid_constant__ CUtensorMap tm_a1,
                   const __grid_constant__ CUtensorMap tm_sft, const __grid_constant__ CUtensorMap tm_w,
                   const __grid_constant__ CUtensorMap tm_sfw, const Params p)
{
    using C = Cfg<T, BK, kResidual, kSwigluOut>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem - ptx::smem_u32(smem_raw));

    uint64_t* full = reinterpret_cast<uint64_t*>(smem_gen + C::kOffBars);
    uint64_t* empty = full + C::kDepth;
    uint64_t* sf_full = empty + C::kDepth;           // [2]: scales of a K block are in tensor memory
    uint64_t* tmem_full = sf_full + 2;               // [2]
    uint64_t* tmem_empty = tmem_full + 2;            // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const uint32_t warp = ptx::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < C::kDepth; ++i) { ptx::mbar_init(full + i, 1); ptx::mbar_init(empty + i, 1); }
        for (uint32_t i = 0; i < 2; ++i) {
            ptx::mbar_init(sf_full + i, kNumSfWarps);
            ptx::mbar_init(tmem_full + i, 1);
            ptx::mbar_init(tmem_empty + i, kNumEpiWarps);
        }
        *abort_flag = 0;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tm_a0);
        if constexpr (kResidual) ptx::prefetch_tensormap(&tm_a1);
        ptx::prefetch_tensormap(&tm_sft);
        ptx::prefetch_tensormap(&tm_w);
        ptx::prefetch_tensormap(&tm_sfw);
    }
    if (warp == kWarpMma) ptx::tmem_alloc<C::kTmemCols>(tmem_slot);
    ptx::tcgen05_fence_before_sync();
    __syncthreads();
    ptx::tcgen05_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    ptx::grid_dependency_wait();

    // contiguous: all weight tiles of a token tile are neighbours; masked: the token tiles of an expert are, per weight tile
    const uint32_t num_kb = p.k / BK;
    gemm::TileWalker<T, kMasked> walk(p.layout, p.m, p.n, BW, kMasked ? 8 : 1, p.groups, p.max_m);
    // this family is the one that is expected to stay: it leaves by finding no tile, its prologue has run ahead
    if constexpr (kMasked)
        if (p.family.leaves(p.layout, p.groups, p.max_m)) walk.groups = 0;
    gemm::Tile t;
    bool ok = true;
    ptx::ProbeAcc pa;
    auto give_up = [&](uint32_t code) {
        *abort_flag = 1;
        if (p.status != nullptr) atomicOr(p.status, static_cast<int32_t>(code));
        ok = false;
    };

    if (warp == kWarpTma) {
        {
            const uint32_t issue = ptx::elect_one();
            Ring r;
            const uint64_t stream_once = ptx::l2_policy_evict_first();
            for (uint32_t tile = blockIdx.x; ok && ptx::uniform(walk.next(tile, t)) != 0; tile += gridDim.x) {
                const uint32_t e = ptx::uniform(static_cast<uint32_t>(t.expert)), n_blk = ptx::uniform(t.n_blk), row0 = ptx::uniform(t.row0);
                const uint32_t w_row = e * p.n + n_blk * BW;
                for (uint32_t kb = 0; kb < num_kb; ++kb) {
                    if (!ptx::all_lanes(ptx::mbar_wait(empty + r.slot, r.phase ^ 1, abort_flag, pa, 0))) { give_up(1); break; }
                    uint64_t* bar = full + r.slot;
                    ptx::mbar_arrive_expect_tx(bar, C::kSlot, issue);
                    uint8_t* w = smem_gen + C::kOffW + r.slot * C::kSlotW;
                    uint8_t* a = smem_gen + C::kOffP + r.slot * C::kSlotP;
                    uint8_t* sft = smem_gen + C::kOffSFT + r.slot * C::kSlotSFT;
                    ptx::tma_load_2d_hint(smem_gen + C::kOffSFW + r.slot * C::kSlotSFW, &tm_sfw, bar, n_blk * BW,
                                          e * (p.k / 64) + kb * C::kAtoms, stream_once, issue);
#pragma unroll
                    for (uint32_t sub = 0; sub < C::kSubs; ++sub) {
                        const uint32_t col = kb * (BK / 2) + sub * 128;
                        ptx::tma_load_2d_hint(w + sub * C::kSubW, &tm_w, bar, col, w_row, stream_once, issue);
                        ptx::tma_load_2d(a + sub * C::kSubP, &tm_a0, bar, col, row0, issue);
                        if constexpr (kResidual) ptx::tma_load_2d(a + sub * C::kSubP + T * 128, &tm_a1, bar, col, row0, issue);
                    }
#pragma unroll
                    for (uint32_t pass = 0; pass < C::kPass; ++pass)
                        ptx::tma_load_2d(sft + pass * T * C::kAtoms * 4, &tm_sft, bar, pass * (p.k / 64) + kb * C::kAtoms, row0, issue);
                    r.advance<C::kDepth>();
                }
            }
            ptx::grid_launch_dependents();          // the last loads are on their way: the next kernel may start its prologue
            if (ok && !gemm::drain_ring<C::kDepth>(r, [&](uint32_t i, uint32_t parity) {
                    return ptx::all_lanes(ptx::mbar_wait(empty + i, parity, abort_flag, pa, 0)); })) give_up(1);
        }
    } else if (warp == kWarpMma) {
        const uint32_t issue = ptx::elect_one();
        Ring r;
        uint32_t it = 0, cnt = 0;
        constexpr uint32_t idesc = ptx::make_idesc_nvf4(BW, C::kRowsP);
        for (uint32_t tile = blockIdx.x; ok && ptx::uniform(walk.next(tile, t)) != 0; tile += gridDim.x, ++it) {
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            if (!ptx::all_lanes(ptx::mbar_wait(tmem_empty + acc, acc_phase ^ 1, abort_flag, pa, 0))) { give_up(1); break; }
            ptx::tcgen05_fence_after_sync();
            const uint32_t tmem_acc = tmem_base + acc * C::kAccStride;
            for (uint32_t kb = 0; kb < num_kb; ++kb, ++cnt) {
                const uint32_t buf = cnt & 1u;
                if (!ptx::all_lanes(ptx::mbar_wait(full + r.slot, r.phase, abort_flag, pa, 1) &&
                                    ptx::mbar_wait(sf_full + buf, (cnt >> 1) & 1u, abort_flag, pa, 2))) { give_up(1); break; }
                ptx::tcgen05_fence_after_sync();
                const uint32_t w = smem + C::kOffW + r.slot * C::kSlotW, a = smem + C::kOffP + r.slot * C::kSlotP;
                const uint32_t sf = tmem_base + C::kColSF + buf * C::kSfBufCols;
#pragma unroll
                for (uint32_t i = 0; i < C::kAtoms; ++i)
                    ptx::tcgen05_mma_nvf4(tmem_acc, ptx::make_smem_desc(w + (i / 4) * C::kSubW + (i % 4) * 32, C::kSBO, ptx::kSwizzle128B),
                                          ptx::make_smem_desc(a + (i / 4) * C::kSubP + (i % 4) * 32, C::kSBO, ptx::kSwizzle128B), idesc,
                                          sf + C::kSfW + 4 * i, sf + C::kSfT + 4 * i, (kb | i) != 0 ? 1u : 0u, issue);
                ptx::tcgen05_commit(empty + r.slot, issue);       // frees the ring position and the block's scale columns
                if (kb == num_kb - 1) ptx::tcgen05_commit(tmem_full + acc, issue);
                r.advance<C::kDepth>();
            }
        }
    } else if (warp >= kWarpSf0) {
        // scale warps, one per 32-lane quadrant of tensor memory: lane i puts the scale words of rows i, i + 32, ... of an
        // atom into consecutive columns.  Two column buffers alternate; one is rewritten once the MMAs of two K blocks
        // earlier have retired.
        const uint32_t quad = warp & 3;
        Ring r;
        uint32_t cnt = 0;
        for (uint32_t tile = blockIdx.x; ok && walk.next(tile, t); tile += gridDim.x) {
            for (uint32_t kb = 0; kb < num_kb; ++kb, ++cnt) {
                const uint32_t buf = cnt & 1u;
                const uint32_t sf = tmem_base + ((quad * 32) << 16) + C::kColSF + buf * C::kSfBufCols;
                if (!ptx::all_lanes(ptx::mbar_wait(full + r.slot, r.phase, abort_flag, pa, 0) &&
                                    (cnt < 2 || ptx::mbar_wait(empty + (cnt - 2) % C::kDepth, ((cnt - 2) / C::kDepth) & 1u, abort_flag,
                                                               pa, 1)))) {
                    give_up(1);
                    break;
                }
                ptx::tcgen05_fence_after_sync();
                const uint32_t sfw = smem + C::kOffSFW + r.slot * C::kSlotSFW + lane * 4;
                uint32_t v[4 * C::kAtoms];
#pragma unroll
                for (uint32_t i = 0; i < C::kAtoms; ++i)
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) v[4 * i + j] = ptx::lds32(sfw + i * 512 + j * 128);
                ptx::tmem_st_32x32b(sf + C::kSfW, v);
                constexpr uint32_t kGroups = (C::kRowsP + 31) / 32;          // 32-row groups of the stacked tile
                const uint32_t sft = smem + C::kOffSFT + r.slot * C::kSlotSFT;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    if (j >= kGroups) {
#pragma unroll
                        for (uint32_t i = 0; i < C::kAtoms; ++i) v[4 * i + j] = 0;
                        continue;
                    }
                    const uint32_t row = (32 * j + lane) % C::kRowsP;
#pragma unroll
                    for (uint32_t i = 0; i < C::kAtoms; i += 4) {
                        const uint4 q = ptx::lds128(sft + (row * C::kAtoms + i) * 4);
                        v[4 * i + j] = q.x; v[4 * i + 4 + j] = q.y; v[4 * i + 8 + j] = q.z; v[4 * i + 12 + j] = q.w;
                    }
                }
                ptx::tmem_st_32x32b(sf + C::kSfT, v);
                ptx::tmem_st_wait();
                ptx::tcgen05_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(sf_full + buf);
                r.advance<C::kDepth>();
            }
        }
    } else if (warp >= kWarpEpi0 && warp < kWarpEpi0 + kNumEpiWarps) {
        // accumulator lane = weight row, column = token (pass 0, then pass 1)
        const uint32_t quad = warp & 3;
        uint32_t it = 0;
        for (uint32_t tile = blockIdx.x; ok && walk.next(tile, t); tile += gridDim.x, ++it) {
            const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
            const float g = __ldg(p.gw + t.expert);
            bool mine = ptx::all_lanes(ptx::mbar_wait(tmem_full + acc, acc_phase, abort_flag, pa, 0));
            // the four warps stay together (they share barriers below): one that gave up takes the others along
            if constexpr (kSwigluOut) {
                uint32_t all;
                asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.aligned.pred q, 1, 128, p;\n selp.u32 %0, 1, 0, q;\n}"
                             : "=r"(all) : "r"(mine ? 1u : 0u) : "memory");
                mine = all != 0;
            }
            if (!mine) { give_up(1); break; }
            ptx::tcgen05_fence_after_sync();
            const uint32_t taddr = tmem_base + ((quad * 32) << 16) + acc * C::kAccStride;
            __nv_bfloat16* dcol = p.d + static_cast<int64_t>(t.row0) * p.ldd + t.n_blk * BW + quad * 32 + lane;
            // interleaved weight rows: quadrants 0 and 2 are gate rows, 1 and 3 the matching up rows
            const uint32_t cell = smem + C::kOffStage + (quad & 1u) * 128 + ((quad >> 1) * 32 + lane) * 2;
#pragma unroll 1
            for (uint32_t c = 0; c < T; c += 16) {
                uint32_t v[16], r[16];
                ptx::tmem_ld_32x32b_x16(taddr + c, v);
                if constexpr (kResidual) ptx::tmem_ld_32x32b_x16(taddr + T + c, r);
                ptx::tmem_ld_wait();
                if (c + 16 == T) {
                    ptx::tcgen05_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(tmem_empty + acc);
                }
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i) {
                    float x = __uint_as_float(v[i]);
                    if constexpr (kResidual) x += __uint_as_float(r[i]);
                    const __nv_bfloat16 y = __float2bfloat16_rn(x * g);
                    if constexpr (kSwigluOut) ptx::sts16(cell + (c + i) * kStageRow, __bfloat16_as_ushort(y));
                    else dcol[static_cast<int64_t>(c + i) * p.ldd] = y;
                }
            }
            if constexpr (kSwigluOut) {
                // a thread per token and 16-block of the tile's 64 products (one K atom of the down-projection); arithmetic and
                // roundings of the stand-alone SwiGLU kernel
                asm volatile("barrier.cta.sync.aligned 1, 128;" ::: "memory");
                const uint32_t k_out = p.n / 2, u = threadIdx.x - kWarpEpi0 * 32, blk = u % 4;
#pragma unroll 1
                for (uint32_t token = u / 4; token < T; token += 32) {
                    const uint32_t at = smem + C::kOffStage + token * kStageRow + blk * 32;
                    const uint4 g0 = ptx::lds128(at), g1 = ptx::lds128(at + 16), u0 = ptx::lds128(at + 128), u1 = ptx::lds128(at + 144);
                    const uint32_t gate[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
                    const uint32_t up[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[i]));
                        const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&up[i]));
                        const __nv_bfloat162 pr = __floats2bfloat162_rn(gf.x / (1.0f + __expf(-gf.x)) * uf.x, gf.y / (1.0f + __expf(-gf.y)) * uf.y);
                        w[i] = *reinterpret_cast<const uint32_t*>(&pr);
                    }
                    xform::Block16 out;
                    xform::decompose_block16<true, 0>(w, out);
                    const uint64_t row = t.row0 + token, code = row * (k_out / 2) + t.n_blk * 32 + blk * 8;
                    *reinterpret_cast<uint2*>(p.out_a0 + code) = make_uint2(out.q0[0], out.q0[1]);
                    *reinterpret_cast<uint2*>(p.out_a1 + code) = make_uint2(out.q1[0], out.q1[1]);
                    uint32_t s0 = out.s0 << (8 * blk), s1 = out.s1 << (8 * blk);
                    s0 |= __shfl_xor_sync(0xffffffffu, s0, 1); s0 |= __shfl_xor_sync(0xffffffffu, s0, 2);
                    s1 |= __shfl_xor_sync(0xffffffffu, s1, 1); s1 |= __shfl_xor_sync(0xffffffffu, s1, 2);
                    uint8_t* sf = p.out_sf + row * (k_out / 8) + t.n_blk * 4;
                    if (blk == 0) *reinterpret_cast<uint32_t*>(sf) = s0;
                    if (blk == 1) *reinterpret_cast<uint32_t*>(sf + k_out / 16) = s1;
                }
                asm volatile("barrier.cta.sync.aligned 1, 128;" ::: "memory");       // the stage may be written again
            }
        }
    }

    ptx::tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == kWarpMma) {
        ptx::tcgen05_fence_after_sync();
        ptx::tmem_dealloc<C::kTmemCols>(tmem_base);
    }
}

// BF16 rows -> packed codes a0, a1 (m, k / 2) and scale rows (m, passes, k / 16).  A block takes 16 rows x 256 K, a thread one
// 16-element block.  HBM-bound; m % 16 == 0, k % 256 == 0.
template <bool kResidual, int kPolicy>
__global__ void __launch_bounds__(256)
stream_quantize_kernel(const __nv_bfloat16* __restrict__ a, int64_t lda, uint32_t k, uint8_t* __restrict__ a0, uint8_t* __restrict__ a1,
                       uint8_t* __restrict__ sf)
{
    constexpr uint32_t kPass = kResidual ? 2 : 1;
    const uint32_t chunks = k / 256, row = blockIdx.x / chunks * 16 + threadIdx.x / 16, col = blockIdx.x % chunks * 256 + threadIdx.x % 16 * 16;
    ptx::grid_dependency_wait();
    const uint4* src = reinterpret_cast<const uint4*>(a + static_cast<int64_t>(row) * lda + col);
    const uint4 lo = __ldg(src), hi = __ldg(src + 1);
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    xform::Block16 out;
    xform::decompose_block16<kResidual, kPolicy>(w, out);
    const uint64_t code = static_cast<uint64_t>(row) * (k / 2) + col / 2;
    *reinterpret_cast<uint2*>(a0 + code) = make_uint2(out.q0[0], out.q0[1]);
    if constexpr (kResidual) *reinterpret_cast<uint2*>(a1 + code) = make_uint2(out.q1[0], out.q1[1]);
    const uint32_t blk = threadIdx.x & 3u;
    uint32_t s0 = out.s0 << (8 * blk), s1 = out.s1 << (8 * blk);
    s0 |= __shfl_xor_sync(0xffffffffu, s0, 1); s0 |= __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 |= __shfl_xor_sync(0xffffffffu, s1, 1); s1 |= __shfl_xor_sync(0xffffffffu, s1, 2);
    uint8_t* dst = sf + static_cast<uint64_t>(row) * kPass * (k / 16) + col / 64 * 4;
    if (blk == 0) *reinterpret_cast<uint32_t*>(dst) = s0;
    if (kResidual && blk == 1) *reinterpret_cast<uint32_t*>(dst + k / 16) = s1;
    ptx::grid_launch_dependents();
}

struct Call {
    const void *a0, *a1, *sf;                        // quantised activations, rows x K
    const void *b, *sfb;
    int rows, N, K, E, num_sms;
    bool pdl;
    cudaStream_t stream;
};

template <uint32_t T, uint32_t BK, bool kResidual, bool kMasked, bool kSwigluOut>
int launch_variant(const Call& c, const Params& p)
{
    using C = Cfg<T, BK, kResidual, kSwigluOut>;
    CUtensorMap tm_a0, tm_a1, tm_sft, tm_w, tm_sfw;
    const uint64_t k = c.K;
    int rc = host::encode_tensor_map_2d(&tm_a0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.a0, k / 2, c.rows, k / 2, 128, T, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = host::encode_tensor_map_2d(&tm_a1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, kResidual ? c.a1 : c.a0, k / 2, c.rows, k / 2, 128, T,
                                    CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = host::encode_tensor_map_2d(&tm_sft, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, c.sf, C::kPass * (k / 64), c.rows, C::kPass * (k / 16), C::kAtoms, T,
                                    CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
    rc = host::encode_tensor_map_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.b, k / 2, static_cast<uint64_t>(c.E) * c.N, k / 2, 128, BW,
                                    CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = host::encode_tensor_map_2d(&tm_sfw, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, c.sfb, c.N, static_cast<uint64_t>(c.E) * (k / 64),
                                    static_cast<uint64_t>(c.N) * 4, BW, C::kAtoms, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
    auto kernel = gemm_stream_kernel<T, BK, kResidual, kMasked, kSwigluOut>;
    static bool attr_set[host::kMaxDevices] = {};
    int dev = 0;
    NVFP4_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev]) {
        NVFP4_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemAlloc));
        attr_set[dev] = true;
    }
    const int64_t tiles = static_cast<int64_t>(c.rows / static_cast<int>(T)) * (c.N / static_cast<int>(BW));
    const int grid = tiles < c.num_sms ? static_cast<int>(tiles) : c.num_sms;
    return host::launch_kernel(kernel, dim3(static_cast<unsigned>(grid)), dim3(kThreads), C::kSmemAlloc, c.stream, c.pdl, tm_a0, tm_a1, tm_sft,
                               tm_w, tm_sfw, p);
}

template <uint32_t T, bool kResidual>
int launch_contiguous(const Call& c, const Params& p)
{
    if constexpr (T <= 32)
        if (c.K % 512 == 0) return launch_variant<T, 512, kResidual, false, false>(c, p);
    return launch_variant<T, 256, kResidual, false, false>(c, p);
}

}  // namespace

// Contiguous layout, BF16 activations: quantised into a workspace first.  token_tile 16, 32 or 64, K % 256 == 0.
int launch_gemm_stream(const void* a, int64_t lda, const void* b, const void* sfb, const float* gw, void* d, int64_t ldd,
                       const int32_t* m_indices, int M, int N, int K, int E, bool residual, int token_tile, int policy, bool pdl, int num_sms,
                       int32_t* status, cudaStream_t stream)
{
    int dev = 0;
    NVFP4_CUDA_CHECK(cudaGetDevice(&dev));
    cudaMemPool_t pool;
    if (int rc = host::workspace_pool(dev, &pool)) return rc;
    const size_t passes = residual ? 2 : 1, codes = static_cast<size_t>(M) * (K / 2), scales = passes * M * static_cast<size_t>(K / 16);
    uint8_t* ws = nullptr;
    NVFP4_CUDA_CHECK(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&ws), passes * codes + scales, pool, stream));
    uint8_t *a0 = ws, *a1 = ws + (passes - 1) * codes, *sf = ws + passes * codes;
    const int rc = [&]() -> int {
        const unsigned blocks = static_cast<unsigned>(M / 16) * static_cast<unsigned>(K / 256);
        const int qrc = host::with_policy(policy, [&](auto pol) {
            constexpr int kP = decltype(pol)::value;
            return host::launch_kernel(residual ? stream_quantize_kernel<true, kP> : stream_quantize_kernel<false, kP>, dim3(blocks), dim3(256), 0,
                                       stream, pdl, static_cast<const __nv_bfloat16*>(a), lda, static_cast<uint32_t>(K), a0, a1, sf);
        });
        if (qrc) return qrc;
        const Params p{gw, m_indices, static_cast<__nv_bfloat16*>(d), ldd, static_cast<uint32_t>(M), static_cast<uint32_t>(N),
                       static_cast<uint32_t>(K), 0u, 1u, gemm::Family{}, nullptr, nullptr, nullptr, status};
        const Call c{a0, a1, sf, b, sfb, M, N, K, E, num_sms, pdl, stream};
        switch (token_tile) {
            case 16: return residual ? launch_contiguous<16, true>(c, p) : launch_contiguous<16, false>(c, p);
            case 32: return residual ? launch_contiguous<32, true>(c, p) : launch_contiguous<32, false>(c, p);
            default: return residual ? launch_contiguous<64, true>(c, p) : launch_contiguous<64, false>(c, p);
        }
    }();
    cudaFreeAsync(ws, stream);
    return rc;
}

// Masked layout over quantised rows (both passes), token tiles of 32 or 64.  out_a0 != nullptr: gate/up-interleaved weights,
// the output is the quantised SwiGLU activation; else BF16 rows in d.  has_rival: the 128-row
// kernels are launched for the same call, see gemm::Family.
int launch_gemm_stream_quantized(const void* a0, const void* a1, const void* scale_rows, const void* b, const void* sfb, const float* gw,
                                 void* d, int64_t ldd, const int32_t* masked_m, int max_m, int N, int K, int E, int token_tile, void* out_a0,
                                 void* out_a1, void* out_sf, bool pdl, int num_sms, int32_t* status, cudaStream_t stream, bool has_rival)
{
    const Params p{gw, masked_m, static_cast<__nv_bfloat16*>(d), ldd, static_cast<uint32_t>(E * max_m), static_cast<uint32_t>(N),
                   static_cast<uint32_t>(K), static_cast<uint32_t>(E), static_cast<uint32_t>(max_m),
                   gemm::Family{has_rival ? static_cast<uint32_t>(token_tile) : 0u, true}, static_cast<uint8_t*>(out_a0),
                   static_cast<uint8_t*>(out_a1), static_cast<uint8_t*>(out_sf), status};
    const Call c{a0, a1, scale_rows, b, sfb, E * max_m, N, K, E, num_sms, pdl, stream};
    const bool swiglu = out_a0 != nullptr;
    if (token_tile == 64) return swiglu ? launch_variant<64, 256, true, true, true>(c, p) : launch_variant<64, 256, true, true, false>(c, p);
    if (K % 512 == 0) return swiglu ? launch_variant<32, 512, true, true, true>(c, p) : launch_variant<32, 512, true, true, false>(c, p);
    return swiglu ? launch_variant<32, 256, true, true, true>(c, p) : launch_variant<32, 256, true, true, false>(c, p);
}

}  // namespace nvfp4
