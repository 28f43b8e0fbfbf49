// Offline NVFP4 weight quantisation on the GPU: w ~= dec(q) * S * G with one FP32 G
// per expert, one E4M3 S per 16 elements and E2M1 codes, written straight into the
// physical layouts the GEMM's tensor maps describe.  Bit-exact with the reference's
// torch implementation (python/nvfp4_gemm/layout.py:68-127): the codes and scales of
// its three FP32 divisions (kept reciprocals where they round alike, see `divide`), the
// same clamps, RNE everywhere.
//
// HBM-bound: 2 or 4 bytes read per element, 9/16 byte written.  G needs the maximum of a whole expert before any of its
// blocks can be quantised, so the weights are read twice; the second read should come out of L2.  The experts are
// therefore taken in batches (one expert, or several small ones, kBatchBytes) and one kernel walks a list of tiles in
// which the quantisation of batch i - 1, which sits in L2, is interleaved with the maxima of batch i, which streams in
// from HBM.  Blocks draw tiles from a counter in list order and a quantisation tile waits only for tiles ahead of it,
// so whatever number of blocks runs at a time, the ones that are waited for are running or done.
// Quantisation goes through a batch backwards, from what was read last: its reads end up further apart the longer the stage
// lasts, and the early ones hit L2 where, in list order, every one would come a whole batch after its first read.
// Measured (BF16): 8 experts of 4096 x 7168 (58 MB each, too large for two of them to share L2) 179-180 us, 184-185 in list
// order, 92 if the weights crossed HBM once; 64 of them 1280 us, 1480 in list order;
// 32 of 4096 x 1536: 132 us, 136 in list order = 3.9 TB/s of 400 MB read and 113 MB written once, the rest is the warps' latency.
// A tile's stage comes from a division: all stages but the first and the last two have as many tiles.  (Walking the stages, a batch each: 256 of
// 4096 x 2048, 256 batches, 2870 us; 1870-1940 so.)  1024 experts in 22 batches (256 x 1024) 166 us.
#include <climits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "host_common.hpp"
#include "launchers.hpp"
#include "ptx.cuh"

namespace nvfp4 {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32, kBlocksPerSm = 3;
constexpr int kUnitRows = 8, kUnitK = 512, kStep = 2;      // a warp's share of a quantisation tile: 8 weight rows x 512 K,
constexpr int kTileRows = kWarps * kUnitRows;              // two rows at a time; the tile: 64 rows
constexpr int kAmaxUnroll = 8, kAmaxSteps = 2;             // a maximum tile: two times eight 32-byte loads per thread
constexpr int64_t kBatchBytes = 24ll << 20;

__device__ __forceinline__ float e4m3_to_f32(uint32_t code)
{
    uint32_t h2;
    asm("{\n .reg .b16 t;\n cvt.u16.u32 t, %1;\n cvt.rn.f16x2.e4m3x2 %0, t;\n}" : "=r"(h2) : "r"(code & 0xffu));
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xffffu)));
}

// 32 bytes of weights.  kLast: the last use of the line, which may leave L2 before the lines that are still to be read.
// kAligned = false: a tensor that starts off a 32-byte boundary, read element by element.
struct Vec { uint32_t w[8]; };
template <typename T, bool kAligned, bool kLast>
__device__ __forceinline__ Vec load32(const T* p)
{
    Vec v;
    if constexpr (!kAligned) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if constexpr (std::is_same_v<T, float>) v.w[i] = __float_as_uint(p[i]);
            else v.w[i] = __bfloat16_as_ushort(p[2 * i]) | static_cast<uint32_t>(__bfloat16_as_ushort(p[2 * i + 1])) << 16;
        }
    } else if constexpr (kLast) {
        asm volatile("ld.global.nc.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    } else {
        asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7]) : "l"(p));
    }
    return v;
}

// max(m, largest magnitude of the vector)
template <typename T>
__device__ __forceinline__ float amax_of(float m, const Vec& v)
{
    if constexpr (std::is_same_v<T, float>) {
#pragma unroll
        for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(__uint_as_float(v.w[i])));
        return m;
    } else {
        uint32_t h = v.w[0];
#pragma unroll
        for (int i = 1; i < 8; ++i) h = ptx::max_abs_bf16x2(h, v.w[i]);
        h = ptx::max_abs_bf16x2(h, h >> 16);
        return fmaxf(m, __uint_as_float((h & 0x7fffu) << 16));
    }
}

// One tile of the maximum pass: 128 KB of one expert; the result is valid in thread 0.
template <typename T, bool kAligned>
__device__ __forceinline__ uint32_t amax_tile(const T* __restrict__ expert, int64_t per_expert, uint32_t tile, uint32_t (&warp_max)[kWarps])
{
    constexpr int kElems = 32 / sizeof(T);
    const int64_t vecs = per_expert / kElems;
    float m = 0.0f;
#pragma unroll 1
    for (int step = 0; step < kAmaxSteps; ++step) {
        const int64_t first = (static_cast<int64_t>(tile) * kAmaxSteps + step) * (kThreads * kAmaxUnroll) + threadIdx.x;
        Vec v[kAmaxUnroll];
#pragma unroll
        for (int u = 0; u < kAmaxUnroll; ++u)
            v[u] = first + u * kThreads < vecs ? load32<T, kAligned, false>(expert + (first + u * kThreads) * kElems) : Vec{};
#pragma unroll
        for (int u = 0; u < kAmaxUnroll; ++u) m = amax_of<T>(m, v[u]);
    }
    uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(m));  // non-negative floats order as integers
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
    __syncthreads();
    return threadIdx.x < 32 ? __reduce_max_sync(0xffffffffu, threadIdx.x < kWarps ? warp_max[threadIdx.x] : 0u) : 0u;
}

// Quotients are rounded to FP32 before they are coded (the torch code divides), so they have to be the correctly rounded
// ones wherever a code depends on it.  With y = 1 / d and an approximate quotient q, the remainder r = x - d * q is exact
// in one FMA and q + r * y, rounded once, is the next approximation; when y is the rounded reciprocal and q is within one
// ulp, it is the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990).  x * y is within 1.5 ulp, so one step
// gets q there and a second one finishes.  Nothing underflows as long as d is of ordinary size, which the caller sees
// to (kOrdinary); the other instantiation divides.  -q is what is computed, so that a zero keeps its sign: q itself would
// be -0 + 0.
template <bool kOrdinary>
__device__ __forceinline__ float divide(float x, float d, float y)
{
    if constexpr (!kOrdinary) return __fdiv_rn(x, d);
    float q = __fmul_rn(x, -y);
    q = __fmaf_rn(__fmaf_rn(d, q, x), -y, q);
    return -__fmaf_rn(__fmaf_rn(d, q, x), -y, q);
}

// E2M1 codes of the 16 quotients x / d.
//
// A BF16 numerator needs one step less, and y may be a few ulp^2 off the rounded reciprocal.  The result is then rounded
// from a value within 2^-47 of x / d, and its code can only be wrong if x / d is that close to a rounding boundary next
// to a threshold t of the E2M1 grid.  With x = X 2^a (X < 2^8), d = D (2^23 <= D < 2^24) and t = T 2^j
// (T in {1, 3, 5, 7}) that asks for X 2^a = D (T 2^b +- 1) + eps with |eps| <= 4, a >= 41 and b in {22, 23, 24}; modulo
// 2^41 the only solution below 2^24 is D = 2^24 - 1 with T = 1 and X a power of two.  For that D the reciprocal
// (1 + 2^-24 + 2^-48 times a power of two) is rounded up by hand; the remainder step then lands above the boundary.
//
// This form takes -x, which costs nothing where the halves of a word are unpacked: what comes out is then +q, with the sign of
// a zero, and a NaN is left to the conversion, which makes it the largest positive code whatever its sign.  (Flipping the sign
// bits of the codes of -q turned a NaN over, too; negating the quotients took 189 us on the 8 experts above, this 183.)
template <typename T, bool kOrdinary>
constexpr bool kNegated = kOrdinary && !std::is_same_v<T, float>;
template <typename T, bool kOrdinary>
__device__ __forceinline__ void quantize_block(const float (&x)[16], float d, uint32_t (&packed)[2])
{
    float q[16];
    if constexpr (kNegated<T, kOrdinary>) {
        const float r = ptx::rcp_approx(d);
        float y = __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r);
        if ((__float_as_uint(d) & 0x7fffffu) == 0x7fffffu) y = __uint_as_float(__float_as_uint(y) | 1u);
        const float2 ny = make_float2(-y, -y), dd = make_float2(d, d);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const float2 xx = make_float2(x[i], x[i + 1]), u = ptx::mul_f32x2(xx, ny);
            const float2 v = ptx::fma_f32x2(ptx::fma_f32x2(dd, u, xx), ny, u);
            q[i] = v.x;
            q[i + 1] = v.y;
        }
    } else {
        const float y = kOrdinary ? __frcp_rn(d) : 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) q[i] = divide<kOrdinary>(x[i], d, y);
    }
    packed[0] = ptx::cvt_e2m1x8(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]);
    packed[1] = ptx::cvt_e2m1x8(q[8], q[9], q[10], q[11], q[12], q[13], q[14], q[15]);
}

// A warp's share of a quantisation tile: 8 weight rows x 512 K of one expert, a row at a time, a lane one 16-element block of
// it, so that reads and code stores are contiguous; four neighbouring lanes make one scale word, and the eight rows' words
// of a K atom are one 32-byte sector of the transposed (K/64, N) array.  The next two rows are on their way while the warp
// computes on the current two; `v` holds the first two at the start.  kFull: the tile lies inside the matrix, nothing
// needs a bounds check.
template <typename T>
using Rows = Vec[kStep][16 * sizeof(T) / 32];
template <typename T, bool kAligned, bool kFull>
__device__ __forceinline__ void request_rows(const T* __restrict__ w, int N, int K, int e, int n0, int k0, Rows<T>& to)
{
    constexpr int kElems = 32 / sizeof(T), kVecs = 16 / kElems;          // 32-byte vectors of a block: 1 or 2
    const int k = k0 + (threadIdx.x & 31) * 16;
    const T* src = w + (static_cast<int64_t>(e) * N + n0) * K + k;
#pragma unroll
    for (int r = 0; r < kStep; ++r)
#pragma unroll
        for (int c = 0; c < kVecs; ++c)
            to[r][c] = kFull || (n0 + r < N && k < K) ? load32<T, kAligned, true>(src + static_cast<int64_t>(r) * K + c * kElems) : Vec{};
}

template <typename T, bool kAligned, bool kFull, bool kOrdinary>
__device__ __forceinline__ void quantize_unit(const T* __restrict__ w, int N, int K, int e, int n0, int k0, uint8_t* __restrict__ b,
                                              int32_t* __restrict__ sfb, Rows<T>& first, float g, float rg)
{
    constexpr int kVecs = 16 * sizeof(T) / 32;
    const float tiny = 1.17549435e-38f;
    const int lane = threadIdx.x & 31, k = k0 + lane * 16;
    uint8_t* dst = b + (static_cast<int64_t>(e) * N + n0) * (K / 2) + k / 2;
    Rows<T> second;
    uint32_t word = 0;                                                   // lane 4 i + j ends up with rows j and j + 4 of K atom i
    uint32_t word_hi = 0;
#pragma unroll
    for (int step = 0; step < kUnitRows / kStep; ++step) {
        Rows<T>& now = step & 1 ? second : first;
        if (step + 1 < kUnitRows / kStep) request_rows<T, kAligned, kFull>(w, N, K, e, n0 + (step + 1) * kStep, k0, step & 1 ? first : second);
#pragma unroll
        for (int r = 0; r < kStep; ++r) {
            const int n = step * kStep + r;
            float m = 0.0f;
            float x[16];
#pragma unroll
            for (int c = 0; c < kVecs; ++c) {
                const Vec& q = now[r][c];
                m = amax_of<T>(m, q);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if constexpr (std::is_same_v<T, float>) {
                        x[8 * c + i] = __uint_as_float(q.w[i]);
                    } else {
                        constexpr uint32_t kSign = kNegated<T, kOrdinary> ? 0x80000000u : 0u;
                        x[2 * i] = __uint_as_float(q.w[i] * 65536u + kSign);
                        x[2 * i + 1] = __uint_as_float((q.w[i] & 0xffff0000u) ^ kSign);
                    }
                }
            }
            // m / 6 is at least 1/6 of a unit away from every rounding boundary: the product with 1/6 (to 2^-49) decides
            const float m6 = kOrdinary ? __fmaf_rn(m, 0x1.555556p-3f, __fmul_rn(m, -0x1.555556p-28f)) : __fdiv_rn(m, 6.0f);
            const uint32_t sc = ptx::cvt_e4m3(fmaxf(divide<kOrdinary>(m6, g, rg), 0.001953125f));
            uint32_t packed[2];
            quantize_block<T, kOrdinary>(x, fmaxf(__fmul_rn(e4m3_to_f32(sc), g), tiny), packed);
            if (kFull || (n0 + n < N && k < K))
                *reinterpret_cast<uint2*>(dst + static_cast<int64_t>(n) * (K / 2)) = make_uint2(packed[0], packed[1]);
            uint32_t s4 = sc << (8 * (lane & 3));
            s4 |= __shfl_xor_sync(0xffffffffu, s4, 1);
            s4 |= __shfl_xor_sync(0xffffffffu, s4, 2);
            if ((lane & 3) == (n & 3)) { if (n < 4) word = s4; else word_hi = s4; }
        }
    }
    const int at = k0 / 64 + (lane >> 2), n = n0 + (lane & 3);
    int32_t* out = sfb + (static_cast<int64_t>(e) * (K / 64) + at) * N + n;
    if (kFull || (at < K / 64 && n < N)) out[0] = static_cast<int32_t>(word);
    if (kFull || (at < K / 64 && n + 4 < N)) out[4] = static_cast<int32_t>(word_hi);
}

// The scratch words of a call, zero at its start: the next tile to draw, whether a wait ran out of time, and per expert the
// maximum (FP32 bits) and the number of its maximum tiles that are done, each spread over kSlots words.  (An atomic per
// warp on one word of either kind was what the kernel waited for: some 7 ns each on one address.)
constexpr int kSlots = 16;
struct Scratch {
    uint32_t* amax_bits;
    uint32_t* done;
    uint32_t* ticket;
    uint32_t* expired;
};
constexpr int64_t scratch_words(int64_t experts) { return 2 * kSlots * experts + 2; }
constexpr long long kDoneBudget = 2000000000ll;      // cycles, about a second; maxima are taken in microseconds

// A wait for an expert's maxima that runs out of time (it does not happen in a healthy run) must not end in weights that look
// like weights: every global scale becomes NaN.  Who stores one looks at `expired` after its store, who found the
// time run out sets `expired` before its own; with a sequentially consistent fence between the two on either side, the
// NaN is what remains whichever comes first.
__device__ __forceinline__ void fence_sc() { asm volatile("fence.sc.gpu;" ::: "memory"); }
__device__ __forceinline__ void poison(const Scratch& scratch, float* gw, int experts)
{
    for (int e = static_cast<int>(threadIdx.x & 31u); e < experts; e += 32) {
        *reinterpret_cast<volatile uint32_t*>(scratch.expired) = 1u;
        fence_sc();
        *reinterpret_cast<volatile float*>(gw + e) = __int_as_float(0x7fffffff);
    }
}
__device__ __forceinline__ void store_global_scale(const Scratch& scratch, float* gw, float g)
{
    *reinterpret_cast<volatile float*>(gw) = g;
    fence_sc();
    if (*reinterpret_cast<const volatile uint32_t*>(scratch.expired) != 0) *reinterpret_cast<volatile float*>(gw) = __int_as_float(0x7fffffff);
}

// List position i: stage 0 is the maxima of batch 0; stage s the quantisation of batch s - 1 and the maxima of batch s
// in proportion; the last stage the quantisation of the last batch.  A stage opens with as many maxima tiles as there are
// blocks: while they are read, the maxima that its quantisation tiles need, drawn just before them, are finished.
// `need`: maxima tiles of an expert to wait for, `at` but in the test of the wait that runs out after `budget` cycles.
template <typename T, bool kAligned>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
quantize_weight_kernel(const T* __restrict__ w, int E, int N, int K, int batch, uint32_t qt, uint32_t at, Scratch scratch,
                       uint32_t need, long long budget, uint8_t* __restrict__ b, int32_t* __restrict__ sfb, float* gw)
{
    __shared__ uint32_t warp_max[kWarps];
    __shared__ uint32_t drawn, stop;
    const uint32_t kt = static_cast<uint32_t>((K + kUnitK - 1) / kUnitK), lane = threadIdx.x & 31;
    const uint32_t total = static_cast<uint32_t>(E) * (at + qt);
    const uint32_t full_stage = static_cast<uint32_t>(batch) * (at + qt), stages = static_cast<uint32_t>((E + batch - 1) / batch);
    uint32_t next = 0;
    if (threadIdx.x == 0) { next = atomicAdd(scratch.ticket, 1u); stop = 0; }
    int known = -1;                                  // expert whose global scale this thread holds
    float g = 0.0f, rg = 0.0f;
    for (;;) {
        if (threadIdx.x == 0) drawn = next;
        __syncthreads();
        uint32_t i = drawn;
        const bool stopped = stop != 0;
        __syncthreads();
        if (stopped || i >= total) return;
        if (threadIdx.x == 0) next = atomicAdd(scratch.ticket, 1u);      // arrives while this tile is worked on
        int first_a = 0;                             // first expert of the stage's maxima
        uint32_t na = min(batch, E) * at, nq = 0;    // tiles of either kind in the stage
        if (i >= na + full_stage) {                  // all stages but the first and the last two are alike
            const uint32_t skip = min((i - na) / full_stage, stages - 2);
            i -= skip * full_stage;
            first_a = static_cast<int>(skip) * batch;
        }
        while (i >= na + nq) {
            i -= na + nq;
            nq = min(batch, E - first_a) * qt;
            first_a += batch;
            na = first_a < E ? min(batch, E - first_a) * at : 0u;
        }
        const uint32_t lead = min(na, gridDim.x);
        const uint64_t here = static_cast<uint64_t>(na - lead) + nq, at_mix = i < lead ? 0 : i - lead;
        const uint32_t q_before = here ? static_cast<uint32_t>(at_mix * nq / here) : 0u;
        const uint32_t q_after = here && i >= lead ? static_cast<uint32_t>((at_mix + 1) * nq / here) : q_before;
        if (q_after > q_before) {
            // last read, first quantised
            const uint32_t back = nq - 1 - q_before, r = back % qt;
            const int e = first_a - batch + static_cast<int>(back / qt);
            const int n0 = static_cast<int>(r / kt) * kTileRows, k0 = static_cast<int>(r % kt) * kUnitK;
            const int nw = n0 + static_cast<int>(threadIdx.x >> 5) * kUnitRows;
            const bool full = n0 + kTileRows <= N && k0 + kUnitK <= K;
            Rows<T> rows;
            if (full) request_rows<T, kAligned, true>(w, N, K, e, nw, k0, rows);
            else request_rows<T, kAligned, false>(w, N, K, e, nw, k0, rows);
            if (known != e) {
                const long long t0 = clock64();
                const uint32_t slot = static_cast<uint32_t>(e) * kSlots + lane % kSlots;
                uint32_t n = 0;
                for (;;) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(scratch.done + slot) : "memory");
                    n = __reduce_add_sync(0xffffffffu, lane < kSlots ? n : 0u);
                    if (n >= need || __any_sync(0xffffffffu, clock64() - t0 > budget)) break;
                    __nanosleep(100);
                }
                if (n < need) {                       // the whole warp: the block ends before its next tile
                    poison(scratch, gw, E);
                    stop = 1;
                    continue;
                }
                const uint32_t bits = __reduce_max_sync(0xffffffffu, *reinterpret_cast<const volatile uint32_t*>(scratch.amax_bits + slot));
                g = fmaxf(__fdiv_rn(__uint_as_float(bits), 2688.0f), 1.17549435e-38f);
                rg = __frcp_rn(g);
                known = e;
            }
            // block scales lie between 2^-9 g and 448 g
            const bool ordinary = g > 0x1p-60f && g < 0x1p60f;
            if (full && ordinary) quantize_unit<T, kAligned, true, true>(w, N, K, e, nw, k0, b, sfb, rows, g, rg);
            else if (ordinary) quantize_unit<T, kAligned, false, true>(w, N, K, e, nw, k0, b, sfb, rows, g, rg);
            else quantize_unit<T, kAligned, false, false>(w, N, K, e, nw, k0, b, sfb, rows, g, rg);
            if (r == 0 && threadIdx.x == 0) store_global_scale(scratch, gw + e, g);
        } else {
            const uint32_t t = i - q_before;
            const int e = first_a + static_cast<int>(t / at);
            const int64_t per_expert = static_cast<int64_t>(N) * K;
            const uint32_t bits = amax_tile<T, kAligned>(w + e * per_expert, per_expert, t % at, warp_max);
            if (threadIdx.x == 0) {
                const uint32_t slot = static_cast<uint32_t>(e) * kSlots + t % kSlots;
                atomicMax(scratch.amax_bits + slot, bits);
                __threadfence();
                atomicAdd(scratch.done + slot, 1u);
            }
        }
    }
}

template <typename T>
int run_batches(const T* w, int E, int N, int K, void* b, void* sfb, float* gw, const Scratch& scratch, uint32_t need_more,
                long long budget, cudaStream_t stream)
{
    const int64_t per_expert = static_cast<int64_t>(N) * K;
    const int64_t fit = kBatchBytes / (per_expert * static_cast<int64_t>(sizeof(T)));
    const int batch = fit < 1 ? 1 : (fit > E ? E : static_cast<int>(fit));
    const int64_t per_tile = static_cast<int64_t>(kThreads) * kAmaxUnroll * kAmaxSteps * 32 / static_cast<int64_t>(sizeof(T));
    const int64_t at = (per_expert + per_tile - 1) / per_tile;
    const int64_t qt = static_cast<int64_t>((K + kUnitK - 1) / kUnitK) * ((N + kTileRows - 1) / kTileRows);
    NVFP4_REQUIRE((at + qt) * E <= INT32_MAX, "weights too large for one call (E=%d, N=%d, K=%d)", E, N, K);
    host::DeviceInfo* dev;
    if (int rc = host::device_info(-1, &dev)) return rc;
    const int64_t blocks = static_cast<int64_t>(dev->hw_sms) * kBlocksPerSm, tiles = (at + qt) * E;
    const bool aligned = (reinterpret_cast<uintptr_t>(w) & 31u) == 0;
    auto kernel = aligned ? quantize_weight_kernel<T, true> : quantize_weight_kernel<T, false>;
    return host::launch_kernel(kernel, dim3(static_cast<unsigned>(blocks < tiles ? blocks : tiles)), dim3(kThreads), 0, stream, false, w, E, N, K,
                               batch, static_cast<uint32_t>(qt), static_cast<uint32_t>(at), scratch,
                               static_cast<uint32_t>(at) + need_more, budget, static_cast<uint8_t*>(b), static_cast<int32_t*>(sfb), gw);
}

// `words`: scratch_words(E) words the caller provides; they are cleared here, on the call's stream.  need_more, budget: for the
// test of a wait that runs out of time.
int run_quantize_weight(const void* w, int w_dtype, int E, int N, int K, void* b, void* sfb, float* gw, uint32_t* words,
                        cudaStream_t stream, uint32_t need_more = 0, long long budget = kDoneBudget)
{
    NVFP4_CUDA_CHECK(cudaMemsetAsync(words, 0, sizeof(uint32_t) * scratch_words(E), stream));
    const int64_t slots = static_cast<int64_t>(kSlots) * E;
    const Scratch scratch{words, words + slots, words + 2 * slots, words + 2 * slots + 1};
    return w_dtype == NVFP4_DTYPE_BF16
               ? run_batches(static_cast<const __nv_bfloat16*>(w), E, N, K, b, sfb, gw, scratch, need_more, budget, stream)
               : run_batches(static_cast<const float*>(w), E, N, K, b, sfb, gw, scratch, need_more, budget, stream);
}

}  // namespace

// The per-expert maxima live in a stream-ordered allocation from the library's memory pool: calls on
// different streams never share it, nothing synchronises the device, and after the first call it is a pool look-up.
int launch_quantize_weight(const void* w, int w_dtype, int E, int N, int K, void* b, void* sfb, float* gw,
                           cudaStream_t stream, int64_t expire_after_cycles)
{
    if (E == 0 || N == 0 || K == 0) return NVFP4_OK;
    int dev = 0;
    NVFP4_CUDA_CHECK(cudaGetDevice(&dev));
    cudaMemPool_t pool;
    if (int rc = host::workspace_pool(dev, &pool)) return rc;
    uint32_t* amax_bits = nullptr;
    NVFP4_CUDA_CHECK(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&amax_bits), sizeof(uint32_t) * scratch_words(E), pool, stream));
    const int rc = expire_after_cycles > 0 ? run_quantize_weight(w, w_dtype, E, N, K, b, sfb, gw, amax_bits, stream, 1u, expire_after_cycles)
                                           : run_quantize_weight(w, w_dtype, E, N, K, b, sfb, gw, amax_bits, stream);
    cudaFreeAsync(amax_bits, stream);
    return rc;
}

// ---- allocation-free variant ----------------------------------------------------------
// The same kernel, but its scratch words are a fixed array that is part of the library
// image instead of an allocation.  Every process that loads the library holds
// scratch_words(NVFP4_STATIC_MAX_EXPERTS) words of it on every GPU it uses, until it exits.
namespace {
static __device__ __align__(256) uint32_t g_static_amax[scratch_words(NVFP4_STATIC_MAX_EXPERTS)];
std::mutex g_static_mutex;
}  // namespace

// In host code `g_static_amax` is only the host-side handle of the symbol, not an address
// a kernel can dereference.  The device address comes from cudaGetSymbolAddress, asked once
// per device with that device current -- here on the first call made on that device.
int launch_quantize_weight_static(const void* w, int w_dtype, int E, int N, int K, void* b, void* sfb, float* gw,
                                  cudaStream_t stream)
{
    if (E == 0 || N == 0 || K == 0) return NVFP4_OK;
    static uint32_t* scratch_addr[host::kMaxDevices] = {};
    int dev = 0;
    NVFP4_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= host::kMaxDevices) return host::fail(NVFP4_E_INVALID_ARGUMENT, "device %d out of range", dev);
    uint32_t* amax_bits = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_mutex);
        if (scratch_addr[dev] == nullptr) {
            void* addr = nullptr;
            NVFP4_CUDA_CHECK(cudaGetSymbolAddress(&addr, g_static_amax));
            if (addr == nullptr) return host::fail(NVFP4_E_CUDA, "cudaGetSymbolAddress gave no address for the scratch array");
            scratch_addr[dev] = static_cast<uint32_t*>(addr);
        }
        amax_bits = scratch_addr[dev];
    }
    // the array keeps whatever the previous call left in it: run_quantize_weight clears its words first
    return run_quantize_weight(w, w_dtype, E, N, K, b, sfb, gw, amax_bits, stream);
}

}  // namespace nvfp4
