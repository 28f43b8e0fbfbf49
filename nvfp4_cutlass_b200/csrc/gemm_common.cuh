// Pieces shared by the GEMM kernels: the ring cursor (ring.cuh), the persistent tile order (contiguous and masked
// layouts) and the epilogue's line-coalesced output stores.
#pragma once
#include <cuda_bf16.h>

#include "ptx.cuh"
#include "ring.cuh"

namespace nvfp4::gemm {

// Tiles are walked in groups of `group_m` row blocks: inside a group the row block changes fastest, so the
// CTAs running at the same time share a few weight tiles and a few activation tiles in L2.
// Counterpart in the reference: include/nvfp4_gemm/scheduler/grouped_gemm.cuh:86-99.
__device__ __forceinline__ void tile_coords(uint32_t tile, uint32_t num_m, uint32_t num_n, uint32_t group_m,
                                            uint32_t& m_blk, uint32_t& n_blk)
{
    const uint32_t per_group = group_m * num_n;
    const uint32_t g = tile / per_group, r = tile % per_group;
    const uint32_t first = g * group_m;
    const uint32_t rows = min(group_m, num_m - first);
    m_blk = first + r % rows;
    n_blk = r / rows;
}

// What a role needs to know about its next tile.
struct Tile {
    uint32_t row0;     // first row of the tile in a / d
    uint32_t n_blk;    // column block
    int32_t expert;    // whose weights
};

// Persistent static-stride tile order over either layout.
//   contiguous: rows grouped by expert, expert of a row block read from m_indices (negative ids read as 0)
//   masked:     `groups` experts with `max_m` rows reserved each, of which the first masked_m[g] (a device-side
//               count, clamped to max_m) are real; row blocks past the count do not exist
//               (counterpart in the reference: scheduler/grouped_gemm.cuh:139-156)
// Two families of kernels can take a masked call whose groups may have few rows or many: the decode kernels, token tiles of
// `tile` rows, and the 128-row kernels.  Only the device knows the counts, so both are launched and the family that is the
// slower one for them leaves at once.  The decode kernels pass an expert's weights once per token tile, the others once
// per block of 128 rows: the decode kernels take the call with up to two and a half tiles of 32, or one and a half of 64, to a
// block.  Expert layer of 128 experts, 4096 / 1536, decode / 128-row kernels, tiles of 32: uniform routing, 1.1 tiles to a block,
// 260 / 359 us; skewed, 1.5, 128 / 152; 1.8, 164 / 165; 2.4, 210 / 199; all tokens on eight experts, 4, 173 / 131; tiles of 64:
// uniform, 1.0, 340 / 378; skewed, 1.6, 225 / 215; 1.8, 300 / 260.  64 experts of 3072 / 1536, skewed, tiles of 32: 2.1, 104 /
// 122, where few blocks leave the 128-row kernels a last wave.  To launch both costs some 7 us.
struct Family {
    uint32_t tile = 0;         // 0: no choice, this kernel takes the call
    bool few = false;          // of the decode kernels
    // For every warp on its own, the same for all; waits for the kernel that wrote the counts.
    __device__ __forceinline__ bool leaves(const int32_t* masked_m, uint32_t groups, uint32_t max_m) const
    {
        if (tile == 0) return false;
        ptx::grid_dependency_wait();
        int balance = 0;
        for (uint32_t g = threadIdx.x & 31u; g < groups; g += 32) {
            const uint32_t rows = min(static_cast<uint32_t>(max(0, __ldg(masked_m + g))), max_m);
            balance += static_cast<int>((rows + tile - 1) / tile * 2) - static_cast<int>((rows + 127) / 128 * (tile == 32 ? 5 : 3));
        }
        return (__reduce_add_sync(0xffffffffu, balance) <= 0) != few;
    }
};

// Every role of a CTA owns a walker and calls next() with the same sequence of linear tile indices.
template <uint32_t kBM, bool kMasked>
struct TileWalker {
    const int32_t* layout;   // m_indices (contiguous) or masked_m (masked)
    uint32_t num_m, num_n, group_m, groups, max_m;
    uint32_t g = 0, blocks_before = 0, blocks_here = 0;
    bool primed = false;

    __device__ __forceinline__ TileWalker(const int32_t* layout_, uint32_t m_rows, uint32_t n_cols, uint32_t bn,
                                          uint32_t group_m_, uint32_t groups_, uint32_t max_m_)
        : layout(layout_), num_m(m_rows / kBM), num_n((n_cols + bn - 1) / bn), group_m(group_m_), groups(groups_), max_m(max_m_)
    {
    }

    __device__ __forceinline__ uint32_t blocks_of(uint32_t group) const
    {
        const uint32_t rows = min(static_cast<uint32_t>(max(0, __ldg(layout + group))), max_m);
        return (rows + kBM - 1) / kBM;
    }

    // false when `linear` is past the last tile
    __device__ __forceinline__ bool next(uint32_t linear, Tile& t)
    {
        if constexpr (!kMasked) {
            if (linear >= num_m * num_n) return false;
            uint32_t m_blk;
            tile_coords(linear, num_m, num_n, group_m, m_blk, t.n_blk);
            t.row0 = m_blk * kBM;
            t.expert = max(0, __ldg(layout + t.row0));
            return true;
        } else {
            if (!primed) { blocks_here = groups ? blocks_of(0) : 0; primed = true; }
            for (;;) {
                if (g >= groups) return false;
                if (linear < (blocks_before + blocks_here) * num_n) break;
                blocks_before += blocks_here;
                if (++g < groups) blocks_here = blocks_of(g);
            }
            uint32_t m_blk;
            tile_coords(linear - blocks_before * num_n, blocks_here, num_n, group_m, m_blk, t.n_blk);
            t.row0 = g * max_m + m_blk * kBM;
            t.expert = static_cast<int32_t>(g);
            return true;
        }
    }
};

// Epilogue stores of one warp: `o` holds this lane's output row as 32 BF16 pairs (64 columns; in tensor memory
// a lane is a row).  A store instruction should write whole 128-byte lines, and with one row per lane every
// 16-byte store of the warp would land in a different line -- 4096 partial-line requests per 128 x 256 tile,
// measured to hold up the operand loads and the tensor pipe of the next tile for thousands of cycles.  So the
// eight lanes of a group first transpose their 8 x 8 pieces of 16 bytes in registers, three butterfly steps, after
// which lane j of the group holds piece j of each of the group's eight rows and a store writes four full lines.
// (Going through shared memory, four rows at a time, was a chain of 24 dependent accesses; under the tensor core's
// operand reads each takes some 300 cycles, and a tile's stores took 7500 -- longer than the MMAs of a tile of
// K = 512: 48.5 us against 39.8 for 32 experts, 16k ragged rows, N = 2048, K = 512.  A 32-byte store per lane straight
// from the row-per-lane layout, which needs d and ldd aligned to 32 bytes: 43.4 us.)
// `d_lane` points at row (lane & 24), column piece (lane & 7) of the warp's 32 rows x 64 columns.
__device__ __forceinline__ void store_rows(uint32_t (&o)[32], __nv_bfloat16* d_lane, int64_t ldd, uint32_t lane)
{
#pragma unroll
    for (uint32_t s = 1; s < 8; s <<= 1) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) {
            if ((c & s) != 0) continue;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                uint32_t& lo = o[4 * c + i];
                uint32_t& hi = o[4 * (c | s) + i];
                const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, s);
                if (up) lo = got;
                else hi = got;
            }
        }
    }
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
        *reinterpret_cast<uint4*>(d_lane + static_cast<int64_t>(c) * ldd) = make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
}

// 32 FP32 accumulator values x gw -> 16 BF16 pairs
__device__ __forceinline__ void scale_pack_bf16(const uint32_t (&v)[32], float g, uint32_t* out16)
{
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * i]) * g, __uint_as_float(v[2 * i + 1]) * g);
        out16[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

}  // namespace nvfp4::gemm
