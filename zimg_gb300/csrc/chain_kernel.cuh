// Tensor-core u16 resize with the two passes chained in registers (exact):
// the tiles and fragments of the chained kernel (chain_tma_kernel.cuh).
//
// Arithmetic is that of mma_kernel.cuh (re-centred fp16 samples, int16 taps
// split into two fp16 halves, fp32 accumulators that the planner proved hold
// exact integers, zimg's rounding and clamping per pass,
// resize_impl.cpp:31-42). The data flow differs: each warp owns one or more
// 16-column tiles of the CTA's strip of output columns and, per group of 16
// output rows, computes both passes itself without shared memory in between:
//
//   H first:  Dh[16 out cols][8 lines]  = Ah[16 out cols][16 in cols] * src[in cols][lines]
//             Dv[16 out rows][8 cols]   = Av[16 out rows][16 lines]   * Dh^T
//   V first:  Dv[16 out rows][8 in cols] = Av * src[lines][in cols]
//             Dh[16 out cols][8 rows]    = Ah * Dv^T
//
// The mma.m16n8k16 accumulator layout (row gid, columns 2tig, 2tig+1) is the
// layout of the B operand of the next product (k = 2tig, 2tig+1, n = gid), so
// the first product's rounded results, converted to centred fp16 pairs, are
// the second product's B fragments as they stand. Source lines stream through
// one ring of raw u16 lines per CTA and are centred to fp16 as they are read;
// results leave through per-warp staging tiles (stmatrix) as 16-byte rows.
#pragma once

#include "mma_kernel.cuh"

namespace zg {
namespace chain_detail {

using mma_detail::find_job;
using mma_detail::mma16816;
using mma_detail::pack_u16x2;
using mma_detail::u16x2_to_centred_h2;

// CTA shape: 7 computing warps and one producer warp at up to 128 registers
// each, two CTAs per SM. A strip is up to 7 warps' tiles.
constexpr int kWsWarps = 7;                // computing warps per CTA
constexpr int kTileW = 16;                 // output columns of one tile (one m16 block)

// Tiles per warp: several share the loop, the loads and the barriers, as far
// as their tap fragments fit in registers next to everything else: four for
// 16-line, 16-column windows (the 2x upscales), two for other small windows.
__host__ __device__ constexpr int tiles_per_warp(int kv, int kh)
{
	return (kv == 1 && kh == 1) ? 4 : ((kv + kh <= 3 || kh == 1) ? 2 : 1);
}

// A kernel instance by its code (FusedJob::variant): the pass order, windows of
// 16 kv lines and 16 kh columns, tiles per warp. kNarrowVariant has H first,
// windows of 16 by 16 and two tiles a warp: where four make strips too wide for one copy
// of their lines (above about 0.53 source samples an output), seven warps of
// two tiles are busy instead of four to six of four. 10-bit planes, bilinear:
// 40 of 640x360 -> 800x450 30.2 -> 24.1 us, 40 of 1280x720 -> 1760x990 74.2 ->
// 60.1 us. (V first, windows of 16 columns from a multiple of 8 have at most
// about half a source sample an output.) kEitherVariant, no job's own, runs such
// jobs and those of four tiles in one launch, where a batch has both: the body
// of four alone is 4 % faster (16 planes 1920x1080 -> 3840x2160 78.5 us, 81.5
// with both in it), two launches, or the mixed one, cost small batches more
// (1280x720 -> 1920x1080 and 1920x1080 -> 3840x2160, a plane each: 14.5 us,
// 20.5 in the mixed launch).
struct ChainVariant {
	bool h_first;
	int kv, kh, tiles;
};
constexpr int kChainKVMax = 3, kChainKHMax = 4;
constexpr int kChainShapes = kChainKVMax * kChainKHMax;
constexpr int kNarrowVariant = 2 * kChainShapes, kEitherVariant = kNarrowVariant + 1;
__host__ __device__ constexpr ChainVariant chain_variant_of(int code)
{
	if (code >= kNarrowVariant)
		return { true, 1, 1, code == kNarrowVariant ? 2 : 0 };
	const int kv = code % kChainShapes / kChainKHMax + 1, kh = code % kChainKHMax + 1;
	return { code >= kChainShapes, kv, kh, tiles_per_warp(kv, kh) };
}
constexpr int kStageBytes = 48;            // staged row: 16 u16 + pad (stmatrix rows without bank conflicts)
constexpr int kTileStage = 16 * kStageBytes + 32;       // a warp's staged tiles lie 32 mod 128 bytes apart

__device__ __forceinline__ void stsm_x4(void *p, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3)
{
	const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(p));
	asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};\n" ::"r"(s), "r"(r0), "r"(r1),
	             "r"(r2), "r"(r3)
	             : "memory");
}

__device__ __forceinline__ void stsm_x4_trans(void *p, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3)
{
	const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(p));
	asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};\n" ::"r"(s), "r"(r0),
	             "r"(r1), "r"(r2), "r"(r3)
	             : "memory");
}

// Stage reads and global stores of a warp's staged tiles, one 16-byte chunk
// per lane and store: with four tiles a store covers 4 rows x 128 bytes (row
// lane >> 3, tile (lane >> 1) & 3, half lane & 1); with two, 8 rows x 64
// bytes (rows q and q + 4, q = lane >> 3, tile (lane >> 1) & 1); with one,
// 16 rows x 32 bytes (rows q', q' + 2, q' + 4, q' + 6 of phase q). The staged
// tiles lie 32 mod 128 bytes apart, so the 8 lanes of a phase always read 8
// different 16-byte bank groups.
__host__ __device__ constexpr int store_rows(int tiles)
{
	return tiles == 4 ? 4 : (tiles == 2 ? 8 : 16);
}
__device__ __forceinline__ int store_row(int tiles, int lane)
{
	return tiles == 4 ? (lane >> 3)
	                  : (tiles == 2 ? (lane >> 3) + 4 * ((lane >> 2) & 1)
	                                : ((lane >> 3) & 1) + 8 * (lane >> 4) + 2 * ((lane >> 1) & 3));
}
__device__ __forceinline__ int store_tile(int tiles, int lane)
{
	return tiles == 4 ? (lane >> 1) & 3 : (tiles == 2 ? (lane >> 1) & 1 : 0);
}

} // namespace chain_detail
} // namespace zg
