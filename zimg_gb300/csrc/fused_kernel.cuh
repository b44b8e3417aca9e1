// The fused two-pass streaming kernel on CUDA cores (template). Instantiated
// per variant in fused_inst_*.cu.
//
// A work item is a strip of up to 128 output columns over consecutive
// streaming steps. Source lines enter a ring in shared memory (256 samples of
// each line) by cp.async a step ahead of use, as zimg's graph keeps a ring of
// lines per filter (zimg.h:387-396), so each source line is read from HBM once
// per strip.
//
//   V-first step (8 output rows):   ring (source lines) --V--> I --H--> destination
//   H-first step (16 output rows):  new source lines --H--> ring of
//                                   intermediate lines --V--> destination
//
// F32 planes: zimg's taps in its order, one fused multiply-add each. U16
// planes, any depth: zimg's int32 arithmetic; with taps that sum to 1 << 14,
// its sum(tap * (v - 32768)) + 8192 is sum(tap * v) + kInit, so raw samples
// stay as they are.
//
// Bound: issue slots and shared-memory bandwidth, not HBM; hence the layout.
//  - A thread's operands come in 16 bytes: in the vertical pass four columns
//    of a line and, in one record of the host's, two rows' taps of the line
//    with the line's place in the ring (no ring arithmetic in the loop); in
//    the horizontal pass four rows of a column. The intermediate block I
//    therefore holds four rows side by side per column, its columns dealt to
//    four planes (column x in plane x mod 4, kPlane apart), so that the
//    vertical pass's stores and the horizontal pass's loads at strides of 1
//    and 2 columns fall in different banks.
//  - A thread's horizontal taps and column offsets stay in registers for the
//    whole item. Multiply-adds are paired (two independent round-to-nearest
//    FMAs an instruction).
//
// Measured against the form before it (one row at a time through planar
// lines, ring slots computed per line, tap and sample loads of 4 bytes, u16
// lines of unaligned planes loaded sample by sample): 16 planes 3996x2160 ->
// 1998x1080 16-bit Spline36 930 -> 214 us; 6 planes 64x64 -> 6400x6400 f32
// Lanczos-3 275 -> 175 us; 96 planes 1920x1080 -> 1280x720 f32 bicubic 321 ->
// 279 us (shared-memory data path 68 % busy, a quarter of it bank conflicts of
// the horizontal pass at 1.5 columns' stride).
//
// The grid is persistent: in a batch CTAs take guided chunks of the units
// (work_chunks.cuh), otherwise an equal contiguous share each.
#pragma once

#include "fused.h"
#include "work_chunks.cuh"

namespace zg {
namespace fused_detail {

constexpr int kThreads = kStreamThreads;
constexpr int kWindow = kStreamWindow;               // source samples of a strip's line in the ring
constexpr int kPlane = 66;                           // columns of a plane of I: 2 mod 4, see above
constexpr int kBlockBytes = 4 * kPlane * 16;         // four rows of I
constexpr int kMidBytes = kStripW * 4;               // H first: a line of the intermediate ring
// 8192 - 32768 * (1 << 14): zimg's rounding term and the centring of raw samples
constexpr int kInit = 8192 - (1 << 29);

__device__ __forceinline__ uint32_t shared_addr(const void *p)
{
	return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, int src_bytes)
{
	const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
	if constexpr (BYTES == 16)
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes) : "memory");
	else
		asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gmem), "n"(BYTES), "r"(src_bytes)
		             : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
	asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait()
{
	asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// zimg's rounding (pack_pixel_u16, resize_impl.cpp:36-42) of
// 8192 + sum(tap * (v - 32768)), clamped to [0, pixel_max].
__device__ __forceinline__ int u16_round(int acc, int pixel_max)
{
	return min(max((acc >> 14) + 32768, 0), pixel_max);
}

__device__ __forceinline__ int find_job(const FusedJob *__restrict__ jobs, int num_jobs, int t)
{
	int lo = 0, hi = num_jobs - 1;
	while (lo < hi) {
		const int mid = (lo + hi + 1) >> 1;
		if (jobs[mid].item_begin <= t)
			lo = mid;
		else
			hi = mid - 1;
	}
	return lo;
}

// Registers-resident description of one work item.
struct Item {
	const char *src;
	ptrdiff_t src_stride;
	char *dst;
	ptrdiff_t dst_stride;
	const char *records;
	const int2 *ranges;
	int src_w, src_h, dst_h, src_align, dst_vec;
	int c0, cols_valid, xlo, pxa;
	int step0, steps, ring_rows, in_rows;
	bool late;
	int pixel_max;
};

// Units t .. t_end - 1 of job J that lie in the strip of unit t: a work item.
// A job's units are its (strip, streaming step) pairs, strip-major.
__device__ __forceinline__ Item make_item(const FusedJob &J, int t, int t_end)
{
	Item it;
	const int local = t - J.item_begin;
	const int strip = local / J.segments;
	it.step0 = local - strip * J.segments;
	it.steps = min(J.segments - it.step0, t_end - t);
	it.src = static_cast<const char *>(J.src);
	it.src_stride = J.src_stride;
	it.dst = static_cast<char *>(J.dst);
	it.dst_stride = J.dst_stride;
	it.records = reinterpret_cast<const char *>(J.v_dense);
	it.ranges = reinterpret_cast<const int2 *>(J.v_base);
	it.src_w = J.src_w;
	it.src_h = J.src_h;
	it.dst_h = J.dst_h;
	it.src_align = J.src_align;
	it.dst_vec = J.dst_align >= (J.kind == static_cast<int>(FusedKind::F32) ? 16 : 8);
	it.c0 = strip * J.strip_w;
	it.cols_valid = min(J.strip_w, J.dst_w - it.c0);
	it.xlo = __ldg(J.win_col + 2 * strip);
	it.pxa = (__ldg(J.win_col + 2 * strip + 1) - it.xlo + 7) & ~7;
	it.ring_rows = J.ring_rows;
	it.in_rows = J.in_rows;
	it.late = J.depth == 0;
	it.pixel_max = static_cast<int>(J.pixel_max);
	return it;
}

// A 16-byte chunk of a line whose samples start 2 mod 4 bytes off a word, or
// on one: aligned 4-byte loads and a shift where the chunk and the samples
// beside it lie in the line, else sample by sample. Zeros outside the plane.
__device__ __forceinline__ uint4 load_chunk_u16(const uint16_t *row, int gx, int src_w)
{
	uint32_t w[4];
	const bool odd = (reinterpret_cast<uintptr_t>(row + gx) & 2) != 0;
	if (gx >= 1 && gx + 9 <= src_w) {
		const uint32_t *p = reinterpret_cast<const uint32_t *>(row + gx - (odd ? 1 : 0));
		uint32_t v[5];
#pragma unroll
		for (int k = 0; k < 4; ++k)
			v[k] = __ldg(p + k);
		v[4] = odd ? __ldg(p + 4) : 0u;
#pragma unroll
		for (int k = 0; k < 4; ++k)
			w[k] = odd ? __byte_perm(v[k], v[k + 1], 0x5432) : v[k];
	} else {
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			const int x = gx + 2 * k;
			const uint32_t lo = x < src_w ? __ldg(row + x) : 0u, hi = x + 1 < src_w ? __ldg(row + x + 1) : 0u;
			w[k] = lo | (hi << 16);
		}
	}
	return make_uint4(w[0], w[1], w[2], w[3]);
}

// Source lines [a, b) of the strip into slots of a ring of `rows` lines, zero
// outside the plane; line a goes to slot `slot`. A thread copies one 16-byte
// chunk of every kLines-th line, with the widest copies that the plane's
// alignment allows.
template <int E>
__device__ __forceinline__ void load_lines(const Item &it, int a, int b, char *ring, int rows, int slot)
{
	constexpr int kPer = 16 / E;                       // samples a chunk
	constexpr int kChunks = kWindow / kPer;            // chunks a line
	constexpr int kLines = kThreads / kChunks;         // lines a pass
	const int q = threadIdx.x % kChunks, l0 = threadIdx.x / kChunks;
	if (q * kPer >= it.pxa)
		return;
	const int gx = it.xlo + q * kPer;
	const int nb = max(0, min(kPer, it.src_w - gx)) * E;
	slot += l0;
	slot = slot >= rows ? slot - rows : slot;
	const char *src = it.src + static_cast<ptrdiff_t>(a + l0) * it.src_stride + static_cast<ptrdiff_t>(gx) * E;
	const ptrdiff_t step = kLines * it.src_stride;
	if (it.src_align == 16) {
		const uint32_t base = shared_addr(ring) + q * 16, end = base + rows * (kWindow * E);
		uint32_t d = base + slot * (kWindow * E);
		if (nb == 16 && b <= it.src_h) {
#pragma unroll 2
			for (int y = a + l0; y < b; y += kLines) {
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
				src += step;
				d += kLines * (kWindow * E);
				d = d >= end ? d - rows * (kWindow * E) : d;
			}
			return;
		}
		if (!nb)
			src = it.src;
		for (int y = a + l0; y < b; y += kLines) {
			const int n = y < it.src_h ? nb : 0;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(n ? src : it.src), "r"(n) : "memory");
			src += step;
			d += kLines * (kWindow * E);
			d = d >= end ? d - rows * (kWindow * E) : d;
		}
		return;
	}
	for (int y = a + l0; y < b; y += kLines, src += step) {
		char *d = ring + slot * (kWindow * E) + q * 16;
		slot += kLines;
		slot = slot >= rows ? slot - rows : slot;
		const int n = y < it.src_h ? nb : 0;
		if (it.src_align == 8) {
#pragma unroll
			for (int k = 0; k < 2; ++k) {
				const int m = max(0, min(8, n - 8 * k));
				cp_async<8>(d + 8 * k, m ? src + 8 * k : it.src, m);
			}
		} else if (E == 4 || it.src_align == 4) {
#pragma unroll
			for (int k = 0; k < 4; ++k) {
				const int m = max(0, min(4, n - 4 * k));
				cp_async<4>(d + 4 * k, m ? src + 4 * k : it.src, m);
			}
		} else {
			uint4 v = make_uint4(0, 0, 0, 0);
			if (n)
				v = load_chunk_u16(reinterpret_cast<const uint16_t *>(src) - gx, gx, it.src_w);
			*reinterpret_cast<uint4 *>(d) = v;
		}
	}
}

// `bytes` (a multiple of 16) of a step's records.
__device__ __forceinline__ void load_records(const char *src, char *dst, int bytes)
{
	for (int i = threadIdx.x * 16; i < bytes; i += kThreads * 16)
		cp_async<16>(dst + i, src + i, 16);
}

// Loads by 32-bit shared address (no generic address arithmetic in the loops).
__device__ __forceinline__ float4 lds_f4(uint32_t a)
{
	float4 v;
	asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
	return v;
}

__device__ __forceinline__ int4 lds_i4(uint32_t a)
{
	int4 v;
	asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
	return v;
}

__device__ __forceinline__ uint2 lds_u2(uint32_t a)
{
	uint2 v;
	asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a));
	return v;
}

__device__ __forceinline__ uint32_t lds_u1(uint32_t a)
{
	uint32_t v;
	asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a));
	return v;
}

__device__ __forceinline__ int lds_u16(uint32_t a)
{
	uint16_t v;
	asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a));
	return v;
}

__device__ __forceinline__ void sts_f4(uint32_t a, float x, float y, float z, float w)
{
	asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

__device__ __forceinline__ float2 dup(float x)
{
	return make_float2(x, x);
}

// V first, vertical pass: thread = four columns (quad q) of four rows (half 0
// or 1 of the step's eight), two groups of two rows. A group's record: the two rows' taps of each line of its
// window, then the lines' byte offsets in the ring. The paired FMAs take the
// two rows of a column, so that four rows end up side by side as I has them.
template <bool INT, int VS>
__device__ __forceinline__ void vfirst_v(const Item &it, uint32_t ring, uint32_t records, uint32_t I, int q, int half)
{
	if (half >= 2)
		return;
	constexpr int kRecord = stream_record_bytes(false, VS), kTaps = 8;
	const uint32_t col = ring + q * (INT ? 8 : 16);
	float2 out[2][4];  // [group][column]: the group's two rows (INT: int bits)
#pragma unroll
	for (int g = 0; g < 2; ++g) {
		const uint32_t rec = records + (2 * half + g) * kRecord;
		if constexpr (INT) {
			int acc[2][4];
#pragma unroll
			for (int j = 0; j < 2; ++j)
#pragma unroll
				for (int e = 0; e < 4; ++e)
					acc[j][e] = kInit;
#pragma unroll (VS <= 8 ? 2 : 1)
			for (int s4 = 0; s4 < VS; s4 += 4) {
				const int4 o = lds_i4(rec + VS * kTaps + s4 * 4);
				const int at[4] = { o.x, o.y, o.z, o.w };
#pragma unroll
				for (int s2 = 0; s2 < 4; s2 += 2) {
					const int4 r = lds_i4(rec + (s4 + s2) * kTaps);
					const int tap[2][2] = { { r.x, r.y }, { r.z, r.w } };
#pragma unroll
					for (int i = 0; i < 2; ++i) {
						const uint2 x = lds_u2(col + at[s2 + i]);
						const int v[4] = { static_cast<int>(x.x & 0xFFFFu), static_cast<int>(x.x >> 16),
						                   static_cast<int>(x.y & 0xFFFFu), static_cast<int>(x.y >> 16) };
#pragma unroll
						for (int e = 0; e < 4; ++e) {
							acc[0][e] += tap[i][0] * v[e];
							acc[1][e] += tap[i][1] * v[e];
						}
					}
				}
			}
#pragma unroll
			for (int e = 0; e < 4; ++e)
				out[g][e] = make_float2(__int_as_float(u16_round(acc[0][e], it.pixel_max)),
				                        __int_as_float(u16_round(acc[1][e], it.pixel_max)));
		} else {
#pragma unroll
			for (int e = 0; e < 4; ++e)
				out[g][e] = dup(0.0f);
#pragma unroll (VS <= 8 ? 2 : 1)
			for (int s4 = 0; s4 < VS; s4 += 4) {
				const int4 o = lds_i4(rec + VS * kTaps + s4 * 4);
				const int at[4] = { o.x, o.y, o.z, o.w };
#pragma unroll
				for (int s2 = 0; s2 < 4; s2 += 2) {
					const float4 r = lds_f4(rec + (s4 + s2) * kTaps);
					const float2 tap[2] = { make_float2(r.x, r.y), make_float2(r.z, r.w) };
#pragma unroll
					for (int i = 0; i < 2; ++i) {
						const float4 x = lds_f4(col + at[s2 + i]);
						out[g][0] = __ffma2_rn(dup(x.x), tap[i], out[g][0]);
						out[g][1] = __ffma2_rn(dup(x.y), tap[i], out[g][1]);
						out[g][2] = __ffma2_rn(dup(x.z), tap[i], out[g][2]);
						out[g][3] = __ffma2_rn(dup(x.w), tap[i], out[g][3]);
					}
				}
			}
		}
	}
	const uint32_t d = I + half * kBlockBytes + q * 16;
#pragma unroll
	for (int e = 0; e < 4; ++e)
		sts_f4(d + e * (kPlane * 16), out[0][e].x, out[0][e].y, out[1][e].x, out[1][e].y);
}

// V first, horizontal pass: thread = one output column of eight rows.
// at[k]: address in I of the column of tap k.
template <bool INT, int HW>
__device__ __forceinline__ void vfirst_h(const Item &it, const float (&taps)[HW], const uint32_t (&at)[HW], int row0)
{
	const int c = threadIdx.x;
	if (c >= it.cols_valid)
		return;
	constexpr int E = INT ? 2 : 4;
	char *d = it.dst + static_cast<ptrdiff_t>(row0) * it.dst_stride + static_cast<ptrdiff_t>(it.c0 + c) * E;
	const int rows = it.dst_h - row0;
#pragma unroll
	for (int b = 0; b < 2; ++b) {
		float v[4];
		if constexpr (INT) {
			int acc[4] = { kInit, kInit, kInit, kInit };
#pragma unroll
			for (int k = 0; k < HW; ++k) {
				const int4 x = lds_i4(at[k] + b * kBlockBytes);
				const int t = __float_as_int(taps[k]);
				acc[0] += t * x.x;
				acc[1] += t * x.y;
				acc[2] += t * x.z;
				acc[3] += t * x.w;
			}
#pragma unroll
			for (int j = 0; j < 4; ++j)
				v[j] = __int_as_float(u16_round(acc[j], it.pixel_max));
		} else {
			float2 a01 = dup(0.0f), a23 = dup(0.0f);
#pragma unroll
			for (int k = 0; k < HW; ++k) {
				const float4 x = lds_f4(at[k] + b * kBlockBytes);
				a01 = __ffma2_rn(dup(taps[k]), make_float2(x.x, x.y), a01);
				a23 = __ffma2_rn(dup(taps[k]), make_float2(x.z, x.w), a23);
			}
			v[0] = a01.x;
			v[1] = a01.y;
			v[2] = a23.x;
			v[3] = a23.y;
		}
		auto store = [&](int j) {
			if constexpr (INT)
				*reinterpret_cast<uint16_t *>(d) = static_cast<uint16_t>(__float_as_int(v[j]));
			else
				*reinterpret_cast<float *>(d) = v[j];
			d += it.dst_stride;
		};
		if (4 * b + 4 <= rows) {
#pragma unroll
			for (int j = 0; j < 4; ++j)
				store(j);
		} else {
			for (int j = 0; j < 4; ++j)
				if (4 * b + j < rows)
					store(j);
		}
	}
}

// H first, horizontal pass: lines [a, b) (multiples of 4) from the ring of
// source lines into the intermediate ring; thread = one output column, four
// lines at a time. l: the column's first input in the strip's lines.
template <bool INT, int HW>
__device__ __forceinline__ void hfirst_h(const Item &it, uint32_t in, const float (&taps)[HW], int l, int a, int b,
                                         int in_slot, char *mid, int mid_slot)
{
	constexpr int E = INT ? 2 : 4, LB = kWindow * E;
	const int c = threadIdx.x;
	for (int y = a; y < b; y += 4) {
		const uint32_t r = in + in_slot * LB + l * E;
		float v[4];
		if constexpr (INT) {
			int acc[4] = { kInit, kInit, kInit, kInit };
#pragma unroll
			for (int k = 0; k < HW; ++k) {
				const int t = __float_as_int(taps[k]);
#pragma unroll
				for (int i = 0; i < 4; ++i)
					acc[i] += t * lds_u16(r + i * LB + k * 2);
			}
#pragma unroll
			for (int i = 0; i < 4; ++i)
				v[i] = __int_as_float(u16_round(acc[i], it.pixel_max));
		} else {
			float2 a01 = dup(0.0f), a23 = dup(0.0f);
#pragma unroll
			for (int k = 0; k < HW; ++k) {
				float x[4];
#pragma unroll
				for (int i = 0; i < 4; ++i)
					x[i] = __uint_as_float(lds_u1(r + i * LB + k * 4));
				a01 = __ffma2_rn(dup(taps[k]), make_float2(x[0], x[1]), a01);
				a23 = __ffma2_rn(dup(taps[k]), make_float2(x[2], x[3]), a23);
			}
			v[0] = a01.x;
			v[1] = a01.y;
			v[2] = a23.x;
			v[3] = a23.y;
		}
		char *d = mid + mid_slot * kMidBytes + c * 4;
#pragma unroll
		for (int i = 0; i < 4; ++i)
			*reinterpret_cast<float *>(d + i * kMidBytes) = v[i];
		in_slot = in_slot + 4 >= it.in_rows ? 0 : in_slot + 4;
		mid_slot = mid_slot + 4 >= it.ring_rows ? 0 : mid_slot + 4;
	}
}

// H first, vertical pass: a warp takes a group of four output rows, a lane
// four columns. A group's record: the four rows' taps of each line of its
// window, then the lines' byte offsets in the intermediate ring.
template <bool INT, int VS>
__device__ __forceinline__ void hfirst_v(const Item &it, uint32_t mid, uint32_t records, int row0)
{
	const int warp = threadIdx.x >> 5, q = threadIdx.x & 31;
	const int r0 = row0 + 4 * warp;
	if (r0 >= it.dst_h || 4 * q >= it.cols_valid)
		return;
	constexpr int E = INT ? 2 : 4;
	constexpr int kTaps = 16;
	const uint32_t rec = records + warp * stream_record_bytes(true, VS);
	const uint32_t col = mid + q * 16;
	char *d = it.dst + static_cast<ptrdiff_t>(r0) * it.dst_stride + static_cast<ptrdiff_t>(it.c0 + 4 * q) * E;
	const bool wide = it.dst_vec && 4 * q + 4 <= it.cols_valid;
	float out[4][4];  // [row][column]
	if constexpr (INT) {
		int acc[4][4];
#pragma unroll
		for (int j = 0; j < 4; ++j)
#pragma unroll
			for (int e = 0; e < 4; ++e)
				acc[j][e] = kInit;
#pragma unroll (VS <= 8 ? 2 : 1)
		for (int s4 = 0; s4 < VS; s4 += 4) {
			const int4 o = lds_i4(rec + VS * kTaps + s4 * 4);
			const int at[4] = { o.x, o.y, o.z, o.w };
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const int4 t = lds_i4(rec + (s4 + i) * kTaps);
				const int4 x = lds_i4(col + at[i]);
				const int tj[4] = { t.x, t.y, t.z, t.w };
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					acc[j][0] += tj[j] * x.x;
					acc[j][1] += tj[j] * x.y;
					acc[j][2] += tj[j] * x.z;
					acc[j][3] += tj[j] * x.w;
				}
			}
		}
#pragma unroll
		for (int j = 0; j < 4; ++j)
#pragma unroll
			for (int e = 0; e < 4; ++e)
				out[j][e] = __int_as_float(u16_round(acc[j][e], it.pixel_max));
	} else {
		float2 acc[4][2];
#pragma unroll
		for (int j = 0; j < 4; ++j)
			acc[j][0] = acc[j][1] = dup(0.0f);
#pragma unroll (VS <= 8 ? 2 : 1)
		for (int s4 = 0; s4 < VS; s4 += 4) {
			const int4 o = lds_i4(rec + VS * kTaps + s4 * 4);
			const int at[4] = { o.x, o.y, o.z, o.w };
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const float4 t = lds_f4(rec + (s4 + i) * kTaps);
				const float4 x = lds_f4(col + at[i]);
				const float2 x01 = make_float2(x.x, x.y), x23 = make_float2(x.z, x.w);
				const float tj[4] = { t.x, t.y, t.z, t.w };
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					acc[j][0] = __ffma2_rn(dup(tj[j]), x01, acc[j][0]);
					acc[j][1] = __ffma2_rn(dup(tj[j]), x23, acc[j][1]);
				}
			}
		}
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			out[j][0] = acc[j][0].x;
			out[j][1] = acc[j][0].y;
			out[j][2] = acc[j][1].x;
			out[j][3] = acc[j][1].y;
		}
	}
#pragma unroll
	for (int j = 0; j < 4; ++j, d += it.dst_stride) {
		if (r0 + j >= it.dst_h)
			break;
		if constexpr (INT) {
			uint32_t u[4];
#pragma unroll
			for (int e = 0; e < 4; ++e)
				u[e] = static_cast<uint32_t>(__float_as_int(out[j][e]));
			if (wide) {
				*reinterpret_cast<uint2 *>(d) = make_uint2(u[0] | (u[1] << 16), u[2] | (u[3] << 16));
			} else {
#pragma unroll
				for (int e = 0; e < 4; ++e)
					if (4 * q + e < it.cols_valid)
						reinterpret_cast<uint16_t *>(d)[e] = static_cast<uint16_t>(u[e]);
			}
		} else if (wide) {
			*reinterpret_cast<float4 *>(d) = make_float4(out[j][0], out[j][1], out[j][2], out[j][3]);
		} else {
#pragma unroll
			for (int e = 0; e < 4; ++e)
				if (4 * q + e < it.cols_valid)
					reinterpret_cast<float *>(d)[e] = out[j][e];
		}
	}
}

template <bool H_FIRST, bool INT, int HW, int VS>
__global__ void __launch_bounds__(kThreads, HW <= 8 ? 5 : 4)
fused_kernel(const FusedJob *__restrict__ jobs, int num_jobs, int total_items, const __grid_constant__ FewJobs few,
             const __grid_constant__ SmemLayout L, const __grid_constant__ WorkChunks C)
{
	constexpr int E = INT ? 2 : 4;
	constexpr int kStepRows = stream_step_rows(H_FIRST);
	constexpr int kRecordBytes = 4 * stream_record_bytes(H_FIRST, VS);  // a step's four groups
	constexpr int kRecordBuffers = stream_record_buffers(H_FIRST);
	extern __shared__ float4 smem4[];
	char *smem = reinterpret_cast<char *>(smem4);
	char *in = smem + L.in_off;      // source lines
	char *mid = smem + L.ring_off;   // V first: I; H first: the intermediate ring
	char *records = smem + L.vcoef_off;
	const uint32_t in_a = shared_addr(in), mid_a = shared_addr(mid), records_a = shared_addr(records);

	// the launch's units in job / strip / step order: guided chunks
	// (C.sched), or this CTA's equal share
	__shared__ int chunk;
	int c_begin = static_cast<int>(static_cast<long long>(blockIdx.x) * total_items / gridDim.x);
	int c_end = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * total_items / gridDim.x);
	for (bool first = true;; first = false) {
		if (C.sched) {
			const int m = next_chunk(C, &chunk);
			if (m < 0)
				break;
			c_begin = __ldg(C.bounds + m);
			c_end = __ldg(C.bounds + m + 1);
		} else if (!first) {
			break;
		}
		for (int t = c_begin; t < c_end;) {
			const FusedJob *table = jobs ? jobs : few.job;
			const FusedJob &J = table[find_job(table, num_jobs, t)];
			const Item it = make_item(J, t, c_end);
			t += it.steps;

			// lines and records of a step, one cp.async group; `next`, `slot`:
			// the first line not yet in the ring and its slot
			int next, slot;
			auto load_step = [&](int k, int rec) {
				const int hi = __ldg(it.ranges + it.step0 + k).y;
				if (hi > next) {
					load_lines<E>(it, next, hi, in, it.in_rows, slot);
					slot += hi - next;
					while (slot >= it.in_rows)
						slot -= it.in_rows;
					next = hi;
				}
				load_records(it.records + static_cast<size_t>(it.step0 + k) * kRecordBytes,
				             records + (H_FIRST ? rec : (k & 1) * kRecordBytes), kRecordBytes);
				cp_async_commit();
			};
			next = __ldg(it.ranges + it.step0).x;
			slot = next % it.in_rows;
			int h_line = next, h_in = slot, h_mid = H_FIRST ? next % it.ring_rows : 0;
			load_step(0, 0);

			// this thread's output column: taps, and where its inputs are
			const int c = min(static_cast<int>(threadIdx.x), it.cols_valid - 1);
			const int left = __ldg(J.h_left + it.c0 + c) - it.xlo;
			float taps[HW];
			const float *tp = J.h_taps + static_cast<size_t>(it.c0 + c) * HW;
#pragma unroll
			for (int k = 0; k < HW; ++k)
				taps[k] = __ldg(tp + k);
			// V first: this thread's part of the vertical pass, its inputs in I
			uint32_t at[H_FIRST ? 1 : HW];
			int q = 0, half = 0;
			if constexpr (!H_FIRST) {
				const int quads = it.pxa / 4;
				q = static_cast<int>(threadIdx.x) % quads;
				half = static_cast<int>(threadIdx.x) / quads;
#pragma unroll
				for (int k = 0; k < HW; ++k)
					at[k] = mid_a + (((left + k) & 3) * kPlane + ((left + k) >> 2)) * 16;
			}

			int rec_at = 0;
			for (int k = 0; k < it.steps; ++k) {
				// early: the next step's lines go into slots that no line of
				// this one's windows holds; late: only after its vertical
				// pass (H first: horizontal pass). Records: H first, a warp may
				// still read those of the step before this one.
				const bool more = k + 1 < it.steps;
				int rec_next = 0;
				if constexpr (H_FIRST)
					rec_next = rec_at == (kRecordBuffers - 1) * kRecordBytes ? 0 : rec_at + kRecordBytes;
				if (more && !it.late) {
					load_step(k + 1, rec_next);
					cp_async_wait<1>();
				} else {
					cp_async_wait<0>();
				}
				__syncthreads();
				const int row0 = (it.step0 + k) * kStepRows;
				const uint32_t rec = records_a + (H_FIRST ? rec_at : (k & 1) * kRecordBytes);
				if constexpr (H_FIRST) {
					const int hi = __ldg(it.ranges + it.step0 + k).y;
					if (hi > h_line) {
						hfirst_h<INT, HW>(it, in_a, taps, left, h_line, hi, h_in, mid, h_mid);
						h_in = (h_in + (hi - h_line)) % it.in_rows;
						h_mid = (h_mid + (hi - h_line)) % it.ring_rows;
						h_line = hi;
					}
				} else {
					vfirst_v<INT, VS>(it, in_a, rec, mid_a, q, half);
				}
				__syncthreads();
				if (more && it.late)
					load_step(k + 1, rec_next);
				if constexpr (H_FIRST)
					hfirst_v<INT, VS>(it, mid_a, rec, row0);
				else
					vfirst_h<INT, HW>(it, taps, at, row0);
				rec_at = rec_next;
			}
			__syncthreads();  // the next item reuses every buffer
		}
	}
	if (C.sched)
		chunks_finish(C);
}

} // namespace fused_detail
} // namespace zg
