// Single-pass resize kernels: one horizontal or vertical banded pass over whole
// planes, for any tap count. These are the general path (and the building
// block of two-pass conversions whose intermediate lives in HBM).
//
// Arithmetic, per output sample, is exactly zimg's C path
// (src/zimg/resize/resize_impl.cpp:31-114):
//   u16: int32 sum of int16 tap * (x - 32768), then ((sum + 8192) >> 14) + 32768
//        clamped to [0, 2^depth - 1]  -> bit-exact;
//   f32: taps applied in order k = 0..width-1 with a fused multiply-add per tap.
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace zg {

namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ uint16_t pack_u16(uint32_t acc, int32_t pixel_max)
{
	int32_t x = (static_cast<int32_t>(acc + 8192u) >> 14) + 32768;
	x = min(max(x, 0), pixel_max);
	return static_cast<uint16_t>(x);
}

// The block's plane: planes of one size and filter run in one launch, one to
// a grid layer. A batch's planes, small ones above all, were bound by a launch
// for each of their passes: a call of 9 4:2:0 frames 496x210 -> 216x92, 17
// taps, 187 -> 19 us, of 32 f32 planes 1920x1080 -> 480x270, Lanczos-3, 426 ->
// 142 us (with the kernels for up to kRegTaps taps below).
#define ZG_PASS_PLANE                                                          \
	const uint8_t *const src = static_cast<const uint8_t *>(P.p[blockIdx.z].src); \
	const ptrdiff_t ss = P.p[blockIdx.z].src_stride;                             \
	uint8_t *const dst = static_cast<uint8_t *>(P.p[blockIdx.z].dst);            \
	const ptrdiff_t ds = P.p[blockIdx.z].dst_stride;

// ---------------------------------------------------------------- vertical --
// Thread = VEC adjacent columns; block = kThreads * VEC columns x `rows_per_block`
// output rows. Every load of a row segment is coalesced across the warp.
template <int VEC>
__global__ void __launch_bounds__(kThreads)
v_u16_kernel(PassTables t, int32_t pixel_max, unsigned plane_w, const __grid_constant__ PassPlanes P,
             unsigned rows_per_block)
{
	ZG_PASS_PLANE
	const unsigned j0 = (blockIdx.x * kThreads + threadIdx.x) * VEC;
	if (j0 >= plane_w)
		return;
	const bool full = j0 + VEC <= plane_w;
	const unsigned i0 = blockIdx.y * rows_per_block;
	const unsigned i1 = min(i0 + rows_per_block, t.rows);

	for (unsigned i = i0; i < i1; ++i) {
		const unsigned top = __ldg(t.left + i);
		const int16_t *c = t.i16 + static_cast<size_t>(i) * t.width;
		uint32_t acc[VEC];
		const uint32_t b = static_cast<uint32_t>(__ldg(t.bias + i));
#pragma unroll
		for (int v = 0; v < VEC; ++v)
			acc[v] = b;

		const uint8_t *row = src + static_cast<ptrdiff_t>(top) * ss + static_cast<size_t>(j0) * 2;
		for (unsigned k = 0; k < t.width; ++k, row += ss) {
			const int32_t ck = __ldg(c + k);
			if (VEC == 8 && full) {
				uint4 q = __ldg(reinterpret_cast<const uint4 *>(row));
				const uint32_t w[4] = { q.x, q.y, q.z, q.w };
#pragma unroll
				for (int v = 0; v < 4; ++v) {
					acc[2 * v] += static_cast<uint32_t>(ck * static_cast<int32_t>(w[v] & 0xFFFFu));
					acc[2 * v + 1] += static_cast<uint32_t>(ck * static_cast<int32_t>(w[v] >> 16));
				}
			} else {
				const uint16_t *r16 = reinterpret_cast<const uint16_t *>(row);
#pragma unroll
				for (int v = 0; v < VEC; ++v)
					if (full || j0 + v < plane_w)
						acc[v] += static_cast<uint32_t>(ck * static_cast<int32_t>(__ldg(r16 + v)));
			}
		}

		uint16_t *out = reinterpret_cast<uint16_t *>(dst + static_cast<ptrdiff_t>(i) * ds) + j0;
		if (VEC == 8 && full) {
			uint32_t w[4];
#pragma unroll
			for (int v = 0; v < 4; ++v)
				w[v] = pack_u16(acc[2 * v], pixel_max) | (static_cast<uint32_t>(pack_u16(acc[2 * v + 1], pixel_max)) << 16);
			*reinterpret_cast<uint4 *>(out) = make_uint4(w[0], w[1], w[2], w[3]);
		} else {
#pragma unroll
			for (int v = 0; v < VEC; ++v)
				if (full || j0 + v < plane_w)
					out[v] = pack_u16(acc[v], pixel_max);
		}
	}
}

// Planes that are not 16-byte aligned, a column a thread (see v_reg_kernel and
// v_f32_dense_kernel for the others).
__global__ void __launch_bounds__(kThreads)
v_f32_kernel(PassTables t, unsigned plane_w, const __grid_constant__ PassPlanes P, unsigned rows_per_block)
{
	ZG_PASS_PLANE
	const unsigned j = blockIdx.x * kThreads + threadIdx.x;
	if (j >= plane_w)
		return;
	const unsigned i0 = blockIdx.y * rows_per_block;
	const unsigned i1 = min(i0 + rows_per_block, t.rows);

	for (unsigned i = i0; i < i1; ++i) {
		const float *c = t.f32 + static_cast<size_t>(i) * t.width;
		const uint8_t *row = src + static_cast<ptrdiff_t>(__ldg(t.left + i)) * ss + static_cast<size_t>(j) * 4;
		float acc = 0.0f;
		for (unsigned k = 0; k < t.width; ++k, row += ss)
			acc = __fmaf_rn(__ldg(c + k), __ldg(reinterpret_cast<const float *>(row)), acc);
		reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(i) * ds)[j] = acc;
	}
}

// -------------------------------------------------------------- horizontal --
// Filters longer than kRegTaps: thread = one output column for
// `rows_per_block` lines; its taps stay in L1.
__global__ void __launch_bounds__(kThreads)
h_u16_kernel(PassTables t, int32_t pixel_max, unsigned lines, const __grid_constant__ PassPlanes P,
             unsigned rows_per_block)
{
	ZG_PASS_PLANE
	const unsigned j = blockIdx.x * kThreads + threadIdx.x;
	if (j >= t.rows)
		return;
	const unsigned l = __ldg(t.left + j);
	const int16_t *c = t.i16 + static_cast<size_t>(j) * t.width;
	const uint32_t b = static_cast<uint32_t>(__ldg(t.bias + j));
	const unsigned r0 = blockIdx.y * rows_per_block;
	const unsigned r1 = min(r0 + rows_per_block, lines);
	for (unsigned r = r0; r < r1; ++r) {
		const uint16_t *s = reinterpret_cast<const uint16_t *>(src + static_cast<ptrdiff_t>(r) * ss) + l;
		uint32_t acc = b;
		for (unsigned k = 0; k < t.width; ++k)
			acc += static_cast<uint32_t>(static_cast<int32_t>(__ldg(c + k)) * static_cast<int32_t>(__ldg(s + k)));
		reinterpret_cast<uint16_t *>(dst + static_cast<ptrdiff_t>(r) * ds)[j] = pack_u16(acc, pixel_max);
	}
}

__global__ void __launch_bounds__(kThreads)
h_f32_kernel(PassTables t, unsigned lines, const __grid_constant__ PassPlanes P,
             unsigned rows_per_block)
{
	ZG_PASS_PLANE
	const unsigned j = blockIdx.x * kThreads + threadIdx.x;
	if (j >= t.rows)
		return;
	const unsigned l = __ldg(t.left + j);
	const float *c = t.f32 + static_cast<size_t>(j) * t.width;
	const unsigned r0 = blockIdx.y * rows_per_block;
	const unsigned r1 = min(r0 + rows_per_block, lines);
	for (unsigned r = r0; r < r1; ++r) {
		const float *s = reinterpret_cast<const float *>(src + static_cast<ptrdiff_t>(r) * ss) + l;
		float acc = 0.0f;
		for (unsigned k = 0; k < t.width; ++k)
			acc = __fmaf_rn(__ldg(c + k), __ldg(s + k), acc);
		reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(r) * ds)[j] = acc;
	}
}

// Up to kRegTaps taps: thread = one output column of kRegRows lines, its taps
// in registers (the width is built in, so that no sample outside an output's
// own taps is read), the loads of kRegBatch lines in flight together. The
// kernels above, left for longer filters, spend two loads and the loop on each
// multiply-add, one line at a time. Bound: a 2- or 4-byte load per tap.
// Measured, one plane, horizontal pass alone, before and now:
//   u16 960x1080 -> 1920x1080, 6 taps    9.0 -> 5.3 us
//   u16 1920x1080 -> 1279x1080, 10 taps  8.0 -> 5.6 us
//   f32 960x1080 -> 1920x1080, 6 taps    8.9 -> 4.5 us
//   f32 3840x2160 -> 1920x2160, 8 taps   40 -> 17 us
//   f32 1920x1080 -> 960x1080, 16 taps   39 -> 11 us
//   u16 1920x1080 -> 640x1080, 17 taps   8.3 -> 5.3 us
//   u16 1920x1080 -> 384x1080, 29 taps   10.5 -> 6.1 us
//   f32 1920x1080 -> 479x1080, 26 taps   18.0 -> 10.8 us
constexpr int kRegTaps = 32;
constexpr unsigned kRegRows = 8;
constexpr unsigned kRegBatch = 4;

template <bool INT, int W>
__global__ void __launch_bounds__(kThreads)
h_reg_kernel(PassTables t, int32_t pixel_max, unsigned lines, const __grid_constant__ PassPlanes P)
{
	ZG_PASS_PLANE
	using S = std::conditional_t<INT, uint16_t, float>;
	using A = std::conditional_t<INT, int32_t, float>;
	const unsigned j = blockIdx.x * kThreads + threadIdx.x;
	if (j >= t.rows)
		return;
	const unsigned l = __ldg(t.left + j);
	A c[W];
#pragma unroll
	for (int k = 0; k < W; ++k) {
		if constexpr (INT)
			c[k] = __ldg(t.i16 + static_cast<size_t>(j) * W + k);
		else
			c[k] = __ldg(t.f32 + static_cast<size_t>(j) * W + k);
	}
	const uint32_t b = INT ? static_cast<uint32_t>(__ldg(t.bias + j)) : 0u;
	const unsigned r0 = blockIdx.y * kRegRows, r1 = min(r0 + kRegRows, lines);
	for (unsigned r = r0; r < r1; r += kRegBatch) {
		S x[kRegBatch][W];
#pragma unroll
		for (unsigned q = 0; q < kRegBatch; ++q) {
			const S *s = reinterpret_cast<const S *>(src + static_cast<ptrdiff_t>(min(r + q, r1 - 1)) * ss) + l;
#pragma unroll
			for (int k = 0; k < W; ++k)
				x[q][k] = __ldg(s + k);
		}
#pragma unroll
		for (unsigned q = 0; q < kRegBatch; ++q) {
			if (r + q >= r1)
				break;
			S *out = reinterpret_cast<S *>(dst + static_cast<ptrdiff_t>(r + q) * ds) + j;
			if constexpr (INT) {
				uint32_t acc = b;
#pragma unroll
				for (int k = 0; k < W; ++k)
					acc += static_cast<uint32_t>(c[k] * static_cast<int32_t>(x[q][k]));
				*out = pack_u16(acc, pixel_max);
			} else {
				float acc = 0.0f;
#pragma unroll
				for (int k = 0; k < W; ++k)
					acc = __fmaf_rn(c[k], x[q][k], acc);
				*out = acc;
			}
		}
	}
}

template <bool INT, int W = kRegTaps>
cudaError_t launch_h_reg(const PassLaunch &l, const PassPlanes &P, cudaStream_t stream)
{
	if constexpr (W > 0) {
		if (l.t.width != W)
			return launch_h_reg<INT, W - 1>(l, P, stream);
		dim3 grid((l.t.rows + kThreads - 1) / kThreads, (l.lines + kRegRows - 1) / kRegRows, l.num_planes);
		h_reg_kernel<INT, W><<<grid, kThreads, 0, stream>>>(l.t, l.pixel_max, l.lines, P);
		return cudaGetLastError();
	} else {
		return cudaErrorInvalidValue;
	}
}

// The vertical counterpart: thread = VEC adjacent columns of kRegColRows output
// rows, the loads of a row's whole window in flight together. Measured, one
// plane, vertical pass alone, before and now:
//   u16 1920x540 -> 1920x1080, 6 taps           6.0 -> 4.1 us
//   u16 1920x1080 -> 1920x721, 10 taps          7.4 -> 4.5 us
//   u16 1919x1080 -> 1919x721 (2-byte loads)    8.5 -> 6.8 us
//   f32 1920x1080 -> 1920x540, 16 taps          9.8 -> 5.4 us
//   f32 3840x2160 -> 3840x1080, 8 taps         15.7 -> 13.0 us
//   u16 1920x1080 -> 1920x360, 17 taps         10.0 -> 4.9 us
//   u16 1920x1080 -> 1920x216, 29 taps         14.8 -> 5.3 us
//   f32 1920x1080 -> 1920x269, 26 taps         12.9 -> 5.8 us
// f32 planes that are not 16-byte aligned stay with v_f32_kernel, whose
// 4-byte loads came to 18.3 us at 3839x2160 -> 3839x1080, 18.6 us here.
constexpr unsigned kRegColRows = 4;

template <bool INT, int VEC, int W>
__global__ void __launch_bounds__(kThreads)
v_reg_kernel(PassTables t, int32_t pixel_max, unsigned plane_w, const __grid_constant__ PassPlanes P)
{
	ZG_PASS_PLANE
	using S = std::conditional_t<INT, uint16_t, float>;
	using A = std::conditional_t<INT, uint32_t, float>;
	const unsigned j0 = (blockIdx.x * kThreads + threadIdx.x) * VEC;
	if (j0 >= plane_w)
		return;
	const bool full = j0 + VEC <= plane_w;
	const unsigned i1 = min((blockIdx.y + 1) * kRegColRows, t.rows);
	for (unsigned i = blockIdx.y * kRegColRows; i < i1; ++i) {
		const uint8_t *row = src + static_cast<ptrdiff_t>(__ldg(t.left + i)) * ss + static_cast<size_t>(j0) * sizeof(S);
		uint4 x[W];
		if (VEC > 1 && full) {
#pragma unroll
			for (int k = 0; k < W; ++k)
				x[k] = __ldg(reinterpret_cast<const uint4 *>(row + k * ss));
		} else {
#pragma unroll
			for (int k = 0; k < W; ++k) {
				uint32_t w[4] = {};
				const S *r = reinterpret_cast<const S *>(row + k * ss);
#pragma unroll
				for (int v = 0; v < VEC; ++v) {
					if (!full && j0 + v >= plane_w)
						continue;
					if constexpr (INT)
						w[v / 2] |= static_cast<uint32_t>(__ldg(r + v)) << (v % 2 * 16);
					else
						w[v] = __float_as_uint(__ldg(r + v));
				}
				x[k] = make_uint4(w[0], w[1], w[2], w[3]);
			}
		}
		A acc[VEC];
#pragma unroll
		for (int v = 0; v < VEC; ++v) {
			if constexpr (INT)
				acc[v] = static_cast<uint32_t>(__ldg(t.bias + i));
			else
				acc[v] = 0.0f;
		}
#pragma unroll
		for (int k = 0; k < W; ++k) {
			const uint32_t w[4] = { x[k].x, x[k].y, x[k].z, x[k].w };
#pragma unroll
			for (int v = 0; v < VEC; ++v) {
				if constexpr (INT)
					acc[v] += static_cast<uint32_t>(static_cast<int32_t>(__ldg(t.i16 + static_cast<size_t>(i) * W + k)) *
					                                static_cast<int32_t>(v % 2 ? w[v / 2] >> 16 : w[v / 2] & 0xFFFFu));
				else
					acc[v] = __fmaf_rn(__ldg(t.f32 + static_cast<size_t>(i) * W + k), __uint_as_float(w[v]), acc[v]);
			}
		}
		S *out = reinterpret_cast<S *>(dst + static_cast<ptrdiff_t>(i) * ds) + j0;
		uint32_t o[4] = {};
#pragma unroll
		for (int v = 0; v < VEC; ++v) {
			if constexpr (INT)
				o[v / 2] |= static_cast<uint32_t>(pack_u16(acc[v], pixel_max)) << (v % 2 * 16);
			else
				o[v] = __float_as_uint(acc[v]);
		}
		if (VEC > 1 && full) {
			*reinterpret_cast<uint4 *>(out) = make_uint4(o[0], o[1], o[2], o[3]);
			continue;
		}
#pragma unroll
		for (int v = 0; v < VEC; ++v) {
			if (!full && j0 + v >= plane_w)
				break;
			if constexpr (INT)
				out[v] = static_cast<uint16_t>(o[v / 2] >> (v % 2 * 16));
			else
				out[v] = __uint_as_float(o[v]);
		}
	}
}

template <bool INT, int VEC, int W = kRegTaps>
cudaError_t launch_v_reg(const PassLaunch &l, const PassPlanes &P, cudaStream_t stream)
{
	if constexpr (W > 0) {
		if (l.t.width != W)
			return launch_v_reg<INT, VEC, W - 1>(l, P, stream);
		dim3 grid((l.lines + kThreads * VEC - 1) / (kThreads * VEC), (l.t.rows + kRegColRows - 1) / kRegColRows, l.num_planes);
		v_reg_kernel<INT, VEC, W><<<grid, kThreads, 0, stream>>>(l.t, l.pixel_max, l.lines, P);
		return cudaGetLastError();
	} else {
		return cudaErrorInvalidValue;
	}
}

// ------------------------------------------------------ wide, CUDA cores --
// FP32 passes of kDenseTaps taps or more, on the dense groups of outputs
// (PassTables::dense). Each output's taps are applied in zimg's order, one
// fused multiply-add each; the block's zeros outside an output's band add
// 0 * x, which leaves an accumulator that started at +0 unchanged for finite
// samples (such an accumulator never becomes -0), so the results are those of
// the per-output kernels above.

constexpr unsigned kVRows = dense_rows(false);  // 8
constexpr unsigned kHRows = dense_rows(true);   // 4

// Vertical: thread = 4 adjacent columns (16-byte loads and stores, planes
// 16-byte aligned); block = kThreads * 4 columns x `groups_per_block` groups
// of 8 output rows. Per input line of a group's window: one load of the 4
// columns, the group's 8 taps of that line (two 16-byte loads, the same for
// every thread), 32 multiply-adds as 16 paired ones. A line is read once per
// group. Group size trades reads against work: a 16x downscale of 129 taps
// reads each line 1.9 times with 8 rows (1.4 with 16, 2.8 with 4) and its
// dense windows are 54 % taps (35 % with 16); 8 measured fastest (16 rows
// leave too few warps per plane).
__global__ void __launch_bounds__(kThreads)
v_f32_dense_kernel(PassTables t, unsigned plane_w, const uint8_t *__restrict__ src, ptrdiff_t ss,
                   uint8_t *__restrict__ dst, ptrdiff_t ds, unsigned groups_per_block)
{
	const unsigned j0 = (blockIdx.x * kThreads + threadIdx.x) * 4;
	if (j0 >= plane_w)
		return;
	const bool full = j0 + 4 <= plane_w;
	const unsigned ngroups = (t.rows + kVRows - 1) / kVRows;
	const unsigned g0 = blockIdx.y * groups_per_block;
	const unsigned g1 = min(g0 + groups_per_block, ngroups);
	for (unsigned g = g0; g < g1; ++g) {
		const unsigned base = __ldg(t.dbase + g), span = __ldg(t.dspan + g);
		const float4 *tap = reinterpret_cast<const float4 *>(t.dense) + static_cast<size_t>(g) * t.dstride * (kVRows / 4);
		float2 acc[kVRows][2];
#pragma unroll
		for (int r = 0; r < static_cast<int>(kVRows); ++r)
			acc[r][0] = acc[r][1] = make_float2(0.0f, 0.0f);
		const uint8_t *row = src + static_cast<ptrdiff_t>(base) * ss + static_cast<size_t>(j0) * 4;
#pragma unroll 2
		for (unsigned u = 0; u < span; ++u, row += ss) {
			float4 x;
			if (full) {
				x = __ldg(reinterpret_cast<const float4 *>(row));
			} else {
				const float *rf = reinterpret_cast<const float *>(row);
				x.x = __ldg(rf);
				x.y = j0 + 1 < plane_w ? __ldg(rf + 1) : 0.0f;
				x.z = j0 + 2 < plane_w ? __ldg(rf + 2) : 0.0f;
				x.w = j0 + 3 < plane_w ? __ldg(rf + 3) : 0.0f;
			}
			const float2 x01 = make_float2(x.x, x.y), x23 = make_float2(x.z, x.w);
#pragma unroll
			for (int q = 0; q < static_cast<int>(kVRows / 4); ++q) {
				const float4 c = __ldg(tap + u * (kVRows / 4) + q);
				const float cr[4] = { c.x, c.y, c.z, c.w };
#pragma unroll
				for (int e = 0; e < 4; ++e) {
					const float2 cc = make_float2(cr[e], cr[e]);
					acc[4 * q + e][0] = __ffma2_rn(cc, x01, acc[4 * q + e][0]);
					acc[4 * q + e][1] = __ffma2_rn(cc, x23, acc[4 * q + e][1]);
				}
			}
		}
#pragma unroll
		for (int r = 0; r < static_cast<int>(kVRows); ++r) {
			const unsigned i = g * kVRows + r;
			if (i >= t.rows)
				break;
			float *out = reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(i) * ds) + j0;
			if (full) {
				*reinterpret_cast<float4 *>(out) = make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
			} else {
				const float v[4] = { acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y };
				for (int q = 0; q < 4 && j0 + q < plane_w; ++q)
					out[q] = v[q];
			}
		}
	}
}

// Horizontal: warp = one line x 32 consecutive groups of 4 outputs (lane =
// group). The warp first copies its groups' input window of the line into
// shared memory with coalesced loads (one pad word per 32, so that lanes
// whose windows start 2^n samples apart read different banks), then each
// lane runs its group: per input one sample from shared memory, the group's
// 4 taps (coalesced across the lanes: the table keeps 32 groups side by
// side), 4 multiply-adds. kHWarps lines per block.
constexpr int kHWarps = 4;

__host__ __device__ __forceinline__ unsigned hpad(unsigned i)
{
	return i + (i >> 5);
}

__global__ void __launch_bounds__(kHWarps * 32)
h_f32_dense_kernel(PassTables t, unsigned lines, const uint8_t *__restrict__ src, ptrdiff_t ss,
                   uint8_t *__restrict__ dst, ptrdiff_t ds)
{
	extern __shared__ float hwin[];
	const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const unsigned ngroups = (t.rows + kHRows - 1) / kHRows;
	const unsigned gw = blockIdx.x * 32;  // first group of the warp
	const unsigned r = blockIdx.y * kHWarps + warp;
	if (r >= lines)
		return;
	float *win = hwin + warp * hpad(t.dwin + 32);
	const unsigned glast = min(gw + 32, ngroups) - 1;
	const unsigned w0 = __ldg(t.dbase + gw);
	const unsigned wn = __ldg(t.dbase + glast) + __ldg(t.dspan + glast) - w0;
	const float *s = reinterpret_cast<const float *>(src + static_cast<ptrdiff_t>(r) * ss) + w0;
	for (unsigned i = lane; i < wn; i += 32)
		win[hpad(i)] = __ldg(s + i);
	__syncwarp();
	const unsigned g = gw + lane;
	if (g >= ngroups)
		return;
	const unsigned off = __ldg(t.dbase + g) - w0, span = __ldg(t.dspan + g);
	const float4 *tap = reinterpret_cast<const float4 *>(t.dense) + g;
	float2 acc01 = make_float2(0.0f, 0.0f), acc23 = make_float2(0.0f, 0.0f);
#pragma unroll 4
	for (unsigned u = 0; u < span; ++u) {
		const float4 c = __ldg(tap + static_cast<size_t>(u) * ngroups);
		const float x = win[hpad(off + u)];
		acc01 = __ffma2_rn(make_float2(c.x, c.y), make_float2(x, x), acc01);
		acc23 = __ffma2_rn(make_float2(c.z, c.w), make_float2(x, x), acc23);
	}
	float *out = reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(r) * ds) + g * kHRows;
	const float v[4] = { acc01.x, acc01.y, acc23.x, acc23.y };
#pragma unroll
	for (int q = 0; q < static_cast<int>(kHRows); ++q)
		if (g * kHRows + q < t.rows)
			out[q] = v[q];
}

bool aligned16(const void *p, ptrdiff_t stride)
{
	return (reinterpret_cast<uintptr_t>(p) % 16) == 0 && (stride % 16) == 0;
}

} // namespace


cudaError_t launch_pass(const PassLaunch &l, cudaStream_t stream)
{
	if (l.num_planes != 1 && (l.wide.frag || l.t.dense))
		return cudaErrorInvalidValue;  // these kernels take a plane
	if (l.wide.frag && l.sample == Sample::F32)
		return launch_wide(l, stream);
	const uint8_t *src = static_cast<const uint8_t *>(l.src);
	uint8_t *dst = static_cast<uint8_t *>(l.dst);
	if (l.sample == Sample::F32 && l.t.dense) {
		if (l.horizontal) {
			// staged windows of 32 groups, up to 16 KB per warp
			const size_t win_bytes = static_cast<size_t>(hpad(l.t.dwin + 32)) * 4;
			if (win_bytes <= 16384) {
				const unsigned groups = (l.t.rows + kHRows - 1) / kHRows;
				dim3 grid((groups + 31) / 32, (l.lines + kHWarps - 1) / kHWarps);
				cudaError_t e = cudaFuncSetAttribute(h_f32_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
				                                     static_cast<int>(kHWarps * 16384 + 4096));
				if (e != cudaSuccess)
					return e;
				h_f32_dense_kernel<<<grid, kHWarps * 32, kHWarps * win_bytes, stream>>>(l.t, l.lines, src,
				                                                                      l.src_stride, dst, l.dst_stride);
				return cudaGetLastError();
			}
		} else if (aligned16(l.src, l.src_stride) && aligned16(l.dst, l.dst_stride)) {
			const unsigned groups = (l.t.rows + kVRows - 1) / kVRows;
			const unsigned col_blocks = (l.lines + kThreads * 4 - 1) / (kThreads * 4);
			dim3 grid(col_blocks, groups);
			v_f32_dense_kernel<<<grid, kThreads, 0, stream>>>(l.t, l.lines, src, l.src_stride, dst, l.dst_stride, 1);
			return cudaGetLastError();
		}
	}
	if (l.num_planes < 1 || l.num_planes > kPassPlanes)
		return cudaErrorInvalidValue;
	// Down the columns, a launch goes in 16-byte accesses if all of its planes
	// are aligned: others get a launch of their own where the aligned ones are
	// more than kSplitBytes. 16 u16 planes of one conversion 3840x2160 ->
	// 3840x1080, one of them unaligned: 122 us a plane a launch, 178 in one
	// launch, 89 in two (712 MB); f32 1920x1080 -> 1920x540, one of 16: 73, 61,
	// 47 (187 MB), one of three: 14.5, 14.4, 16.5 (25 MB).
	constexpr size_t kSplitBytes = 32 << 20;
	PassPlanes P{};
	P.p[0] = { l.src, l.src_stride, l.dst, l.dst_stride };
	int aligned = 0;
	for (int k = 0, other = l.num_planes; k < l.num_planes; ++k) {
		const PassPlane &p = l.planes ? l.planes[k] : P.p[0];
		const bool a = aligned16(p.src, p.src_stride) && aligned16(p.dst, p.dst_stride);
		P.p[a ? aligned++ : --other] = p;
	}
	const bool vec = aligned == l.num_planes;
	const size_t aligned_bytes = static_cast<size_t>(aligned) * l.lines * (l.t.input_width + l.t.rows) *
	                             (l.sample == Sample::U16 ? 2 : 4);
	if (!l.horizontal && !vec && aligned_bytes > kSplitBytes) {
		PassLaunch part = l;
		part.planes = P.p;
		part.num_planes = aligned;
		const cudaError_t e = launch_pass(part, stream);
		if (e != cudaSuccess)
			return e;
		part.planes = P.p + aligned;
		part.num_planes = l.num_planes - aligned;
		return launch_pass(part, stream);
	}
	if (l.horizontal && l.t.width <= kRegTaps)
		return l.sample == Sample::U16 ? launch_h_reg<true>(l, P, stream) : launch_h_reg<false>(l, P, stream);
	if (l.horizontal) {
		const unsigned rpb = 8;
		dim3 grid((l.t.rows + kThreads - 1) / kThreads, (l.lines + rpb - 1) / rpb, l.num_planes);
		if (l.sample == Sample::U16)
			h_u16_kernel<<<grid, kThreads, 0, stream>>>(l.t, l.pixel_max, l.lines, P, rpb);
		else
			h_f32_kernel<<<grid, kThreads, 0, stream>>>(l.t, l.lines, P, rpb);
	} else {
		const unsigned rpb = 4;
		if (l.t.width <= kRegTaps && (l.sample == Sample::U16 || vec)) {
			if (l.sample == Sample::F32)
				return launch_v_reg<false, 4>(l, P, stream);
			return vec ? launch_v_reg<true, 8>(l, P, stream) : launch_v_reg<true, 1>(l, P, stream);
		}
		if (l.sample == Sample::U16) {
			const int V = vec ? 8 : 1;
			dim3 grid((l.lines + kThreads * V - 1) / (kThreads * V), (l.t.rows + rpb - 1) / rpb, l.num_planes);
			if (vec)
				v_u16_kernel<8><<<grid, kThreads, 0, stream>>>(l.t, l.pixel_max, l.lines, P, rpb);
			else
				v_u16_kernel<1><<<grid, kThreads, 0, stream>>>(l.t, l.pixel_max, l.lines, P, rpb);
		} else {
			dim3 grid((l.lines + kThreads - 1) / kThreads, (l.t.rows + rpb - 1) / rpb, l.num_planes);
			v_f32_kernel<<<grid, kThreads, 0, stream>>>(l.t, l.lines, P, rpb);
		}
	}
	return cudaGetLastError();
}

} // namespace zg
