// Colorspace conversion of three FLOAT planes (zimg's ColorspaceConversionImpl,
// src/zimg/colorspace/colorspace.cpp:16-78, operations of
// operation_impl.cpp:21-258): every operation of the plan applied to a pixel
// in registers, one pass over the planes. Every product, sum and quotient is
// written with the separately rounding CS_* forms, as zimg's C code rounds
// them.
//
// Plans of matrices alone are HBM-bound (12 bytes read and 12 written per
// pixel): matrix_kernel, runs of 4 pixels a thread, 16-byte vectors where all
// planes allow. Transfer functions make a pixel some 900 instructions, and
// the bound is the instruction supply: with four pixels a thread and every
// operation inlined twelve times, the warps waited for instructions 8 of 17
// cycles (issue slots 44 % busy). pixel_kernel therefore has one copy of each
// operation, a pixel a thread, its three channels taken in turn by a loop that
// rotates them: 2,073,600 pixels BT.2020 PQ -> BT.709, 103 -> 60 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "colorspace_plan.h"
#include "colorspace_tf.cuh"

namespace zg {
namespace csp {

namespace {

constexpr int kThreads = 256;
constexpr int kPixelThreads = 128;

__device__ __forceinline__ void apply_matrix(const Op &o, float &a, float &b, float &c)
{
	const float x = CS_ADD(CS_ADD(CS_MUL(o.m[0][0], a), CS_MUL(o.m[0][1], b)), CS_MUL(o.m[0][2], c));
	const float y = CS_ADD(CS_ADD(CS_MUL(o.m[1][0], a), CS_MUL(o.m[1][1], b)), CS_MUL(o.m[1][2], c));
	const float z = CS_ADD(CS_ADD(CS_MUL(o.m[2][0], a), CS_MUL(o.m[2][1], b)), CS_MUL(o.m[2][2], c));
	a = x;
	b = y;
	c = z;
}

// The transfer function of an operation on the three channels: found once
// (F counts up to it at compile time; the compiler makes it a jump), then one
// copy of it in a loop that rotates the channels.
template <int F>
__device__ __forceinline__ void apply_gamma(const Op &o, float &a, float &b, float &c)
{
	if constexpr (F < TF_COUNT) {
		if (o.f != F) {
			apply_gamma<F + 1>(o, a, b, c);
			return;
		}
		const float pre = o.pre, post = o.post;
#pragma unroll 1
		for (int k = 0; k < 3; ++k) {
			const float v = CS_MUL(post, apply_tf(F, CS_MUL(a, pre)));
			a = b;
			b = c;
			c = v;
		}
	}
}

__device__ __forceinline__ void apply_op(const Op &o, float &a, float &b, float &c)
{
	switch (o.kind) {
	case OP_MATRIX: apply_matrix(o, a, b, c); break;
	case OP_GAMMA: apply_gamma<0>(o, a, b, c); break;
	case OP_HLG: {
		// display-referred HLG: system gamma 1.2 on the luma (operation_impl.cpp:76-114)
		const float gamma = 1.2f;
		const float r = CS_MUL(a, o.scale), g = CS_MUL(b, o.scale), bb = CS_MUL(c, o.scale);
		float yd = CS_ADD(CS_ADD(CS_MUL(o.kr, r), CS_MUL(o.kg, g)), CS_MUL(o.kb, bb));
		yd = yd < FLT_MIN ? FLT_MIN : yd;
		const float ys_inv = powf(yd, (1.0f - gamma) / gamma);
		a = hlg_oetf(CS_MUL(r, ys_inv));
		b = hlg_oetf(CS_MUL(g, ys_inv));
		c = hlg_oetf(CS_MUL(bb, ys_inv));
		break;
	}
	case OP_HLG_INV: {
		const float gamma = 1.2f;
		float r = hlg_inv_oetf(a), g = hlg_inv_oetf(b), bb = hlg_inv_oetf(c);
		float ys = CS_ADD(CS_ADD(CS_MUL(o.kr, r), CS_MUL(o.kg, g)), CS_MUL(o.kb, bb));
		ys = ys < FLT_MIN ? FLT_MIN : ys;
		ys = powf(ys, gamma - 1.0f);
		r = CS_MUL(r, ys);
		g = CS_MUL(g, ys);
		bb = CS_MUL(bb, ys);
		a = CS_MUL(r, o.scale);
		b = CS_MUL(g, o.scale);
		c = CS_MUL(bb, o.scale);
		break;
	}
	case OP_CL_TO_RGB: {
		// BT.2020 constant luminance to linear RGB (operation_impl.cpp:156-206)
		const float y = a, u = b, v = c;
		const float bmy = u < 0 ? CS_MUL(CS_MUL(u, 2.0f), o.nb) : CS_MUL(CS_MUL(u, 2.0f), o.pb);
		const float rmy = v < 0 ? CS_MUL(CS_MUL(v, 2.0f), o.nr) : CS_MUL(CS_MUL(v, 2.0f), o.pr);
		const float bl = apply_tf(o.f, CS_ADD(bmy, y)), rl = apply_tf(o.f, CS_ADD(rmy, y)), yl = apply_tf(o.f, y);
		const float g = CS_DIV(CS_SUB(CS_SUB(yl, CS_MUL(o.kr, rl)), CS_MUL(o.kb, bl)), o.kg);
		a = CS_MUL(rl, o.scale);
		b = CS_MUL(g, o.scale);
		c = CS_MUL(bl, o.scale);
		break;
	}
	case OP_CL_TO_YUV: {
		// linear RGB to BT.2020 constant luminance (operation_impl.cpp:209-258)
		float r = CS_MUL(a, o.scale), g = CS_MUL(b, o.scale), bb = CS_MUL(c, o.scale);
		const float y = apply_tf(o.f, CS_ADD(CS_ADD(CS_MUL(o.kr, r), CS_MUL(o.kg, g)), CS_MUL(o.kb, bb)));
		bb = apply_tf(o.f, bb);
		r = apply_tf(o.f, r);
		const float bmy = CS_SUB(bb, y), rmy = CS_SUB(r, y);
		const float u = bmy < 0.0f ? CS_DIV(bmy, CS_MUL(2.0f, o.nb)) : CS_DIV(bmy, CS_MUL(2.0f, o.pb));
		const float v = rmy < 0.0f ? CS_DIV(rmy, CS_MUL(2.0f, o.nr)) : CS_DIV(rmy, CS_MUL(2.0f, o.pr));
		a = y;
		b = u;
		c = v;
		break;
	}
	default: break;
	}
}

__global__ void __launch_bounds__(kThreads) matrix_kernel(const __grid_constant__ Launch L)
{
	const int quads = (L.width + 3) / 4;
	const long long total = static_cast<long long>(quads) * L.height;
	for (long long u = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x; u < total;
	     u += static_cast<long long>(gridDim.x) * kThreads) {
		const int i = static_cast<int>(u / quads);
		const int j0 = static_cast<int>(u - static_cast<long long>(i) * quads) * 4;
		const int n = min(4, L.width - j0);
		const float *s[3];
		float *d[3];
#pragma unroll
		for (int p = 0; p < 3; ++p) {
			s[p] = reinterpret_cast<const float *>(static_cast<const char *>(L.src[p]) +
			                                       static_cast<ptrdiff_t>(i) * L.src_stride[p]) + j0;
			d[p] = reinterpret_cast<float *>(static_cast<char *>(L.dst[p]) + static_cast<ptrdiff_t>(i) * L.dst_stride[p]) +
			       j0;
		}
		float x[3][4];
		if (L.vec && n == 4) {
#pragma unroll
			for (int p = 0; p < 3; ++p) {
				const float4 v = *reinterpret_cast<const float4 *>(s[p]);
				x[p][0] = v.x;
				x[p][1] = v.y;
				x[p][2] = v.z;
				x[p][3] = v.w;
			}
		} else {
#pragma unroll
			for (int e = 0; e < 4; ++e)
#pragma unroll
				for (int p = 0; p < 3; ++p)
					x[p][e] = e < n ? s[p][e] : 0.0f;
		}
		for (int k = 0; k < L.plan.num_ops; ++k) {
			const Op &o = L.plan.ops[k];
#pragma unroll
			for (int e = 0; e < 4; ++e)
				apply_matrix(o, x[0][e], x[1][e], x[2][e]);
		}
		if (L.vec && n == 4) {
#pragma unroll
			for (int p = 0; p < 3; ++p)
				*reinterpret_cast<float4 *>(d[p]) = make_float4(x[p][0], x[p][1], x[p][2], x[p][3]);
		} else {
			for (int e = 0; e < n; ++e)
#pragma unroll
				for (int p = 0; p < 3; ++p)
					d[p][e] = x[p][e];
		}
	}
}

__global__ void __launch_bounds__(kPixelThreads) pixel_kernel(const __grid_constant__ Launch L)
{
	const int j = blockIdx.x * kPixelThreads + threadIdx.x;
	if (j >= L.width)
		return;
	for (int i = blockIdx.y; i < L.height; i += gridDim.y) {
		float x[3];
#pragma unroll
		for (int p = 0; p < 3; ++p)
			x[p] = reinterpret_cast<const float *>(static_cast<const char *>(L.src[p]) +
			                                       static_cast<ptrdiff_t>(i) * L.src_stride[p])[j];
#pragma unroll 1
		for (int k = 0; k < L.plan.num_ops; ++k)
			apply_op(L.plan.ops[k], x[0], x[1], x[2]);
#pragma unroll
		for (int p = 0; p < 3; ++p)
			reinterpret_cast<float *>(static_cast<char *>(L.dst[p]) + static_cast<ptrdiff_t>(i) * L.dst_stride[p])[j] =
				x[p];
	}
}

} // namespace

cudaError_t launch_colorspace(const Launch &L, cudaStream_t stream)
{
	if (L.width <= 0 || L.height <= 0)
		return cudaSuccess;
	bool matrices = true;
	for (int k = 0; k < L.plan.num_ops; ++k)
		matrices = matrices && L.plan.ops[k].kind == OP_MATRIX;
	if (!matrices) {
		const dim3 grid((L.width + kPixelThreads - 1) / kPixelThreads, std::min(L.height, 65535));
		pixel_kernel<<<grid, kPixelThreads, 0, stream>>>(L);
		return cudaGetLastError();
	}
	static int sms = 0;
	if (!sms) {
		int dev = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		if (sms < 1)
			sms = 1;
	}
	const long long units = static_cast<long long>((L.width + 3) / 4) * L.height;
	const int grid = static_cast<int>(std::min<long long>((units + kThreads - 1) / kThreads, static_cast<long long>(sms) * 8));
	matrix_kernel<<<grid, kThreads, 0, stream>>>(L);
	return cudaGetLastError();
}

} // namespace csp
} // namespace zg
