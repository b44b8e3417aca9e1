// Unresize passes on the GPU (zimg's unresize_impl.cpp:27-97, C path): per
// output sample a banded FP32 dot product with A''s row, then the forward
// substitution of the tridiagonal LU, then the back substitution; every
// product, sum and difference rounded on its own, as in zimg's C code.
//
// unresize_lines runs a pass as one launch. The substitutions are recurrences
// along the line, 12 and 8 cycles of dependent operations a sample, but each
// step keeps only a fraction of the one before (|c l|, |u| about 0.3 for a
// 1.5x upscale): after `reach` steps a wrong start has shrunk by 2^60, 24 of
// them to a sample's last place and the rest to let two roundings meet, and
// the samples are as a rule the same bits. So a line is cut into chunks that run
// side by side, each from `reach` steps before it with a zero start; then every
// chunk compares the bits it started from with the bits its neighbour ended
// on, and runs again from those where they differ, until none does. What is
// left is the serial result, whatever the data (a NaN, or denormals dying out
// in a black border, only cost rounds). Blocks hold whole lines or columns in
// shared memory, so the dot products, both substitutions and the comparison
// need no pass over memory in between.
//
// Lines too long for shared memory, contexts whose factors do not shrink
// (bilinear weights of a half: no reach) and long rows of taps (chunk_shape) take
// two launches: the dot products,
// one thread per output sample (k in zimg's order), into the pass's output
// plane, then the substitutions, one thread per line or column, rewriting the
// plane in place, with the next inputs loaded before the dependent steps so
// that memory latency overlaps the chain (down a column in groups of kAhead
// values; along lines a warp moves tiles of 32 lines x 32 values through
// shared memory).
//
// Measured, three planes 1920x1080 -> 1280x720 one after another: 514 us in
// two launches a pass (subst_h 106, subst_v 62, dots 18 a plane), 91 us
// here.
#include "unresize.h"

#include "launch_attr.h"

#include <algorithm>

namespace zg {

namespace {

constexpr int kThreads = 128;
constexpr int kAhead = 32;  // recurrence inputs loaded per group

// dst[line][j] = sum_k coef[j][k] * src[line][offset[j] + k]
__global__ void __launch_bounds__(kThreads)
unresize_dot_h(UnresizeTables t, unsigned lines, const char *__restrict__ src, ptrdiff_t ss, char *__restrict__ dst,
               ptrdiff_t ds)
{
	const unsigned j = blockIdx.x * kThreads + threadIdx.x;
	if (j >= t.orig)
		return;
	const float *cf = t.coef + static_cast<size_t>(j) * t.row_size;
	const unsigned off = __ldg(t.offset + j);
	for (unsigned line = blockIdx.y; line < lines; line += gridDim.y) {
		const float *x = reinterpret_cast<const float *>(src + static_cast<ptrdiff_t>(line) * ss) + off;
		float accum = 0.0f;
		for (unsigned k = 0; k < t.row_size; ++k)
			accum = __fadd_rn(accum, __fmul_rn(__ldg(cf + k), __ldg(x + k)));
		reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(line) * ds)[j] = accum;
	}
}

// dst[i][col] = sum_k coef[i][k] * src[offset[i] + k][col]
__global__ void __launch_bounds__(kThreads)
unresize_dot_v(UnresizeTables t, unsigned cols, const char *__restrict__ src, ptrdiff_t ss, char *__restrict__ dst,
               ptrdiff_t ds)
{
	const unsigned col = blockIdx.x * kThreads + threadIdx.x;
	if (col >= cols)
		return;
	for (unsigned i = blockIdx.y; i < t.orig; i += gridDim.y) {
		const float *cf = t.coef + static_cast<size_t>(i) * t.row_size;
		const char *x = src + static_cast<ptrdiff_t>(__ldg(t.offset + i)) * ss + static_cast<size_t>(col) * 4;
		float accum = 0.0f;
		for (unsigned k = 0; k < t.row_size; ++k)
			accum = __fadd_rn(accum, __fmul_rn(__ldg(cf + k),
			                                   __ldg(reinterpret_cast<const float *>(x + static_cast<ptrdiff_t>(k) * ss))));
		reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(i) * ds)[col] = accum;
	}
}

// The substitutions over n values at p, p + step, ... (step in floats):
// z_i = (a_i - c_i z_{i-1}) * l_i, then w_i = z_i - u_i w_{i+1}. Inputs go
// in groups of kAhead; group g + 1 is loaded before group g's steps run.
__device__ __forceinline__ void substitute(const UnresizeTables &t, float *p, ptrdiff_t step, unsigned n)
{
	auto at = [&](unsigned i) -> float & { return p[static_cast<ptrdiff_t>(i) * step]; };
	float z = 0.0f;
	const unsigned full = n / kAhead * kAhead;
	float cur[kAhead], nxt[kAhead];
	if (full) {
#pragma unroll
		for (int e = 0; e < kAhead; ++e)
			cur[e] = at(e);
	}
	for (unsigned i = 0; i < full; i += kAhead) {
		if (i + kAhead < full) {
#pragma unroll
			for (int e = 0; e < kAhead; ++e)
				nxt[e] = at(i + kAhead + e);
		}
#pragma unroll
		for (int e = 0; e < kAhead; ++e) {
			z = __fmul_rn(__fsub_rn(cur[e], __fmul_rn(__ldg(t.lu_c + i + e), z)), __ldg(t.lu_l + i + e));
			at(i + e) = z;
		}
#pragma unroll
		for (int e = 0; e < kAhead; ++e)
			cur[e] = nxt[e];
	}
	for (unsigned i = full; i < n; ++i) {
		z = __fmul_rn(__fsub_rn(at(i), __fmul_rn(__ldg(t.lu_c + i), z)), __ldg(t.lu_l + i));
		at(i) = z;
	}
	// back substitution from the last value: the partial group first
	float w = 0.0f;
	for (unsigned r = n; r > full; --r) {
		w = __fsub_rn(at(r - 1), __fmul_rn(__ldg(t.lu_u + r - 1), w));
		at(r - 1) = w;
	}
	if (full) {
#pragma unroll
		for (int e = 0; e < kAhead; ++e)
			cur[e] = at(full - 1 - e);
	}
	for (unsigned r = full; r != 0; r -= kAhead) {
		if (r > kAhead) {
#pragma unroll
			for (int e = 0; e < kAhead; ++e)
				nxt[e] = at(r - kAhead - 1 - e);
		}
#pragma unroll
		for (int e = 0; e < kAhead; ++e) {
			w = __fsub_rn(cur[e], __fmul_rn(__ldg(t.lu_u + r - 1 - e), w));
			at(r - 1 - e) = w;
		}
#pragma unroll
		for (int e = 0; e < kAhead; ++e)
			cur[e] = nxt[e];
	}
}

// Horizontal substitutions, one warp per 32 lines: a line's values are
// contiguous, so a thread per line would read 32 rows per warp load. The warp
// moves tiles of 32 lines x 32 values through shared memory instead (one
// 128-byte row per load instruction, the next two tiles in flight in
// registers), and each lane runs its own line's recurrence on the tile;
// the arithmetic and its order are those of substitute().
constexpr int kTile = 32;

struct HTile {
	float v[kTile];  // this lane's column of the tile: rows 0 .. 31
};

__device__ __forceinline__ void load_tile(HTile &r, const char *dst, ptrdiff_t ds, unsigned line0, unsigned lines,
                                          unsigned col0, unsigned n)
{
	const unsigned lane = threadIdx.x & 31, c = col0 + lane;
#pragma unroll
	for (int i = 0; i < kTile; ++i)
		r.v[i] = (line0 + i < lines && c < n)
		             ? reinterpret_cast<const float *>(dst + static_cast<ptrdiff_t>(line0 + i) * ds)[c]
		             : 0.0f;
}

__global__ void __launch_bounds__(32)
unresize_subst_h(UnresizeTables t, unsigned lines, char *__restrict__ dst, ptrdiff_t ds)
{
	__shared__ float tile[kTile][kTile + 1];
	const unsigned lane = threadIdx.x & 31, line0 = blockIdx.x * kTile;
	const unsigned n = t.orig, tiles = (n + kTile - 1) / kTile;
	const bool mine = line0 + lane < lines;
	// one pass over the tiles, forward (z) or backward (w); row `lane` of a
	// tile is this lane's line
	auto pass = [&](bool forward) {
		HTile a, b;
		float carry = 0.0f;
		const unsigned first = forward ? 0 : tiles - 1;
		load_tile(a, dst, ds, line0, lines, first * kTile, n);
		if (tiles > 1)
			load_tile(b, dst, ds, line0, lines, (forward ? first + 1 : first - 1) * kTile, n);
		for (unsigned k = 0; k < tiles; ++k) {
			const unsigned j = forward ? k : tiles - 1 - k;
			const unsigned col0 = j * kTile, cnt = min(static_cast<unsigned>(kTile), n - col0);
#pragma unroll
			for (int i = 0; i < kTile; ++i)
				tile[i][lane] = a.v[i];
			a = b;
			if (k + 2 < tiles)
				load_tile(b, dst, ds, line0, lines, (forward ? j + 2 : j - 2) * kTile, n);
			__syncwarp();
			if (mine) {
				// whole tiles unrolled, so that the coefficient loads run ahead of the chain
				if (forward && cnt == kTile) {
#pragma unroll
					for (int c = 0; c < kTile; ++c) {
						carry = __fmul_rn(__fsub_rn(tile[lane][c], __fmul_rn(__ldg(t.lu_c + col0 + c), carry)),
						                  __ldg(t.lu_l + col0 + c));
						tile[lane][c] = carry;
					}
				} else if (forward) {
					for (unsigned c = 0; c < cnt; ++c) {
						carry = __fmul_rn(__fsub_rn(tile[lane][c], __fmul_rn(__ldg(t.lu_c + col0 + c), carry)),
						                  __ldg(t.lu_l + col0 + c));
						tile[lane][c] = carry;
					}
				} else if (cnt == kTile) {
#pragma unroll
					for (int c = kTile - 1; c >= 0; --c) {
						carry = __fsub_rn(tile[lane][c], __fmul_rn(__ldg(t.lu_u + col0 + c), carry));
						tile[lane][c] = carry;
					}
				} else {
					for (unsigned c = cnt; c-- > 0;) {
						carry = __fsub_rn(tile[lane][c], __fmul_rn(__ldg(t.lu_u + col0 + c), carry));
						tile[lane][c] = carry;
					}
				}
			}
			__syncwarp();
			const unsigned cc = col0 + lane;
			if (cc < n) {
#pragma unroll
				for (int i = 0; i < kTile; ++i)
					if (line0 + i < lines)
						reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(line0 + i) * ds)[cc] = tile[i][lane];
			}
			__syncwarp();
		}
	};
	pass(true);
	pass(false);
}

__global__ void __launch_bounds__(kThreads)
unresize_subst_v(UnresizeTables t, unsigned cols, char *__restrict__ dst, ptrdiff_t ds)
{
	const unsigned col = blockIdx.x * kThreads + threadIdx.x;
	if (col < cols)
		substitute(t, reinterpret_cast<float *>(dst) + col, ds / 4, t.orig);
}

// ----------------------------------------------------- chunks side by side --

constexpr int kChunkThreads = 512;

struct ChunkShape {
	int series;   // lines or columns of a block (columns: a power of two)
	int chunks, length;  // chunks of a line, samples of a chunk (odd: distinct banks)
	int pitch;    // lines: samples of a line in shared memory
};

// One pass over `count` lines (H) or columns: a block takes L.series of them.
template <bool H>
__global__ void __launch_bounds__(kChunkThreads)
unresize_lines(UnresizeTables t, const __grid_constant__ ChunkShape L, unsigned count, const char *__restrict__ src,
               ptrdiff_t ss, char *__restrict__ dst, ptrdiff_t ds)
{
	extern __shared__ float unresize_smem[];
	const int n = static_cast<int>(t.orig), rs = static_cast<int>(t.row_size);
	float *lc = unresize_smem, *ll = lc + n, *lu = ll + n, *coef = lu + n;
	unsigned *offset = reinterpret_cast<unsigned *>(coef + static_cast<size_t>(n) * rs);
	float *v = reinterpret_cast<float *>(offset + n);
	const int first = blockIdx.x * L.series, left = static_cast<int>(count) - first;
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		lc[i] = __ldg(t.lu_c + i);
		ll[i] = __ldg(t.lu_l + i);
		lu[i] = __ldg(t.lu_u + i);
		offset[i] = __ldg(t.offset + i);
	}
	for (int i = threadIdx.x; i < n * rs; i += blockDim.x)
		coef[i] = __ldg(t.coef + i);
	__syncthreads();
	auto at = [&](int i, int s) -> float & { return H ? v[s * L.pitch + i] : v[i * L.series + s]; };
	// kDots dot products side by side, sum_k coef[i][k] * src[offset[i] + k]
	// with k in zimg's order: samples i, i + i_step, ... of lines or columns
	// s, s + s_step, ... (past the last sample or line: the last one again)
	constexpr int kDots = 8;
	const int series = min(L.series, left);
	const ptrdiff_t along = H ? 4 : ss, across = H ? ss : 4;
	auto dots = [&](int i0, int i_step, int end, int s0, int s_step) {
		const char *x[kDots];
		float sum[kDots];
		int cf[kDots];
#pragma unroll
		for (int q = 0; q < kDots; ++q) {
			const int i = min(i0 + q * i_step, end - 1), s = min(s0 + q * s_step, series - 1);
			cf[q] = i * rs;
			x[q] = src + (first + s) * across + static_cast<ptrdiff_t>(offset[i]) * along;
			sum[q] = 0.0f;
		}
		for (int k = 0; k < rs; ++k) {
			float in[kDots];
#pragma unroll
			for (int q = 0; q < kDots; ++q)
				in[q] = __ldg(reinterpret_cast<const float *>(x[q] + k * along));
#pragma unroll
			for (int q = 0; q < kDots; ++q)
				sum[q] = __fadd_rn(sum[q], __fmul_rn(coef[cf[q] + k], in[q]));
		}
#pragma unroll
		for (int q = 0; q < kDots; ++q)
			if (i0 + q * i_step < end && s0 + q * s_step < series)
				at(i0 + q * i_step, s0 + q * s_step) = sum[q];
	};
	if (H) {
		for (int i = threadIdx.x; i < n; i += blockDim.x)
			for (int s = 0; s < series; s += kDots)
				dots(i, 0, n, s, 1);
	} else {
		const int s = threadIdx.x & (L.series - 1), rows = blockDim.x / L.series;
		if (s < series)
			for (int i = threadIdx.x / L.series; i < n; i += kDots * rows)
				dots(i, rows, n, s, 0);
	}
	__syncthreads();

	const int s = H ? threadIdx.x / L.chunks : threadIdx.x & (L.series - 1);
	const int chunk = H ? threadIdx.x % L.chunks : threadIdx.x / L.series;
	const int b = chunk * L.length, e = min(n, b + L.length);
	const bool on = s < series && b < n;
	const int reach = static_cast<int>(t.reach);
	// z_i = (a_i - c_i z_{i-1}) * l_i over [i, end), w_i = z_i - u_i w_{i+1} over
	// [end, i] downwards; the values written back where `keep`. Eight steps'
	// operands at a time, loaded before the dependent steps.
	constexpr int kBlock = 8;
	auto forward = [&](float z, int i, int end, bool keep) {
		for (; i + kBlock <= end; i += kBlock) {
			float a[kBlock], c[kBlock], l[kBlock];
#pragma unroll
			for (int k = 0; k < kBlock; ++k) {
				a[k] = at(i + k, s);
				c[k] = lc[i + k];
				l[k] = ll[i + k];
			}
#pragma unroll
			for (int k = 0; k < kBlock; ++k) {
				z = __fmul_rn(__fsub_rn(a[k], __fmul_rn(c[k], z)), l[k]);
				a[k] = z;
			}
			if (keep)
#pragma unroll
				for (int k = 0; k < kBlock; ++k)
					at(i + k, s) = a[k];
		}
		for (; i < end; ++i) {
			z = __fmul_rn(__fsub_rn(at(i, s), __fmul_rn(lc[i], z)), ll[i]);
			if (keep)
				at(i, s) = z;
		}
		return z;
	};
	auto backward = [&](float w, int i, int end, bool keep) {
		for (; i - kBlock + 1 >= end; i -= kBlock) {
			float a[kBlock], u[kBlock];
#pragma unroll
			for (int k = 0; k < kBlock; ++k) {
				a[k] = at(i - k, s);
				u[k] = lu[i - k];
			}
#pragma unroll
			for (int k = 0; k < kBlock; ++k) {
				w = __fsub_rn(a[k], __fmul_rn(u[k], w));
				a[k] = w;
			}
			if (keep)
#pragma unroll
				for (int k = 0; k < kBlock; ++k)
					at(i - k, s) = a[k];
		}
		for (; i >= end; --i) {
			w = __fsub_rn(at(i, s), __fmul_rn(lu[i], w));
			if (keep)
				at(i, s) = w;
		}
		return w;
	};

	float z0 = on ? forward(0.0f, max(0, b - reach), b, false) : 0.0f;
	__syncthreads();
	if (on)
		forward(z0, b, e, true);
	__syncthreads();
	for (;;) {
		const float is = on && chunk > 0 ? at(b - 1, s) : z0;
		const bool redo = __float_as_uint(is) != __float_as_uint(z0);
		if (!__syncthreads_or(redo))
			break;
		if (redo) {
			z0 = is;
			for (int i = b; i < e; i += kDots)
				dots(i, 1, e, s, 0);
			forward(z0, b, e, true);
		}
		__syncthreads();
	}
	float w0 = on ? backward(0.0f, min(n, e + reach) - 1, e, false) : 0.0f;
	__syncthreads();
	if (on)
		backward(w0, e - 1, b, true);
	__syncthreads();
	for (;;) {
		const float is = on && e < n ? at(e, s) : w0;
		const bool redo = __float_as_uint(is) != __float_as_uint(w0);
		if (!__syncthreads_or(redo))
			break;
		if (redo) {
			w0 = is;
			for (int i = b; i < e; i += kDots)
				dots(i, 1, e, s, 0);
			forward(z0, b, e, true);
			backward(w0, e - 1, b, true);
		}
		__syncthreads();
	}
	if (H) {
		for (int q = 0; q < series; ++q)
			for (int i = threadIdx.x; i < n; i += blockDim.x)
				reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(first + q) * ds)[i] = at(i, q);
	} else {
		const int q = threadIdx.x & (L.series - 1), rows = blockDim.x / L.series;
		if (q < series)
			for (int i = threadIdx.x / L.series; i < n; i += rows)
				reinterpret_cast<float *>(dst + static_cast<ptrdiff_t>(i) * ds)[first + q] = at(i, q);
	}
}

// Shape of a block, or series = 0 where the chunked form does not apply.
// Chunks about as long as the reach (their work doubles then), within one
// block; columns 16 to a block (64-byte segments), lines 8, or as many as
// fit the shared memory. Rows of more than kMaxRow taps (about 16x) take the two
// launches: a block has its few outputs' dot products for whole lines then, and
// the two launches spread them out. Two launches against chunks, us: 1920x1080
// -> 192x108 (20 taps) 39 and 23, 8000x4000 -> 400x200 (40) 110 and 116,
// 1920x1080 -> 64x36 (60) 26 and 31, 20000x64 -> 200x64 (200) 35 and 121.
constexpr unsigned kMaxRow = 32;

ChunkShape chunk_shape(const UnresizeTables &t, bool horizontal, size_t *smem)
{
	constexpr size_t kMaxSmem = 227 * 1024;
	ChunkShape L{};
	if (!t.reach || t.row_size > kMaxRow)
		return L;
	const int n = static_cast<int>(t.orig);
	L.pitch = n | 1;
	for (int series = horizontal ? 8 : 16; series >= 1; series /= 2) {
		*smem = ((4 + static_cast<size_t>(t.row_size)) * n + static_cast<size_t>(L.pitch) * series) * 4;
		if (*smem > kMaxSmem)
			continue;
		const int most = kChunkThreads / series;
		L.length = std::max<int>(t.reach + 8, (n + most - 1) / most) | 1;
		L.chunks = (n + L.length - 1) / L.length;
		L.series = series;
		return L;
	}
	return L;
}

} // namespace

cudaError_t launch_unresize(const UnresizeTables &t, bool horizontal, unsigned lines_or_cols, const void *src,
                            ptrdiff_t src_stride, void *dst, ptrdiff_t dst_stride, cudaStream_t stream)
{
	if (!lines_or_cols || !t.orig)
		return cudaSuccess;
	const unsigned n = lines_or_cols;
	const char *s = static_cast<const char *>(src);
	char *d = static_cast<char *>(dst);
	constexpr unsigned kGridY = 65535;  // CUDA's limit; the kernels stride over the rest
	size_t smem = 0;
	const ChunkShape L = chunk_shape(t, horizontal, &smem);
	if (L.series) {
		const auto kernel = horizontal ? unresize_lines<true> : unresize_lines<false>;
		static std::atomic<unsigned long long> devices[2] = {};
		cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(kernel), 227 * 1024, devices[horizontal]);
		if (e != cudaSuccess)
			return e;
		// the dot products and the copies out want more threads than the chunks
		const unsigned threads = kChunkThreads;
		kernel<<<(n + L.series - 1) / L.series, threads, smem, stream>>>(t, L, n, s, src_stride, d, dst_stride);
		return cudaGetLastError();
	}
	if (horizontal) {
		unresize_dot_h<<<dim3((t.orig + kThreads - 1) / kThreads, std::min(n, kGridY)), kThreads, 0, stream>>>(
			t, n, s, src_stride, d, dst_stride);
		unresize_subst_h<<<(n + kTile - 1) / kTile, 32, 0, stream>>>(t, n, d, dst_stride);
	} else {
		unresize_dot_v<<<dim3((n + kThreads - 1) / kThreads, std::min(t.orig, kGridY)), kThreads, 0, stream>>>(
			t, n, s, src_stride, d, dst_stride);
		unresize_subst_v<<<(n + kThreads - 1) / kThreads, kThreads, 0, stream>>>(t, n, d, dst_stride);
	}
	return cudaGetLastError();
}

} // namespace zg
