// Floyd-Steinberg error diffusion of whole planes to BYTE or WORD (zimg's
// ErrorDiffusion, src/zimg/depth/dither.cpp:59-85 per line and 291-345 over
// the plane), equal bit for bit to zimg's C path.
//
// The recurrence is serial along a line (each sample takes the error of its
// left neighbour) and across lines (the three samples above it, columns
// c - 1 .. c + 1). Lines therefore run as a wavefront: one lane per line,
// 32 lines to a warp ("band"), line r of a band at column c on band step
// c + 3r. A lane needs the line above's error at column c + 1 two steps after
// that lane made it, so the value crosses lanes by shuffle off the critical
// path, which is the left neighbour's error (nine dependent float operations
// a sample). The last line of a band hands its errors to the first line of
// the next.
//
// ed_cluster_kernel runs a plane on a cluster of up to 8 SMs, two or four
// computing warps each (cluster_warps), one to a scheduler; two more warps for
// each of them move its data, with two on schedulers of their own, with four
// beside them. The warps run free of one another and hand errors on through
// distributed shared memory. ed_kernel (one block a plane, a block barrier every 16 steps)
// stays for planes whose lines do not fit the cluster's hand-off buffers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "depth.h"
#include "depth_device.cuh"
#include "launch_attr.h"
#include "pipeline.cuh"

namespace zg {

namespace {

constexpr int kBandLines = 32;
constexpr int kTile = kBandLines * kEdPitch;       // words per staging tile
constexpr int kTail = kEdLag * (kBandLines - 1);   // steps line 31 runs behind line 0
// Line 0 of a band reads the line above at column c + 3 on step c, written
// on step c + 3 + kTail of the previous band: spacing - kTail - 3 >= kEdChunk
// puts the write one barrier before the read.
constexpr int kMinSpacing = ((kTail + 3 + kEdChunk + kEdChunk - 1) / kEdChunk) * kEdChunk;
constexpr int kMaxWarps = 32;
constexpr size_t kMaxSmem = 227 * 1024;

// Where a warp is on the current chunk: the band it owns and the band's
// step; live while that band has work left. Warp w starts at global step
// w * spacing and moves to band + warps every `cycle` steps.
struct Where {
	int band, step;
	bool live;
};

__device__ __forceinline__ bool where_live(const Where &x, int rel, const EdPlane &p)
{
	return rel >= 0 && x.band < p.bands && x.step < kTail + p.width;
}

// The next chunk's position (rel: global step - w * spacing, advanced here).
__device__ __forceinline__ void where_next(Where &x, int &rel, int w, int nw, const EdPlane &p)
{
	rel += kEdChunk;
	if (rel == 0) {
		x.band = w;
		x.step = 0;
	} else if (rel > 0) {
		x.step += kEdChunk;
		if (x.step >= p.cycle) {
			x.step -= p.cycle;
			x.band += nw;
		}
	}
	x.live = where_live(x, rel, p);
}

template <class T, class U>
__global__ void __launch_bounds__(kMaxWarps * 32) ed_kernel(const __grid_constant__ EdLaunch L)
{
	extern __shared__ __align__(16) float ed_smem[];
	const EdPlane &p = L.planes[blockIdx.x];
	const int nw = L.warps, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int per_warp = 2 * kTile + L.ring;
	float *tile_in = ed_smem + w * per_warp;
	uint32_t *tile_out = reinterpret_cast<uint32_t *>(tile_in + kTile);
	float *ring = tile_in + 2 * kTile;
	const float *ring_above = ed_smem + ((w + nw - 1) % nw) * per_warp + 2 * kTile;
	const int rmask = L.ring - 1;
	const int W = p.width, H = p.height;
	const float scale = p.scale, offset = p.offset, vmax = p.vmax;
	// staging: transfer j of a lane covers line 2j + half of the band, step t16
	const int half = lane >> 4, t16 = lane & 15;

	T pre[kEdChunk];
	auto fetch = [&](const Where &wh) {
		if (!wh.live) {
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j)
				pre[j] = T{};
			return;
		}
		const int rows_left = H - wh.band * kBandLines - half;  // line 2j + half exists iff 2j < rows_left
		const char *base = static_cast<const char *>(p.src) +
		                   static_cast<ptrdiff_t>(wh.band * kBandLines + half) * p.src_stride;
		const ptrdiff_t step2 = 2 * p.src_stride;
		const int cb = wh.step + t16 - kEdLag * half;
#pragma unroll
		for (int j = 0; j < kEdChunk; ++j) {
			const int c = cb - 2 * kEdLag * j;
			const bool ok = 2 * j < rows_left && static_cast<unsigned>(c) < static_cast<unsigned>(W);
			pre[j] = ok ? reinterpret_cast<const T *>(base + j * step2)[c] : T{};
		}
	};

	// errors: left neighbour; h2 / h3 / h4 the line above at columns c + 1,
	// c, c - 1 for this step, h1 the one for the next step
	float left = 0.0f, h1 = 0.0f, h2 = 0.0f, h3 = 0.0f, h4 = 0.0f;
	int rel = -w * p.spacing;
	Where cur{ w, 0, false };
	cur.live = where_live(cur, rel, p);
	fetch(cur);
	for (int s0 = 0; s0 < p.steps; s0 += kEdChunk) {
		Where nxt = cur;
		int rel_next = rel;
		where_next(nxt, rel_next, w, nw, p);
		if (cur.live) {
			// x = sample * scale + offset, two roundings (dither.cpp:76)
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j)
				tile_in[(2 * j + half) * kEdPitch + t16] =
					__fadd_rn(__fmul_rn(sample_to_float(pre[j]), scale), offset);
		}
		fetch(nxt);
		__syncwarp();
		if (cur.live) {
			if (cur.step == 0) {
				// a band starts: line 0 takes the first three errors of the
				// line above from the previous band's ring (zero above line 0)
				left = h1 = h2 = h3 = h4 = 0.0f;
				if (lane == 0 && cur.band > 0) {
					h3 = ring_above[0];
					h2 = W > 1 ? ring_above[1] : 0.0f;
					h1 = W > 2 ? ring_above[2] : 0.0f;
				}
			}
			const bool row_ok = cur.band * kBandLines + lane < H;
			const bool above = cur.band > 0;
			const int c0 = cur.step - kEdLag * lane;
			// Branch-free steps: every lane computes, inactive lanes (before
			// or after their line, or below the plane) keep a zero error.
#pragma unroll
			for (int t = 0; t < kEdChunk; ++t) {
				const int c = c0 + t;
				const bool act = row_ok && static_cast<unsigned>(c) < static_cast<unsigned>(W);
				// left * 7/16 + top-right * 3/16 + top * 5/16 + top-left *
				// 1/16, in that order (dither.cpp:78-83). zimg's sum starts
				// from 0, which only turns a -0 into +0: the sample's base is
				// never -0 (x * scale + offset with offset never -0), so a
				// zero's sign cannot reach x and the start is left out.
				float err = __fmul_rn(left, 0.4375f);
				err = __fadd_rn(err, __fmul_rn(h2, 0.1875f));
				err = __fadd_rn(err, __fmul_rn(h3, 0.3125f));
				err = __fadd_rn(err, __fmul_rn(h4, 0.0625f));
				const float x = __fadd_rn(tile_in[lane * kEdPitch + t], err);
				// std::clamp to [0, vmax] (x is never -0); a NaN clamps to 0
				// here, stores 0 as zimg's lrint does, and keeps its NaN as
				// the error below
				const float xc = fminf(fmaxf(x, 0.0f), vmax);
				// nearest even: xc + 1.5 * 2^23 has an ulp of 1 for
				// 0 <= xc < 2^22
				const float r = __fadd_rn(xc, 12582912.0f);
				const float y = __fsub_rn(r, 12582912.0f);
				tile_out[lane * kEdPitch + t] = __float_as_uint(r) & 0xFFFFu;
				const float e = act ? (x != x ? x : __fsub_rn(xc, y)) : 0.0f;
				if (lane == kBandLines - 1 && act)
					ring[c & rmask] = e;
				left = e;
				const float down = __shfl_up_sync(0xffffffffu, e, 1);
				// line 0 reads the previous band's last line instead; every
				// lane loads its slot (lanes are 3 columns apart: distinct
				// banks) and line 0 keeps it
				const int c3 = c + kEdLag;
				const float ra = ring_above[c3 & rmask];
				const float u = lane != 0 ? down : ((above && static_cast<unsigned>(c3) < static_cast<unsigned>(W)) ? ra : 0.0f);
				h4 = h3;
				h3 = h2;
				h2 = h1;
				h1 = u;
			}
		}
		__syncwarp();
		if (cur.live) {
			const int rows_left = H - cur.band * kBandLines - half;
			char *base = static_cast<char *>(p.dst) + static_cast<ptrdiff_t>(cur.band * kBandLines + half) * p.dst_stride;
			const ptrdiff_t step2 = 2 * p.dst_stride;
			const int cb = cur.step + t16 - kEdLag * half;
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j) {
				const int c = cb - 2 * kEdLag * j;
				if (2 * j < rows_left && static_cast<unsigned>(c) < static_cast<unsigned>(W))
					reinterpret_cast<U *>(base + j * step2)[c] = static_cast<U>(tile_out[(2 * j + half) * kEdPitch + t16]);
			}
		}
		// ring writes of this chunk become visible to the next band's warp
		__syncthreads();
		cur = nxt;
		rel = rel_next;
	}
}

// ------------------------------------------------- one plane on a cluster --
// Bound: the chain of a step (multiply, four adds, the clamp, the rounding add
// and subtract, the error) times width + 93 steps of a band plus about 120
// steps per band before it. Warp w of the cluster's computing warps takes
// bands w, w + warps, ...; warps, not blocks, wait on each other.
//
// A computing warp does the steps alone; two more warps move its data
// meanwhile. The loading one converts the next chunk's inputs into a staging
// tile and waits for the errors of the band above, the storing one hands the
// band's last errors on and stores the previous chunk's outputs (one named
// barrier of the three per chunk of 16 steps, two tiles each way). In one warp
// the transfers ran after the steps and not beside them, 4,600 cycles a chunk,
// 860 of them the steps. A block has two computing warps on two of its
// schedulers and the moving ones on the other two, or, for planes that need
// more bands in flight, four with the moving ones beside them (cluster_warps).
//
// Hand-off: the errors of a band's last line go, by band step, into the
// receive buffer of the next band's warp with st.async, 16 bytes a lane,
// which completes on the mbarrier of that chunk beside the buffer (one a
// chunk, so that the writer may run any number of chunks ahead; a phase a
// band). Plain stores and a flag with release order instead cost the writer
// 900 cycles a chunk. A buffer holds a whole line, so the writer never waits:
// a warp's next band is written only by a band that depends on every sample
// the warp's current band has read. Waits are bounded (hand_off_wait): one that
// runs out is recorded in g_ed_wait_error and the warp goes on without waiting,
// so that the launch ends, its outputs wrong from there on; the cluster's blocks
// then stay until every hand-off on its way must have landed (leave_cluster).
//
// Measured, a 1920x1080 4:2:0 frame, WORD 10 bits -> BYTE, its planes side by
// side: 1,185 us in ed_kernel, 224 us here (about 1,250 cycles a chunk; the
// steps alone, one warp on an idle SM, take 52 cycles, 47 without the
// shuffle, of which the dependent operations are 40).
constexpr int kMaxClusterWarps = 4;                   // computing warps per block: 2 or 4
constexpr int kClusterThreads = 3 * kMaxClusterWarps * 32;
constexpr int kMaxCluster = 8;                        // blocks per cluster (the portable limit)
constexpr int kRowPitch = 20;                         // words of a line in a staging tile: conflict-free 16-byte rows
constexpr int kStage = kBandLines * kRowPitch;        // words of a staging tile
constexpr int kReadAhead = kTail + kEdLag;            // line 0's step s reads the writer's step s + 96
constexpr int kWarpFloats = 4 * kStage + 2 * kEdChunk;
constexpr int kAheadChunks = kReadAhead / kEdChunk + 1;  // so chunk k needs the writer's chunks below k + 7
static_assert(kReadAhead % kEdChunk == 0, "receive reads start on chunk boundaries");

__device__ int g_ed_wait_error;
// Wait limit in ns (0: kWaitNs), and a test hook: the chunk whose hand-off a
// plane's first band leaves out (-1: none).
__device__ unsigned long long g_ed_wait_ns;
__device__ int g_ed_drop_chunk = -1;

// floats of one warp's receive buffer for lines of `width` samples: a slot
// per band step, and the zeros that the last chunks read past them
__host__ __device__ constexpr int receive_floats(int chunks)
{
	return chunks * kEdChunk + kReadAhead + 2 * kEdChunk;
}

// its receive buffer and the mbarriers of its chunks, in floats
__host__ __device__ constexpr int hand_off_floats(int chunks)
{
	return receive_floats(chunks) + (2 * chunks + 3) / 4 * 4;
}

__host__ __device__ constexpr int band_chunks(int width)
{
	return (width + kTail + kEdChunk - 1) / kEdChunk;
}

size_t cluster_smem_bytes(int warps, int hand_off)
{
	return static_cast<size_t>(warps) * (kWarpFloats + hand_off) * 4;
}

__device__ __forceinline__ uint32_t cluster_addr(const void *p, unsigned rank)
{
	uint32_t r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;\n"
	    : "=r"(r)
	    : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
	return r;
}

__device__ __forceinline__ void cluster_barrier()
{
	asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// Wait for a hand-off. Gives up (false) after the limit in ns of the clock and
// then kOwnPolls polls of the warp's own, a microsecond apart: while the GPU
// runs another process's work the clock goes on, but neither side of a hand-off
// does. (A call of its own: inlined, it costs the loading warp spills.)
constexpr int kOwnPolls = 1 << 15;

__device__ __noinline__ bool hand_off_pending(uint64_t *bar, unsigned parity)
{
	if (mbar_wait(bar, parity, g_ed_wait_ns ? g_ed_wait_ns : kWaitNs))
		return true;
	for (int i = 0; i < kOwnPolls; ++i) {
		if (mbar_test(bar, parity))
			return true;
		__nanosleep(1000);
	}
	return false;
}

__device__ __forceinline__ bool hand_off_wait(uint64_t *bar, unsigned parity)
{
	return mbar_test(bar, parity) || hand_off_pending(bar, parity);
}

// A word of a block's shared memory that is 0 until a warp of the cluster has
// given up a wait: the last float of its first warp's receive buffer, beyond
// what a line reads.
__device__ __forceinline__ float *lost_word(float *smem, int chunks)
{
	return smem + kWarpFloats + receive_floats(chunks) - 1;
}

// The end of a block: none leaves while another may write to its shared memory.
// All hand-offs were sent by then, and waited for unless a warp has given up;
// then they get a millisecond, thousands of times what they take.
__device__ __forceinline__ void leave_cluster(float *smem, int chunks)
{
	cluster_barrier();
	for (int i = 0; i < 1000 && *static_cast<volatile float *>(lost_word(smem, chunks)) != 0.0f; ++i)
		__nanosleep(1000);
}

// Clamps that keep a NaN (PTX max.NaN / min.NaN), as zimg's std::clamp does.
__device__ __forceinline__ float clamp_nan(float x, float hi)
{
	asm("max.NaN.f32 %0, %0, 0f00000000;\n"
	    "min.NaN.f32 %0, %0, %1;\n"
	    : "+f"(x)
	    : "f"(hi));
	return x;
}

// The barrier of computing warp `warp` and the two that move its data.
__device__ __forceinline__ void chunk_barrier(int warp)
{
	asm volatile("bar.sync %0, 96;\n" ::"r"(warp + 1) : "memory");
}

// An integer sample as float without a conversion instruction (a quarter of
// the issue rate): its bits below 2^23, minus 2^23.
template <class T>
__device__ __forceinline__ float staged_sample(T v)
{
	if constexpr (std::is_same_v<T, uint8_t> || std::is_same_v<T, uint16_t>)
		return __fsub_rn(__uint_as_float(0x4B000000u | v), 8388608.0f);
	else
		return sample_to_float(v);
}

// A store under a predicate, without a branch.
__device__ __forceinline__ void store_if(bool on, uint8_t *p, uint8_t v)
{
	asm volatile("{\n.reg .pred q;\nsetp.ne.s32 q, %0, 0;\n@q st.global.u8 [%1], %2;\n}\n" ::"r"(static_cast<int>(on)),
	             "l"(p), "r"(static_cast<unsigned>(v))
	             : "memory");
}

__device__ __forceinline__ void store_if(bool on, uint16_t *p, uint16_t v)
{
	asm volatile("{\n.reg .pred q;\nsetp.ne.s32 q, %0, 0;\n@q st.global.u16 [%1], %2;\n}\n" ::"r"(static_cast<int>(on)),
	             "l"(p), "h"(v)
	             : "memory");
}

// One warp's shared memory: two input tiles, two output tiles, the last
// line's errors of two chunks, the receive buffer and its mbarriers.
struct EdShared {
	float *tile_in;
	uint32_t *tile_out;
	float *last;
	float *recv;
	uint64_t *bars;
};

// Transfer j of a moving warp's lane covers line 2j + half of the band at step
// t16 of the chunk: half a warp along 16 samples of a line.
struct EdLane {
	int half, t16, c16;
	__device__ __forceinline__ EdLane()
	{
		const int lane = threadIdx.x & 31;
		half = lane >> 4;
		t16 = lane & 15;
		c16 = t16 - kEdLag * half;
	}
};

// Chunks whose 32 x 16 samples all exist need no compares.
__device__ __forceinline__ bool whole_chunk(const EdPlane &p, int band, int k)
{
	return (band + 1) * kBandLines <= p.height && k * kEdChunk >= kTail && (k + 1) * kEdChunk <= p.width;
}

// The loading warp: inputs into tile_in, and the wait for the errors that the
// computing warp reads next.
template <class T>
__device__ __forceinline__ void ed_load(const EdPlane &p, int first_band, int nw, int warp, const EdShared &m, float *lost,
                                        int cluster)
{
	const EdLane l;
	const int lane = threadIdx.x & 31;
	const int W = p.width, H = p.height, chunks = band_chunks(W);
	const float scale = p.scale, offset = p.offset;
	const ptrdiff_t step = 2 * p.src_stride - 2 * kEdLag * static_cast<ptrdiff_t>(sizeof(T));
	unsigned phase = 0;
	bool gave_up = false;
	for (int band = first_band; band < p.bands; band += nw) {
		const char *in0 = static_cast<const char *>(p.src) +
		                  static_cast<ptrdiff_t>(band * kBandLines + l.half) * p.src_stride +
		                  static_cast<ptrdiff_t>(l.c16) * static_cast<ptrdiff_t>(sizeof(T));
		// inputs of two chunks in flight: one chunk's time does not cover the
		// memory's latency
		T even[kEdChunk], odd[kEdChunk];
		auto fetch = [&](T (&pre)[kEdChunk], int k) {
			if (whole_chunk(p, band, k)) {
				const char *a = in0 + static_cast<ptrdiff_t>(k) * static_cast<ptrdiff_t>(kEdChunk * sizeof(T));
#pragma unroll
				for (int j = 0; j < kEdChunk; ++j)
					pre[j] = *reinterpret_cast<const T *>(a + j * step);
				return;
			}
			// lines below the plane are read from its last one, columns
			// outside it from its ends: no branches here either, since a
			// band's first chunks hold up the bands below
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j) {
				const int line = min(band * kBandLines + 2 * j + l.half, H - 1);
				const int c = min(max(k * kEdChunk + l.c16 - 2 * kEdLag * j, 0), W - 1);
				pre[j] = reinterpret_cast<const T *>(static_cast<const char *>(p.src) +
				                                     static_cast<ptrdiff_t>(line) * p.src_stride)[c];
			}
		};
		// x = sample * scale + offset, two roundings (dither.cpp:76)
		auto convert = [&](const T (&pre)[kEdChunk], int k) {
			float *t = m.tile_in + (k & 1) * kStage + l.half * kRowPitch + l.t16;
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j)
				t[2 * j * kRowPitch] = __fadd_rn(__fmul_rn(staged_sample(pre[j]), scale), offset);
			if (whole_chunk(p, band, k))
				return;
			// columns outside the plane: a base so low that the sample clamps
			// to 0 and its error is 0. (A NaN among the errors above makes it
			// one, but then the same errors do that to the neighbour inside
			// the plane that would read it.)
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j)
				if (static_cast<unsigned>(k * kEdChunk + l.c16 - 2 * kEdLag * j) >= static_cast<unsigned>(W))
					t[2 * j * kRowPitch] = -1.0e9f;
		};
		// the errors that chunk k reads have arrived; their mbarriers are
		// armed again for the warp's next band
		int arrived = 0;
		auto receive = [&](int k) {
			if (band == 0)
				return;
			for (const int need = min(k + kAheadChunks, chunks); arrived < need && !gave_up; ++arrived) {
				if (!__all_sync(0xffffffffu, hand_off_wait(m.bars + arrived, phase))) {
					gave_up = true;
					atomicExch(&g_ed_wait_error, 1);
					if (lane < cluster)
						asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(cluster_addr(lost, lane)), "f"(1.0f) : "memory");
				} else if (lane == 0) {
					mbar_arrive_expect_tx(m.bars + arrived, kEdChunk * 4);
				}
			}
		};
		fetch(even, 0);
		fetch(odd, 1);
		convert(even, 0);
		fetch(even, 2);
		receive(0);
		chunk_barrier(warp);  // chunk 0's inputs are there
		auto chunk = [&](T (&pre)[kEdChunk], int k) {
			convert(pre, k + 1);
			fetch(pre, k + 3);
			if (k + 1 < chunks)
				receive(k + 1);
			chunk_barrier(warp);  // chunk k is done, chunk k + 1's inputs are there
		};
		for (int k = 0; k < chunks; k += 2) {
			chunk(odd, k);
			if (k + 1 < chunks)
				chunk(even, k + 1);
		}
		if (band > 0)
			phase ^= 1;
	}
}

// The storing warp: outputs from tile_out, the last line's errors from `last`
// to the next band's warp (next_recv, next_bars: its buffer and mbarriers).
template <class U>
__device__ __forceinline__ void ed_store(const EdPlane &p, int first_band, int nw, int warp, const EdShared &m,
                                         uint32_t next_recv, uint32_t next_bars)
{
	const EdLane l;
	const int lane = threadIdx.x & 31;
	const int W = p.width, H = p.height, chunks = band_chunks(W);
	const ptrdiff_t step = 2 * p.dst_stride - 2 * kEdLag * static_cast<ptrdiff_t>(sizeof(U));
	const int drop = first_band == 0 ? g_ed_drop_chunk : -1;
	for (int band = first_band; band < p.bands; band += nw) {
		const int rows_left = H - band * kBandLines - l.half;  // line 2j + half exists iff 2j < rows_left
		char *out0 = static_cast<char *>(p.dst) + static_cast<ptrdiff_t>(band * kBandLines + l.half) * p.dst_stride +
		             static_cast<ptrdiff_t>(l.c16) * static_cast<ptrdiff_t>(sizeof(U));
		chunk_barrier(warp);
		for (int k = 0; k < chunks; ++k) {
			chunk_barrier(warp);  // chunk k is done
			if (lane < kEdChunk / 4 && band + 1 < p.bands && (band > 0 || k != drop)) {
				const float4 v = *reinterpret_cast<const float4 *>(m.last + (k & 1) * kEdChunk + 4 * lane);
				asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(
					             next_recv + static_cast<uint32_t>(k * kEdChunk + 4 * lane) * 4),
				             "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(next_bars + static_cast<uint32_t>(k) * 8)
				             : "memory");
			}
			__syncwarp();
			char *a = out0 + static_cast<ptrdiff_t>(k) * static_cast<ptrdiff_t>(kEdChunk * sizeof(U));
			const U *t = reinterpret_cast<const U *>(m.tile_out + (k & 1) * kStage + l.half * kRowPitch) + l.t16;
			constexpr int kLine2 = 2 * kRowPitch * (4 / static_cast<int>(sizeof(U)));
			U v[kEdChunk];
#pragma unroll
			for (int j = 0; j < kEdChunk; ++j)
				v[j] = t[j * kLine2];
			if (whole_chunk(p, band, k)) {
#pragma unroll
				for (int j = 0; j < kEdChunk; ++j)
					*reinterpret_cast<U *>(a + j * step) = v[j];
			} else {
				const int cb = k * kEdChunk + l.c16;
#pragma unroll
				for (int j = 0; j < kEdChunk; ++j)
					store_if(2 * j < rows_left && static_cast<unsigned>(cb - 2 * kEdLag * j) < static_cast<unsigned>(W),
					         reinterpret_cast<U *>(a + j * step), v[j]);
			}
		}
	}
}

template <class T, class U>
__global__ void __launch_bounds__(kClusterThreads, 1) ed_cluster_kernel(const __grid_constant__ EdLaunch L)
{
	extern __shared__ __align__(16) float ed_smem[];
	// C computing warps in each of `cluster` blocks. C = 2: warps 0, 1 compute,
	// 2, 3 load, 6, 7 store (4 and 5 would share the computing warps'
	// schedulers and do nothing); C = 4: 0-3, 4-7, 8-11
	const int C = blockDim.x == kClusterThreads ? 4 : 2;
	const int cluster = L.warps / C;
	const EdPlane &p = L.planes[blockIdx.x / cluster];
	const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int role = C == 4 ? wid >> 2 : (wid < 2 ? 0 : (wid < 4 ? 1 : (wid < 6 ? 3 : 2)));
	const int warp = wid % C;
	const int nw = L.warps, g = (blockIdx.x % cluster) * C + warp;
	const int next = (g + 1) % nw;
	const int W = p.width, chunks = band_chunks(W);
	const int per_warp = kWarpFloats + L.ring;
	EdShared m;
	m.tile_in = ed_smem + warp * per_warp;
	m.tile_out = reinterpret_cast<uint32_t *>(m.tile_in + 2 * kStage);
	m.last = m.tile_in + 4 * kStage;
	m.recv = m.tile_in + kWarpFloats;
	m.bars = reinterpret_cast<uint64_t *>(m.recv + receive_floats(chunks));
	if (role == 0) {
		// the first band's reads find zeros, as the last chunks' past the line do
		for (int i = (g == 0 ? 0 : chunks * kEdChunk) + lane; i < receive_floats(chunks); i += 32)
			m.recv[i] = 0.0f;
		for (int i = lane; i < chunks; i += 32) {
			mbar_init(m.bars + i, 1);
			mbar_arrive_expect_tx(m.bars + i, kEdChunk * 4);
		}
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
	}
	cluster_barrier();

	if (role == 1) {
		ed_load<T>(p, g, nw, warp, m, lost_word(ed_smem, chunks), cluster);
		leave_cluster(ed_smem, chunks);
		return;
	}
	if (role >= 2) {
		const float *next_recv = ed_smem + (next % C) * per_warp + kWarpFloats;
		if (role == 2)
			ed_store<U>(p, g, nw, warp, m, cluster_addr(next_recv, next / C),
			            cluster_addr(next_recv + receive_floats(chunks), next / C));
		leave_cluster(ed_smem, chunks);
		return;
	}
	const float vmax = p.vmax;
	constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: an ulp of 1 for 0 <= x < 2^22, so nearest even
	for (int band = g; band < p.bands; band += nw) {
		// errors: left neighbour; h2 / h3 / h4 the line above at columns
		// c + 1, c, c - 1 for this step; down / above the one for the next
		// step, chosen only then, so that no step waits for its own shuffle
		float left = 0.0f, h2 = 0.0f, h3 = 0.0f, h4 = 0.0f, down = 0.0f, above = 0.0f;
		chunk_barrier(warp);
		for (int k = 0; k < chunks; ++k) {
			const float *xin = m.tile_in + (k & 1) * kStage + lane * kRowPitch;
			const float *uin = m.recv + k * kEdChunk + kReadAhead;
			uint32_t *row = m.tile_out + (k & 1) * kStage + lane * kRowPitch;
			float *last = m.last + (k & 1) * kEdChunk;
			if (k == 0 && band > 0 && lane == 0) {
				h3 = m.recv[kTail];
				h2 = m.recv[kTail + 1];
				above = m.recv[kTail + 2];
			}
			float u[kEdChunk], x0[kEdChunk], err[kEdChunk];
			uint32_t out[kEdChunk];
#pragma unroll
			for (int q = 0; q < kEdChunk / 4; ++q) {
				*reinterpret_cast<float4 *>(x0 + 4 * q) = *reinterpret_cast<const float4 *>(xin + 4 * q);
				*reinterpret_cast<float4 *>(u + 4 * q) = *reinterpret_cast<const float4 *>(uin + 4 * q);
			}
#pragma unroll
			for (int t = 0; t < kEdChunk; ++t) {
				// left * 7/16 + top-right * 3/16 + top * 5/16 + top-left *
				// 1/16, in that order (dither.cpp:78-83). zimg's sum starts
				// from 0, which only turns a -0 into +0: the sample's base
				// is never -0 (x * scale + offset with offset never -0), so
				// a zero's sign cannot reach x and the start is left out.
				float d = __fmul_rn(left, 0.4375f);
				d = __fadd_rn(d, __fmul_rn(h2, 0.1875f));
				d = __fadd_rn(d, __fmul_rn(h3, 0.3125f));
				d = __fadd_rn(d, __fmul_rn(h4, 0.0625f));
				// the clamp keeps a NaN as the error; it stores 0, as
				// zimg's lrint does. Compares and a select instead of the
				// clamp measured 63 cycles a step against 52: a predicate
				// comes later than a clamped value.
				const float x = clamp_nan(__fadd_rn(x0[t], d), vmax);
				const float r = __fadd_rn(x, kMagic);
				const float e = __fsub_rn(x, __fsub_rn(r, kMagic));
				out[t] = __float_as_uint(fmaxf(r, kMagic));
				err[t] = e;
				left = e;
				h4 = h3;
				h3 = h2;
				h2 = lane != 0 ? down : above;
				down = __shfl_up_sync(0xffffffffu, e, 1);
				above = u[t];
			}
#pragma unroll
			for (int q = 0; q < kEdChunk / 4; ++q) {
				if (lane == kBandLines - 1)
					*reinterpret_cast<float4 *>(last + 4 * q) =
						make_float4(err[4 * q], err[4 * q + 1], err[4 * q + 2], err[4 * q + 3]);
				if constexpr (sizeof(U) == 2)
					*reinterpret_cast<uint2 *>(row + 2 * q) = make_uint2(__byte_perm(out[4 * q], out[4 * q + 1], 0x5410),
					                                                     __byte_perm(out[4 * q + 2], out[4 * q + 3], 0x5410));
			}
			if constexpr (sizeof(U) == 1) {
				uint32_t w[4];
#pragma unroll
				for (int q = 0; q < 4; ++q)
					w[q] = __byte_perm(__byte_perm(out[4 * q], out[4 * q + 1], 0x0040),
					                   __byte_perm(out[4 * q + 2], out[4 * q + 3], 0x0040), 0x5410);
				*reinterpret_cast<uint4 *>(row) = make_uint4(w[0], w[1], w[2], w[3]);
			}
			chunk_barrier(warp);
		}
	}
	leave_cluster(ed_smem, chunks);
}

// Chunk times until a plane's last band ends, with nw warps: a band starts
// about 8 chunks after the one above (7 by the skew, the rest the hand-off),
// or when its warp is free.
long long wavefront_chunks(const EdPlane &p, int nw)
{
	const long long chunks = band_chunks(p.width), b = (p.height + kBandLines - 1) / kBandLines - 1;
	const long long lag = kAheadChunks + 1;
	return lag * nw >= chunks ? b * lag + chunks : b / nw * chunks + b % nw * lag + chunks;
}

// Computing warps per block for these planes: 2 where 16 warps in a cluster
// (2 x 8 blocks) are as fast, 4 otherwise; 0 when the hand-off buffers do not
// fit. A chunk takes about 1,000 cycles with the moving warps on other
// schedulers and 1,300 beside them. 2 admits lines of about 21,000 samples, 4
// of 10,000.
int cluster_warps(const EdLaunch &L)
{
	long long t2 = 0, t4 = 0;
	int hand_off = 0;
	for (int k = 0; k < L.num_planes; ++k) {
		if (L.planes[k].width > (1 << 16))
			return 0;
		t2 = std::max(t2, wavefront_chunks(L.planes[k], 2 * kMaxCluster) * 10);
		t4 = std::max(t4, wavefront_chunks(L.planes[k], 4 * kMaxCluster) * 13);
		hand_off = std::max(hand_off, hand_off_floats(band_chunks(L.planes[k].width)));
	}
	if (t4 < t2 && cluster_smem_bytes(4, hand_off) <= kMaxSmem)
		return 4;
	return cluster_smem_bytes(2, hand_off) <= kMaxSmem ? 2 : 0;
}

template <class T, class U>
cudaError_t launch_cluster(const EdLaunch &L, int warps, cudaStream_t st)
{
	// blocks per cluster: enough warps for the bands
	EdLaunch C = L;
	int cluster = 1;
	C.ring = 0;
	for (int k = 0; k < L.num_planes; ++k) {
		while (cluster < kMaxCluster && cluster * warps < L.planes[k].bands)
			cluster *= 2;
		C.ring = std::max(C.ring, hand_off_floats(band_chunks(L.planes[k].width)));
	}
	C.warps = cluster * warps;
	static std::atomic<unsigned long long> devices{ 0 };
	cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(&ed_cluster_kernel<T, U>),
	                                    static_cast<int>(kMaxSmem), devices);
	if (e != cudaSuccess)
		return e;
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(static_cast<unsigned>(L.num_planes * cluster));
	cfg.blockDim = dim3(warps == 4 ? kClusterThreads : 256);
	cfg.dynamicSmemBytes = cluster_smem_bytes(warps, C.ring);
	cfg.stream = st;
	cudaLaunchAttribute attr{};
	attr.id = cudaLaunchAttributeClusterDimension;
	attr.val.clusterDim.x = static_cast<unsigned>(cluster);
	attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
	cfg.attrs = &attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, ed_cluster_kernel<T, U>, C);
}

template <class T, class U>
cudaError_t launch_tu(const EdLaunch &L, size_t smem, cudaStream_t st)
{
	if (const int warps = cluster_warps(L))
		return launch_cluster<T, U>(L, warps, st);
	static std::atomic<unsigned long long> devices{ 0 };
	cudaError_t e = allow_shared_memory(reinterpret_cast<const void *>(&ed_kernel<T, U>), static_cast<int>(kMaxSmem),
	                                    devices);
	if (e != cudaSuccess)
		return e;
	ed_kernel<T, U><<<L.num_planes, L.warps * 32, smem, st>>>(L);
	return cudaGetLastError();
}

template <class T>
cudaError_t launch_t(const EdLaunch &L, size_t smem, cudaStream_t st)
{
	switch (L.out_type) {
	case 0: return launch_tu<T, uint8_t>(L, smem, st);
	case 1: return launch_tu<T, uint16_t>(L, smem, st);
	default: return cudaErrorInvalidValue;
	}
}

int round_up(int v, int m)
{
	return (v + m - 1) / m * m;
}

} // namespace

int ed_set_fault(int drop_chunk, unsigned long long wait_ns)
{
	if (cudaMemcpyToSymbol(g_ed_drop_chunk, &drop_chunk, sizeof(drop_chunk)) != cudaSuccess ||
	    cudaMemcpyToSymbol(g_ed_wait_ns, &wait_ns, sizeof(wait_ns)) != cudaSuccess)
		return -1;
	return 0;
}

int ed_wait_error(bool reset)
{
	int v = 0;
	if (cudaMemcpyFromSymbol(&v, g_ed_wait_error, sizeof(v)) != cudaSuccess)
		return -1;
	if (reset && v) {
		const int zero = 0;
		cudaMemcpyToSymbol(g_ed_wait_error, &zero, sizeof(zero));
	}
	return v;
}

size_t ed_smem_bytes(int warps, int ring)
{
	return static_cast<size_t>(warps) * (2 * kTile + ring) * sizeof(float);
}

bool ed_shape(EdPlane &p, int warps, int *ring)
{
	if (p.width <= 0 || p.height <= 0 || warps < 1 || warps > kMaxWarps)
		return false;
	p.bands = (p.height + kBandLines - 1) / kBandLines;
	long long spacing = kMinSpacing, cycle = 1LL << 30;
	int r = 32;
	if (p.bands > warps) {
		if (warps < 2)
			return false;
		// a warp's next band starts after its current one ends, and after
		// the next band's line 0 has read the whole ring
		const long long w = p.width;
		spacing = std::max<long long>(spacing, (w + kTail + 1 + warps - 1) / warps);
		spacing = std::max<long long>(spacing, (w + kEdChunk + warps - 2) / (warps - 1));
		spacing = (spacing + kEdChunk - 1) / kEdChunk * kEdChunk;
		cycle = spacing * warps;
		// the ring holds a column until line 0 of the next band has read it
		// one barrier later
		while (r < spacing - (kTail + 3) + kEdChunk && r < (1 << 20))
			r <<= 1;
	}
	if (spacing > (1 << 24) || cycle > (1LL << 30))
		return false;
	const long long steps = (static_cast<long long>(p.bands) - 1) * spacing + kTail + p.width;
	if (steps > (1LL << 30))
		return false;
	p.spacing = static_cast<int>(spacing);
	p.cycle = static_cast<int>(cycle);
	p.steps = round_up(static_cast<int>(steps), kEdChunk);
	*ring = r;
	return ed_smem_bytes(warps, r) <= kMaxSmem;
}

int ed_choose_warps(int width, int height)
{
	const int bands = (height + kBandLines - 1) / kBandLines;
	if (bands <= 1)
		return 1;
	// one step of a warp: ~190 cycles of latency, plus ~54 issued
	// instructions per warp in flight over four schedulers (fitted to
	// measured 540p, 1080p and 2160p planes at 4 to 32 warps)
	constexpr double kChain = 190.0, kIssue = 54.0;
	int best = 0;
	double best_cost = 0.0;
	for (int nw = 2; nw <= kMaxWarps; ++nw) {
		EdPlane p{};
		p.width = width;
		p.height = height;
		int ring = 0;
		if (!ed_shape(p, nw, &ring))
			continue;
		const int in_flight = std::min({ nw, bands, (kTail + width + p.spacing - 1) / p.spacing });
		const double cost = static_cast<double>(p.steps) * (kChain + in_flight * kIssue / 4.0);
		if (!best || cost < best_cost) {
			best = nw;
			best_cost = cost;
		}
	}
	return best;
}

cudaError_t launch_error_diffusion(const EdLaunch &L, cudaStream_t stream)
{
	if (L.num_planes <= 0)
		return cudaSuccess;
	if (L.num_planes > kEdMaxPlanes || L.warps < 1 || L.warps > kMaxWarps || L.ring < 1 || (L.ring & (L.ring - 1)))
		return cudaErrorInvalidValue;
	const size_t smem = ed_smem_bytes(L.warps, L.ring);
	if (smem > kMaxSmem)
		return cudaErrorInvalidValue;
	switch (L.in_type) {
	case 0: return launch_t<uint8_t>(L, smem, stream);
	case 1: return launch_t<uint16_t>(L, smem, stream);
	case 2: return launch_t<Half>(L, smem, stream);
	case 3: return launch_t<float>(L, smem, stream);
	default: return cudaErrorInvalidValue;
	}
}

} // namespace zg
