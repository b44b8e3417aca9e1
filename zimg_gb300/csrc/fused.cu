// Host planning and launch of the fused two-pass tile kernel.
#include "fused.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

namespace zg {

// per-(H_FIRST, kind) instantiation units (fused_inst_*.cu)
const void *fused_kernel_ptr_v_f32(int hw, int vs);
const void *fused_kernel_ptr_h_f32(int hw, int vs);
const void *fused_kernel_ptr_v_i16(int hw, int vs);
const void *fused_kernel_ptr_h_i16(int hw, int vs);

namespace {

constexpr int kHwBuckets[] = { 6, 8, 12, 16 };
constexpr int kVsBuckets[] = { 8, 12, 16, 24 };
constexpr size_t kSmemBudget = 56 * 1024;   // preferred: four CTAs of 128 threads per SM
constexpr size_t kSmemMax = 110 * 1024;     // hard limit: two CTAs per SM
constexpr int kBlockColumns = 4 * 66;       // columns of the intermediate block (fused_kernel.cuh)
constexpr size_t kUnusedBytes = 24 << 20;   // see plan_fused

int bucket_index(const int *b, int n, int v)
{
	for (int i = 0; i < n; ++i)
		if (v <= b[i])
			return i;
	return -1;
}

size_t align_up(size_t x, size_t a)
{
	return (x + a - 1) / a * a;
}

// zimg's int32 sums cannot overflow (sum |tap| * 2^15 + 8192 < 2^31 per row),
// and a row's taps sum to 1 << 14, so that centring the samples is a constant.
bool u16_fits_int32(const FilterTable &t)
{
	for (unsigned i = 0; i < t.rows; ++i) {
		long long mag = 8192, sum = 0;
		for (unsigned k = 0; k < t.width; ++k) {
			const int c = t.i16[static_cast<size_t>(i) * t.width + k];
			mag += static_cast<long long>(std::abs(c)) << 15;
			sum += c;
		}
		if (mag >= (1LL << 31) || sum != (1 << 14))
			return false;
	}
	return true;
}

// A tap's 32 bits as the kernel reads them: the f32 tap or the int16 tap as int32.
uint32_t tap_bits(const FilterTable &t, bool u16, unsigned i, unsigned k)
{
	const size_t at = static_cast<size_t>(i) * t.width + k;
	if (u16)
		return static_cast<uint32_t>(static_cast<int32_t>(t.i16[at]));
	uint32_t v;
	std::memcpy(&v, &t.f32[at], sizeof(v));
	return v;
}

} // namespace


bool plan_fused(const FilterTable &first, const FilterTable &second, bool h_first, bool u16, unsigned depth,
                unsigned src_w, unsigned src_h, unsigned dst_w, unsigned dst_h, FusedPlan *out)
{
	const FilterTable &H = h_first ? first : second;
	const FilterTable &V = h_first ? second : first;
	if (H.rows != dst_w || V.rows != dst_h || H.input_width != src_w || V.input_width != src_h)
		return false;
	if (u16 && (!u16_fits_int32(H) || !u16_fits_int32(V)))
		return false;

	int hw_i = bucket_index(kHwBuckets, 4, static_cast<int>(H.width));
	if (hw_i < 0)
		return false;
	if (!u16 && kHwBuckets[hw_i] == 12)
		hw_i = 3;  // F32: how far a NaN under a zero tap spreads is part of the result
	const int HW = kHwBuckets[hw_i];

	// dense vertical groups; streaming needs non-decreasing group bases
	const int kGroup = group_rows(h_first);
	const int groups = static_cast<int>((dst_h + kGroup - 1) / kGroup);
	int max_span = 0;
	std::vector<int> gbase(groups);
	for (int g = 0; g < groups; ++g) {
		int lo = INT_MAX, hi = INT_MIN;
		for (int j = 0; j < kGroup; ++j) {
			const unsigned i = static_cast<unsigned>(g * kGroup + j);
			if (i >= dst_h)
				break;
			lo = std::min(lo, static_cast<int>(V.left[i]));
			hi = std::max(hi, static_cast<int>(V.left[i] + V.width));
		}
		gbase[g] = lo;
		max_span = std::max(max_span, hi - lo);
		if (g && gbase[g] < gbase[g - 1])
			return false;
	}
	const int vs_i = bucket_index(kVsBuckets, 4, max_span);
	if (vs_i < 0)
		return false;
	const int VS = kVsBuckets[vs_i];

	// V first, the streaming kernel reads every line, a vertical pass alone the
	// lines that have a tap (and its output comes and goes once more): far down
	// with a point filter, and planes so large that the lines between cost more
	// than the second launch, the separate passes are faster. One plane, 9x down,
	// streaming and separate: u16 3840x2160 8.2 and 11.0 us (10 MB), 7680x4320
	// 18.5 and 12.3 (39 MB), f32 3840x2160 10.3 and 11.2 (19 MB), 7680x4320 30.6
	// and 12.4 (77 MB).
	if (!h_first) {
		std::vector<bool> tapped(src_h, false);
		for (unsigned i = 0; i < dst_h; ++i)
			for (unsigned k = 0; k < V.width; ++k)
				tapped[V.left[i] + k] = true;
		const size_t lines = static_cast<size_t>(std::count(tapped.begin(), tapped.end(), true)) + 2 * static_cast<size_t>(dst_h);
		if (lines < src_h && (src_h - lines) * src_w * (u16 ? 2 : 4) > kUnusedBytes)
			return false;
	}

	// strips: output columns (a multiple of 8, at most kStripW) whose inputs
	// stay within the kernel's window; of those the width that needs the
	// fewest warp passes per output: V first, the vertical pass's (quad of
	// columns, half of a step's rows) items fill whole warps or not
	const int col_align = u16 ? 8 : 4;
	const int blocks = static_cast<int>((dst_w + 7) / 8);  // of 8 columns: their first and last inputs
	std::vector<int> block_lo(blocks, INT_MAX), block_hi(blocks, INT_MIN);
	for (unsigned c = 0; c < dst_w; ++c) {
		block_lo[c / 8] = std::min(block_lo[c / 8], static_cast<int>(H.left[c]));
		block_hi[c / 8] = std::max(block_hi[c / 8], static_cast<int>(H.left[c]) + HW);
	}
	auto windows = [&](int w, std::vector<int> &win) {
		const int n = static_cast<int>((dst_w + w - 1) / w);
		win.assign(2 * n, 0);
		int widest = 0;
		for (int s = 0; s < n; ++s) {
			int lo = INT_MAX, hi = INT_MIN;
			for (int k = s * w / 8; k < std::min(blocks, (s + 1) * w / 8); ++k) {
				lo = std::min(lo, block_lo[k]);
				hi = std::max(hi, block_hi[k]);
			}
			win[2 * s] = lo / col_align * col_align;
			win[2 * s + 1] = hi;
			widest = std::max(widest, (hi - win[2 * s] + 7) & ~7);
		}
		return widest;
	};
	int strip_w = 0;
	double best = 0;
	std::vector<int> win_col, win;
	for (int w = kStripW; w >= 8; w -= 8) {
		const int widest = windows(w, win);
		if (widest > kStreamWindow)
			continue;
		const int v_warps = h_first ? 4 : (widest / 2 + 31) / 32, h_warps = (w + 31) / 32;
		const double cost = (2.0 * v_warps * VS + h_warps * 2.0 * HW + 40) / w;
		if (!strip_w || cost < 0.97 * best) {
			strip_w = w;
			best = cost;
			win_col = win;
		}
	}
	if (!strip_w)
		return false;
	const int strips = static_cast<int>(win_col.size() / 2);

	// steps of four groups; the lines a step's windows span. H first: in
	// multiples of four, the lines of a horizontal iteration
	const int steps = (groups + 3) / 4;
	std::vector<int> ranges(2 * steps);
	for (int k = 0; k < steps; ++k) {
		const int lo = gbase[4 * k], hi = gbase[std::min(groups, 4 * k + 4) - 1] + VS;
		ranges[2 * k] = h_first ? lo / 4 * 4 : lo;
		ranges[2 * k + 1] = h_first ? (hi + 3) / 4 * 4 : hi;
	}
	// any step may start an item, when its new lines are its whole range, and
	// brings in every line from the end of the step before: more than its range
	// where that starts beyond (a point filter 5.5x and more down the columns);
	// early: the next step's lines arrive beside this one's
	int rows_late = 4, rows_early = 4;
	for (int k = 0; k < steps; ++k) {
		rows_late = std::max(rows_late, ranges[2 * k + 1] - (k ? std::min(ranges[2 * k], ranges[2 * k - 1]) : ranges[0]));
		rows_early = std::max(rows_early, ranges[2 * std::min(k + 1, steps - 1) + 1] - ranges[2 * k]);
	}

	FusedPlan &p = *out;
	p = FusedPlan{};
	FusedJob &J = p.job;
	J.h_first = h_first ? 1 : 0;
	J.kind = static_cast<int>(u16 ? FusedKind::U16_INT : FusedKind::F32);
	J.hw = HW;
	J.vs = VS;
	J.step_groups = 4;
	J.groups = groups;
	J.seg_groups = 4;  // work units: (strip, step) pairs
	J.segments = steps;
	J.ring_rows = h_first ? rows_late : 0;
	// lines a step ahead where four CTAs still fit an SM, else only after the
	// pass that reads the ring if that lets them fit
	bool fits = false;
	for (size_t budget : { kSmemBudget, kSmemMax })
		for (int ahead = 1; ahead >= 0 && !fits; --ahead) {
			J.depth = ahead;
			J.in_rows = ahead ? rows_early : rows_late;
			const FusedPlan *pp = &p;
			fits = static_cast<size_t>(fused_layout(&pp, 1).total_bytes) <= budget;
		}
	if (!fits)
		return false;

	// host blob: h_taps | h_left | records | ranges | win_col
	const int padded = 4 * steps, rec_bytes = stream_record_bytes(h_first, VS);
	size_t off = 0;
	p.off_h_taps = off;  off = align_up(off + static_cast<size_t>(dst_w) * HW * 4, 256);
	p.off_h_left = off;  off = align_up(off + static_cast<size_t>(dst_w) * sizeof(int), 256);
	p.off_v_dense = off; off = align_up(off + static_cast<size_t>(padded) * rec_bytes, 256);
	p.off_v_base = off;  off = align_up(off + ranges.size() * sizeof(int), 256);
	p.off_win_col = off; off = align_up(off + win_col.size() * sizeof(int), 256);
	p.blob.assign(off, 0);

	uint32_t *h_taps = reinterpret_cast<uint32_t *>(p.blob.data() + p.off_h_taps);
	int *h_left = reinterpret_cast<int *>(p.blob.data() + p.off_h_left);
	for (unsigned c = 0; c < dst_w; ++c) {
		for (unsigned k = 0; k < H.width; ++k)
			h_taps[static_cast<size_t>(c) * HW + k] = tap_bits(H, u16, c, k);
		h_left[c] = static_cast<int>(H.left[c]);
	}
	uint32_t *rec = reinterpret_cast<uint32_t *>(p.blob.data() + p.off_v_dense);
	const int rows = h_first ? J.ring_rows : J.in_rows;
	const int line_bytes = h_first ? kStripW * 4 : kStreamWindow * (u16 ? 2 : 4);
	for (int g = 0; g < padded; ++g) {
		const int base = gbase[std::min(g, groups - 1)];
		uint32_t *r = rec + static_cast<size_t>(g) * (rec_bytes / 4);
		for (int s = 0; s < VS; ++s)
			r[VS * kGroup + s] = static_cast<uint32_t>((base + s) % rows * line_bytes);
		for (int j = 0; j < kGroup && g < groups; ++j) {
			const unsigned i = static_cast<unsigned>(g * kGroup + j);
			if (i >= dst_h)
				break;
			const int d = static_cast<int>(V.left[i]) - base;
			for (unsigned k = 0; k < V.width; ++k)
				r[(d + k) * kGroup + j] = tap_bits(V, u16, i, k);
		}
	}
	std::memcpy(p.blob.data() + p.off_v_base, ranges.data(), ranges.size() * sizeof(int));
	std::memcpy(p.blob.data() + p.off_win_col, win_col.data(), win_col.size() * sizeof(int));

	J.src_w = static_cast<int>(src_w);
	J.src_h = static_cast<int>(src_h);
	J.dst_w = static_cast<int>(dst_w);
	J.dst_h = static_cast<int>(dst_h);
	J.strips = strips;
	J.strip_w = strip_w;
	J.pixel_max = u16 ? static_cast<float>((1UL << depth) - 1) : 0.0f;
	p.variant = ((J.h_first * 2 + (u16 ? 1 : 0)) * 4 + hw_i) * 4 + vs_i;
	return true;
}

void fused_segment(FusedPlan *const *plans, int n, int num_items_target)
{
	long strips = 0;
	for (int i = 0; i < n; ++i)
		strips += plans[i]->job.strips;
	const int want = static_cast<int>(std::max<long>(1, (num_items_target + strips - 1) / std::max<long>(1, strips)));
	for (int i = 0; i < n; ++i) {
		FusedJob &J = plans[i]->job;
		if (!plans[i]->mma || plans[i]->chain) {
			// the CUDA-core and chained kernels split their (strip, step)
			// units evenly over their CTAs: one unit per segment
			J.seg_groups = J.step_groups;
			J.segments = (J.groups + J.step_groups - 1) / J.step_groups;
			continue;
		}
		const int steps = (J.groups + J.step_groups - 1) / J.step_groups;
		const int segs = std::max(1, std::min(want, steps));
		const int steps_per_seg = (steps + segs - 1) / segs;
		J.seg_groups = steps_per_seg * J.step_groups;
		J.segments = (J.groups + J.seg_groups - 1) / J.seg_groups;
	}
}

int fused_items(const FusedJob &j)
{
	return j.strips * j.segments;
}

int fused_wave_items()
{
	int dev = 0, sms = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	return std::max(1, sms) * 4;
}

void fused_bind(FusedPlan &p, const void *device_blob)
{
	const char *b = static_cast<const char *>(device_blob);
	p.job.h_taps = reinterpret_cast<const float *>(b + p.off_h_taps);
	p.job.h_left = reinterpret_cast<const int *>(b + p.off_h_left);
	p.job.v_dense = reinterpret_cast<const float *>(b + p.off_v_dense);
	p.job.v_base = reinterpret_cast<const int *>(b + p.off_v_base);
	p.job.win_col = reinterpret_cast<const int *>(b + p.off_win_col);
}

namespace {

const void *kernel_ptr(int variant)
{
	if (variant >= 100)
		return mma_kernel_ptr(variant);
	const int vs = variant % 4, hw = variant / 4 % 4;
	switch (variant / 16) {
	case 0: return fused_kernel_ptr_v_f32(hw, vs);
	case 1: return fused_kernel_ptr_v_i16(hw, vs);
	case 2: return fused_kernel_ptr_h_f32(hw, vs);
	default: return fused_kernel_ptr_h_i16(hw, vs);
	}
}

} // namespace

SmemLayout fused_layout(const FusedPlan *const *plans, int n)
{
	if (n > 0 && plans[0]->mma)
		return mma_layout(plans, n);
	int in = 0, ring = 0;
	for (int i = 0; i < n; ++i) {
		in = std::max(in, plans[i]->job.in_rows);
		ring = std::max(ring, plans[i]->job.ring_rows);
	}
	const FusedJob &J = plans[0]->job;  // one variant: what follows is the same for every plan
	const bool h_first = J.h_first != 0;
	const int sample = J.kind == static_cast<int>(FusedKind::F32) ? 4 : 2;
	SmemLayout L{};
	int off = 0;
	L.in_off = off;
	off += in * kStreamWindow * sample;
	L.ring_off = off;
	off += h_first ? ring * kStripW * 4 : 2 * kBlockColumns * 16;
	L.vcoef_off = off;
	off += stream_record_buffers(h_first) * 4 * stream_record_bytes(h_first, J.vs);
	L.total_bytes = off;
	return L;
}

size_t fused_max_smem()
{
	return kSmemMax;
}

int fused_grid_size(int variant, size_t smem_bytes)
{
	int dev = 0, sms = 0, per_sm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	const void *k = kernel_ptr(variant);
	cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemMax));
	const int threads = variant >= 100 ? mma_threads() : kStreamThreads;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem_bytes) != cudaSuccess || per_sm < 1)
		per_sm = 1;
	return std::max(1, sms) * per_sm;
}

bool fused_takes_chunks(int variant)
{
	return variant >= 0 && variant < 100;
}

cudaError_t launch_fused(int variant, const FusedJob *jobs, int num_jobs, int total_tiles, const SmemLayout &smem_bytes,
                         int grid, const FewJobs &few, cudaStream_t stream, const WorkChunks &chunks)
{
	if (variant >= 100)
		return launch_mma(variant, jobs, num_jobs, total_tiles, smem_bytes, grid, few.job[0], stream);
	grid = std::max(1, std::min(grid, chunks.sched ? chunks.num : total_tiles));
	if (smem_bytes.total_bytes > static_cast<int>(kSmemMax))
		return cudaErrorInvalidValue;
	const void *k = kernel_ptr(variant);
	FewJobs by_value = few;
	SmemLayout layout = smem_bytes;
	WorkChunks c = chunks;
	void *args[] = { &jobs, &num_jobs, &total_tiles, &by_value, &layout, &c };
	return cudaLaunchKernel(k, dim3(grid), dim3(kStreamThreads), args, static_cast<size_t>(layout.total_bytes), stream);
}

void fused_set_io(FusedJob &j, const void *src, ptrdiff_t src_stride, void *dst, ptrdiff_t dst_stride)
{
	j.src = src;
	j.src_stride = src_stride;
	j.dst = dst;
	j.dst_stride = dst_stride;
	auto al = [](const void *p, ptrdiff_t s) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && s % 16 == 0; };
	j.vec_ok = al(src, src_stride) && al(dst, dst_stride) ? 1 : 0;
	auto divides = [](const void *p, ptrdiff_t s) {
		const uintptr_t a = reinterpret_cast<uintptr_t>(p) | static_cast<uintptr_t>(s);
		return a % 16 == 0 ? 16 : (a % 8 == 0 ? 8 : (a % 4 == 0 ? 4 : 2));
	};
	j.src_align = divides(src, src_stride);
	j.dst_align = divides(dst, dst_stride);
	j.tmap = nullptr;
}

} // namespace zg
