"""The CUDA-core streaming kernel's plans (fused.cu), on the CPU: a driver
links the planner and walks every plan's steps as the kernel loads them, with
the rings held line by line. No step brings two lines into one slot or replaces
a line that is still read, and every line of a step's windows is where the
step's records say."""
from __future__ import annotations

import math
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zimg_gb300", "csrc")
CUDA = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.isdir(d)), None)

DRIVER = r"""
#include "fused.h"
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace zg;

// nullptr, or what is wrong with the steps from `start` on
const char *walk(const FusedPlan &p, const std::vector<int> &gbase, int start)
{
	const FusedJob &J = p.job;
	const bool h_first = J.h_first != 0, u16 = J.kind != static_cast<int>(FusedKind::F32), early = J.depth != 0;
	const int *ranges = reinterpret_cast<const int *>(p.blob.data() + p.off_v_base);
	const int rec_words = stream_record_bytes(h_first, J.vs) / 4;
	const uint32_t *rec = reinterpret_cast<const uint32_t *>(p.blob.data() + p.off_v_dense);
	const int line_bytes = h_first ? kStripW * 4 : kStreamWindow * (u16 ? 2 : 4);
	std::vector<int> in(J.in_rows, -1), mid(std::max(1, J.ring_rows), -1);
	int next = ranges[2 * start], h_line = next;
	auto load = [&](int k) -> const char * {  // the lines of step k; early: step k - 1 is being read
		const int hi = ranges[2 * k + 1], a = next;
		if (hi - a > J.in_rows)
			return "a step brings in more lines than the ring holds";
		for (int y = a; y < hi; ++y) {
			int &slot = in[y % J.in_rows];
			if (early && k > start && slot >= ranges[2 * (k - 1)] && slot < ranges[2 * (k - 1) + 1])
				return "a line that is still read is replaced";
			slot = y;
		}
		next = std::max(next, hi);
		return nullptr;
	};
	if (const char *e = load(start))
		return e;
	for (int k = start; k < J.segments; ++k) {
		const bool more = k + 1 < J.segments;
		if (more && early)
			if (const char *e = load(k + 1))
				return e;
		if (h_first) {
			for (int y = h_line; y < ranges[2 * k + 1]; ++y) {
				if (in[y % J.in_rows] != y)
					return "a source line is not in its slot";
				mid[y % J.ring_rows] = y;
			}
			h_line = std::max(h_line, ranges[2 * k + 1]);
		}
		for (int g = 4 * k; g < 4 * k + 4; ++g)
			for (int s = 0; s < J.vs; ++s) {
				const int base = gbase[std::min<int>(g, static_cast<int>(gbase.size()) - 1)];
				const uint32_t at = rec[static_cast<size_t>(g) * rec_words + J.vs * group_rows(h_first) + s];
				if (at % line_bytes || (h_first ? mid : in).at(at / line_bytes) != base + s)
					return "a line of a window is not where its record says";
			}
		if (more && !early)
			if (const char *e = load(k + 1))
				return e;
	}
	return nullptr;
}

// lines of stdin: kind a b src_w src_h dst_w dst_h shift_h u16
int main()
{
	int kind, sw, sh, dw, dh, u16;
	double a, b, shift;
	while (std::scanf("%d %lf %lf %d %d %d %d %lf %d", &kind, &a, &b, &sw, &sh, &dw, &dh, &shift, &u16) == 9) {
		const Kernel f(kind, a, b);
		bool order[2];
		if (plan_pass_order(sw, sh, dw, dh, 0.0, shift, sw, sh, order) != 2) {
			std::printf("- none\n");
			continue;
		}
		const FilterTable H = compute_filter(f, sw, dw, 0.0, sw), V = compute_filter(f, sh, dh, shift, sh);
		const bool h_first = order[0];
		FusedPlan p;
		if (!plan_fused(h_first ? H : V, h_first ? V : H, h_first, u16 != 0, 16, sw, sh, dw, dh, &p)) {
			std::printf("- refused\n");
			continue;
		}
		const int rows = group_rows(h_first);
		std::vector<int> gbase((dh + rows - 1) / rows, sh);
		for (int i = 0; i < dh; ++i)
			gbase[i / rows] = std::min(gbase[i / rows], static_cast<int>(V.left[i]));
		const char *e = nullptr;
		for (int start : { 0, 1, p.job.segments / 3, p.job.segments - 1 })
			if (!e && start < p.job.segments)
				e = walk(p, gbase, start);
		std::printf("%s %s\n", h_first ? (p.job.depth ? "h-early" : "h-late") : (p.job.depth ? "v-early" : "v-late"),
		            e ? e : "ok");
	}
	return 0;
}
"""

FILTERS = [(0, math.nan, math.nan), (1, math.nan, math.nan), (2, 0.0, 0.5), (3, math.nan, math.nan),
           (4, math.nan, math.nan), (6, math.nan, math.nan), (5, 3.0, math.nan), (5, 4.0, math.nan)]
RATIOS = (0.1, 0.31, 0.7, 1.5, 2, 2.3, 3, 4, 5, 5.6, 6, 6.3, 7, 7.9, 9, 10.5, 12, 13.1, 16, 19, 21.7, 24)


@pytest.fixture(scope="module")
def walk(lib, tmp_path_factory):
    from zimg_gb300 import build as zbuild
    gxx = shutil.which("g++")
    if not gxx or not CUDA:
        pytest.skip("g++ or the CUDA headers not available")
    d = tmp_path_factory.mktemp("streaming")
    drv = d / "driver.cpp"
    drv.write_text(DRIVER)
    exe = d / "walk"
    objs = [os.path.join(zbuild.OBJ_DIR, s + ".o") for s in zbuild.SOURCES]
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(CUDA, "include"), str(drv), *objs,
                    "-L", os.path.join(CUDA, "lib64"), "-Wl,-rpath," + os.path.join(CUDA, "lib64"), "-lcudart",
                    "-lpthread", "-o", str(exe)], check=True, capture_output=True)

    def run(jobs):
        text = "".join(" ".join(str(v) for v in j) + "\n" for j in jobs)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        return [line.split(" ", 1) for line in out.splitlines()]
    return run


def test_no_step_overruns_its_rings(walk):
    jobs = []
    for kind, a, b in FILTERS:
        for ratio in RATIOS:
            for (sw, sh), across in (((640, 1201), ratio), ((64, 1201), 0.25), ((333, 877), 1.7), ((1600, 877), 3 * ratio)):
                for shift in (0.0, 0.3):
                    for u16 in (0, 1):
                        dh, dw = max(2, round(sh / ratio)), max(2, round(sw / across))
                        jobs.append((kind, a, b, sw, sh, dw, dh, shift, u16))
    got = walk(jobs)
    assert len(got) == len(jobs)
    modes = [m for m, _ in got]
    assert {"h-early", "h-late", "v-early", "v-late"} <= set(modes)
    bad = [(j, m, e) for j, (m, e) in zip(jobs, got) if e not in ("ok", "none", "refused")]
    assert not bad, (len(bad), bad[:5])


@pytest.mark.parametrize("kind", [0, 1, 2, 4, 5])
def test_planes_of_mostly_unused_lines_stay_separate(walk, kind):
    """A point filter far down large planes leaves most lines without a tap;
    no other filter does."""
    a = {2: 0.0, 5: 3.0}.get(kind, math.nan)
    b = 0.5 if kind == 2 else math.nan
    jobs, want = [], []
    for sw, sh, large in ((7680, 4320, True), (3840, 2160, False), (1920, 1080, False)):
        for ratio in (2, 3, 7, 9, 12):
            for u16 in (0, 1):
                jobs.append((kind, a, b, sw, sh, sw // ratio, sh // ratio, 0.0, u16))
                want.append(kind == 0 and large and ratio >= 7)
    for job, (mode, e), separate in zip(jobs, walk(jobs), want):
        if kind == 0 and (separate or job[3] < 7680 or job[5] > 3000):
            assert (e == "refused") == separate, (job, mode, e)
        elif kind:
            assert e == "ok" or job[3] // job[5] >= 3, (job, mode, e)  # refused for their taps, if at all
