"""Plans of the chained tensor-core kernel (chain.cu), on the CPU: a driver
links the planner and prints what a plan chose."""
from __future__ import annotations

import math
import os
import shutil
import subprocess

import pytest

from test_streaming_plan import CSRC, CUDA, FILTERS

DRIVER = r"""
#include "chain_kernel.cuh"
#include "fused.h"
#include <cstdio>

using namespace zg;

// lines of stdin: kind a b src_w src_h dst_w dst_h
int main()
{
	int kind, sw, sh, dw, dh;
	double a, b;
	while (std::scanf("%d %lf %lf %d %d %d %d", &kind, &a, &b, &sw, &sh, &dw, &dh) == 7) {
		const Kernel f(kind, a, b);
		bool order[2];
		if (plan_pass_order(sw, sh, dw, dh, 0.0, 0.0, sw, sh, order) != 2) {
			std::printf("0 0 0 0 0 0 0 0\n");
			continue;
		}
		const FilterTable H = compute_filter(f, sw, dw, 0.0, sw), V = compute_filter(f, sh, dh, 0.0, sh);
		FusedPlan p;
		SmemLayout L;
		const FusedPlan *pp = &p;
		if (!plan_chain(order[0] ? H : V, order[0] ? V : H, order[0], 10, sw, sh, dw, dh, &p) ||
		    !chain_tma_layout(&pp, 1, &L)) {
			std::printf("0 0 0 0 0 0 0 0\n");
			continue;
		}
		std::printf("%d %d %d %d %d %d %d %d\n", p.variant, p.job.vs, p.job.hw, p.max_pxa, p.depth, p.job.in_rows,
		            p.job.groups, p.job.strip_w);
	}
	return 0;
}
"""


@pytest.fixture(scope="module")
def plan(lib, tmp_path_factory):
    from zimg_gb300 import build as zbuild
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) or not CUDA:
        pytest.skip("the CUDA toolkit is not available")
    d = tmp_path_factory.mktemp("chain")
    drv = d / "driver.cu"
    drv.write_text(DRIVER)
    exe = d / "plan"
    objs = [os.path.join(zbuild.OBJ_DIR, s + ".o") for s in zbuild.SOURCES]
    subprocess.run([nvcc, "-std=c++17", "-O1", *zbuild.ARCH, "-I", CSRC, "--expt-relaxed-constexpr", str(drv), *objs,
                    "--cudart", "shared", "-Xlinker", "-rpath=" + os.path.join(CUDA, "lib64"), "-o", str(exe)],
                   check=True, capture_output=True)

    def run(jobs):
        text = "".join(" ".join(str(v) for v in j) + "\n" for j in jobs)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
        keys = ("variant", "kv", "kh", "window", "depth", "lines", "groups", "strip_w")
        return [dict(zip(keys, map(int, line.split()))) for line in out.splitlines()]
    return run


def jobs_of_ratios():
    for kind, a, b in FILTERS:
        for sw, sh in ((1920, 1080), (640, 360), (768, 576), (331, 247)):
            for ratio in (0.25, 0.4, 0.5, 0.55, 0.66, 0.75, 0.86, 0.95, 1.2, 1.5, 1.9, 2.0, 2.1, 2.5, 3.0):
                yield kind, a, b, sw, sh, max(16, round(sw / ratio)), max(16, round(sh / ratio))
        for sizes in ((1541, 2164, 748, 1051), (1897, 2207, 944, 1098), (670, 863, 327, 421), (768, 576, 368, 280),
                      (986, 2196, 483, 754)):  # windows of just 248 samples
            yield kind, a, b, *sizes


def test_prefetch_depth_fits_unshrunk(plan):
    """The depth of the pipeline is what two CTAs' shared memory holds of its
    lines, stages, staged tiles (28 at most) and bases as they are, or one."""
    n = 0
    for job, p in zip(jobs_of_ratios(), plan(jobs_of_ratios())):
        if not p["variant"] or p["depth"] == 1:
            continue
        n += 1
        pitch = (p["window"] + 15) // 16 * 16 + 8
        tiles = p["strip_w"] // 16
        held = p["lines"] * pitch * 2 + (p["depth"] + 2) * p["kv"] * 1024 + tiles * 800 + p["groups"] * 4
        assert held <= 110 * 1024, (job, p, held)
    assert n > 100


def test_small_windows_keep_seven_warps_busy(plan):
    """Windows of 16 lines and 16 columns: strips of seven warps' tiles, four a
    warp where the strip's lines fit one copy, else two."""
    n = {2: 0, 4: 0}
    for job, p in zip(jobs_of_ratios(), plan(jobs_of_ratios())):
        if not p["variant"] or (p["kv"], p["kh"]) != (1, 1):
            continue
        tiles = p["strip_w"] / (7 * 16)
        assert tiles in (2, 4), (job, p)
        n[int(tiles)] += 1
    assert min(n.values()) > 20
