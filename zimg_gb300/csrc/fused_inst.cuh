// One (H_FIRST, INT) instantiation unit of the fused streaming kernel: kernel
// pointers per (HW, VS) bucket and the launcher. Each fused_inst_*.cu expands
// ZG_FUSED_INSTANCE once; the units are separate to compile in parallel.
#pragma once

#include "fused_kernel.cuh"

#include <algorithm>

#define ZG_FUSED_INSTANCE(NAME, HF, INT)                                                                           \
	namespace zg {                                                                                                 \
	namespace {                                                                                                    \
	template <int HW, int VS>                                                                                      \
	const void *ptr_##NAME()                                                                                       \
	{                                                                                                              \
		return reinterpret_cast<const void *>(&fused_detail::fused_kernel<HF, INT, HW, VS>);                       \
	}                                                                                                              \
	template <int HW>                                                                                              \
	const void *ptr_vs_##NAME(int vs)                                                                              \
	{                                                                                                              \
		switch (vs) {                                                                                              \
		case 0: return ptr_##NAME<HW, 8>();                                                                        \
		case 1: return ptr_##NAME<HW, 12>();                                                                       \
		case 2: return ptr_##NAME<HW, 16>();                                                                       \
		default: return ptr_##NAME<HW, 24>();                                                                      \
		}                                                                                                          \
	}                                                                                                              \
	}                                                                                                              \
	const void *fused_kernel_ptr_##NAME(int hw, int vs)                                                            \
	{                                                                                                              \
		return hw == 0 ? ptr_vs_##NAME<6>(vs) : (hw == 1 ? ptr_vs_##NAME<8>(vs)                                    \
		                                                  : (hw == 2 ? ptr_vs_##NAME<12>(vs) : ptr_vs_##NAME<16>(vs))); \
	}                                                                                                              \
	}
