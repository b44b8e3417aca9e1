// One form of the chained kernel (chain_tma_kernel.cuh) in one translation
// unit: its instances by variant and its copies of the kernel's device
// variables, behind a table of functions.
#pragma once

#include "chain_tma_kernel.cuh"
#include "fused.h"

namespace zg {

constexpr int kKVMax = 3;
constexpr int kKHMax = 4;

namespace {

template <ChainForm F, bool HF, int KV>
const void *form_ptr_kh(int kh)
{
	switch (kh) {
	case 1: return reinterpret_cast<const void *>(&chain_detail::chain_tma_kernel<HF, KV, 1, F>);
	case 2: return reinterpret_cast<const void *>(&chain_detail::chain_tma_kernel<HF, KV, 2, F>);
	case 3: return reinterpret_cast<const void *>(&chain_detail::chain_tma_kernel<HF, KV, 3, F>);
	default: return reinterpret_cast<const void *>(&chain_detail::chain_tma_kernel<HF, KV, 4, F>);
	}
}

template <ChainForm F, bool HF>
const void *form_ptr_kv(int kv, int kh)
{
	return kv == 1 ? form_ptr_kh<F, HF, 1>(kh) : (kv == 2 ? form_ptr_kh<F, HF, 2>(kh) : form_ptr_kh<F, HF, 3>(kh));
}

template <ChainForm F>
const void *form_ptr(int variant)
{
	const int v = variant - 200;
	const int per = kKVMax * kKHMax;
	const int kv = (v % per) / kKHMax + 1, kh = v % kKHMax + 1;
	return v >= per ? form_ptr_kv<F, true>(kv, kh) : form_ptr_kv<F, false>(kv, kh);
}

int form_set_fault(int drop_group, unsigned long long wait_ns)
{
	if (cudaMemcpyToSymbol(chain_detail::g_chain_drop_group, &drop_group, sizeof(drop_group)) != cudaSuccess ||
	    cudaMemcpyToSymbol(chain_detail::g_chain_wait_ns, &wait_ns, sizeof(wait_ns)) != cudaSuccess)
		return -1;
	return 0;
}

int form_error(bool reset)
{
	int v = 0;
	if (cudaMemcpyFromSymbol(&v, chain_detail::g_chain_pipeline_error, sizeof(v)) != cudaSuccess)
		return -1;
	if (reset && v) {
		const int zero = 0;
		cudaMemcpyToSymbol(chain_detail::g_chain_pipeline_error, &zero, sizeof(zero));
	}
	return v;
}

} // namespace

} // namespace zg
