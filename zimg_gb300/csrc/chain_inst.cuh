// One form of the chained kernel (chain_tma_kernel.cuh) in one translation
// unit: its instances by variant and its copies of the kernel's device
// variables, behind a table of functions.
#pragma once

#include "chain_tma_kernel.cuh"
#include "fused.h"

namespace zg {

namespace {

// The instances from code CODE on.
template <ChainForm F, int CODE = 0>
const void *form_ptr_from(int code)
{
	constexpr chain_detail::ChainVariant V = chain_detail::chain_variant_of(CODE);
	if constexpr (CODE < chain_detail::kEitherVariant) {
		if (code != CODE)
			return form_ptr_from<F, CODE + 1>(code);
	}
	return reinterpret_cast<const void *>(&chain_detail::chain_tma_kernel<V.h_first, V.kv, V.kh, V.tiles, F>);
}

template <ChainForm F>
const void *form_ptr(int variant)
{
	return form_ptr_from<F>(variant - 200);
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
