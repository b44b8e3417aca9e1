// The chained kernel with tensor copies, for destinations of any alignment
// and strips of any width.
#include "chain_inst.cuh"

namespace zg {

const ChainKernels kChainAnyDst = { form_ptr<ChainForm::ANY_DST>, form_set_fault, form_error };

} // namespace zg
