// The chained kernel without tensor copies, for planes of any alignment and
// order of lines.
#include "chain_inst.cuh"

namespace zg {

const ChainKernels kChainLines = { form_ptr<ChainForm::LINES>, form_set_fault, form_error };

} // namespace zg
