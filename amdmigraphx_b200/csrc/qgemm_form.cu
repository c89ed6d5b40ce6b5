// One form of the quant_dot kernel: MGX_FORM of qgemm_host.cuh's list, given on the command line with its operand type
// (MGX_FORM_TYPE 0: int8, 1: fp8, 2: fp16), kind (MGX_FORM_KIND) and columns (MGX_FORM_BN).  The first launch of a kernel
// loads its translation unit: with a type's forms in one unit the first tile of one CTA cost 16 ms, of a pair 16 to 22, a
// shared K 12; so 2 to 3 ms each.
#include "qgemm_kernel.cuh"
#include <atomic>

#define MGX_FORM_CAT_(A, B) A##B
#define MGX_FORM_CAT(A, B) MGX_FORM_CAT_(A, B)

namespace mgx {

static std::atomic<bool> form_launched{false};

int MGX_FORM_CAT(qgemm_launch_, MGX_FORM)(const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, int split,
                                          cudaStream_t stream)
{
    form_launched.store(true, std::memory_order_relaxed);
    return dispatch_out<MGX_FORM_BN, MGX_FORM_TYPE == 0, MGX_FORM_TYPE == 2, MGX_FORM_KIND == QGEMM_PAIR,
                        MGX_FORM_KIND == QGEMM_SPLIT>(d, o, qo, stream, split);
}

int MGX_FORM_CAT(qgemm_status_, MGX_FORM)(unsigned int* out)
{
    *out = 0;
    return form_launched.load(std::memory_order_relaxed) ? read_and_clear_status(out) : 0;
}

} // namespace mgx
