// quant_dot kernels: int8 operands, tiles of two CTAs.
#include "qgemm_kernel.cuh"

namespace mgx {

int qgemm_pair_i8_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream)
{
    switch(bn)
    {
    case 256: return dispatch_out<256, true, false, true>(d, o, qo, stream);
    case 224: return dispatch_out<224, true, false, true>(d, o, qo, stream);
    case 192: return dispatch_out<192, true, false, true>(d, o, qo, stream);
    default: return dispatch_out<128, true, false, true>(d, o, qo, stream);
    }
}

int qgemm_pair_i8_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
