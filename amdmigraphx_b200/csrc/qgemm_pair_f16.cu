// quant_dot kernels: fp16 operands, tiles of two CTAs.
#include "qgemm_kernel.cuh"

namespace mgx {

int qgemm_pair_f16_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream)
{
    switch(bn)
    {
    case 256: return dispatch_out<256, false, true, true>(d, o, qo, stream);
    case 224: return dispatch_out<224, false, true, true>(d, o, qo, stream);
    case 192: return dispatch_out<192, false, true, true>(d, o, qo, stream);
    default: return dispatch_out<128, false, true, true>(d, o, qo, stream);
    }
}

int qgemm_pair_f16_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
