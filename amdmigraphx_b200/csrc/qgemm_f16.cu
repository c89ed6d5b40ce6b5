// quant_dot kernels: fp16 operands, tiles of one CTA.
#include "qgemm_kernel.cuh"

namespace mgx {

int qgemm_f16_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream)
{
    switch(bn)
    {
    case 256: return dispatch_out<256, false, true, false>(d, o, qo, stream);
    case 128: return dispatch_out<128, false, true, false>(d, o, qo, stream);
    default: return dispatch_out<64, false, true, false>(d, o, qo, stream);
    }
}

int qgemm_f16_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
