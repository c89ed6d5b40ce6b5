// What the C ABI of quant_dot (qgemm.cu) hands to the translation units that hold its kernels.
#pragma once
#include "common.cuh"

namespace mgx {

// a quantizelinear of the result, fused into the epilogue
struct qout_args
{
    void* Dq        = nullptr;
    int64_t ldq     = 0;
    int64_t stride_q = 0;
    float scale     = 1.0f;
    float zp        = 0.0f;
    int fp8         = 0;
    int write_d     = 1;
    const void* lut = nullptr;
};

struct qgemm_operands
{
    const void* A;
    const void* B; // [N, K], K contiguous
    void* D;
    const float* scale;
    const float* bias;
    const void* residual;
    int64_t ldb, stride_b;
};

// tiles of one CTA, 128 x bn (bn = 64, 128, 256), and of a pair of CTAs, 256 x bn (bn = 128, 192, 224, 256)
int qgemm_i8_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_f8_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_f16_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_pair_i8_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_pair_f8_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_pair_f16_launch(int bn, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_i8_status(unsigned int* out);
int qgemm_f8_status(unsigned int* out);
int qgemm_f16_status(unsigned int* out);
int qgemm_pair_i8_status(unsigned int* out);
int qgemm_pair_f8_status(unsigned int* out);
int qgemm_pair_f16_status(unsigned int* out);

// tiles of 128 x 64 whose K is shared by the split (2, 4 or 8) CTAs of a cluster, and how many such clusters run at once
int qgemm_split_launch(int split, const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream);
int qgemm_split_clusters(int split);
int qgemm_split_status(unsigned int* out);

} // namespace mgx
