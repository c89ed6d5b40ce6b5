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

// The forms of the kernel, each compiled by itself from qgemm_form.cu (build.py): the first launch of a form loads what
// its translation unit holds.  X(name, operand type, kind, bn): tiles of one CTA, 128 x bn, or of a pair of CTAs, 256 x
// bn, or tiles of 128 x bn whose K a cluster shares.
enum qgemm_kind { QGEMM_ONE, QGEMM_PAIR, QGEMM_SPLIT };
#define MGX_QGEMM_FORMS_OF(X, T, TYPE)                                                                        \
    X(T##_one_64, TYPE, QGEMM_ONE, 64)                                                                        \
    X(T##_one_128, TYPE, QGEMM_ONE, 128)                                                                      \
    X(T##_one_256, TYPE, QGEMM_ONE, 256)                                                                      \
    X(T##_pair_128, TYPE, QGEMM_PAIR, 128)                                                                    \
    X(T##_pair_192, TYPE, QGEMM_PAIR, 192)                                                                    \
    X(T##_pair_224, TYPE, QGEMM_PAIR, 224)                                                                    \
    X(T##_pair_256, TYPE, QGEMM_PAIR, 256)                                                                    \
    X(T##_split_64, TYPE, QGEMM_SPLIT, 64)
#define MGX_QGEMM_FORMS(X)                     \
    MGX_QGEMM_FORMS_OF(X, i8, MGX_I8)          \
    MGX_QGEMM_FORMS_OF(X, f8, MGX_FP8_E4M3FN)  \
    MGX_QGEMM_FORMS_OF(X, f16, MGX_F16)

// split: CTAs of a cluster that share a tile's K (2, 4 or 8; 1 for the other kinds).  The status word is read only where
// the form has been launched: reading it would load the form.
#define MGX_QGEMM_DECLARE(NAME, TYPE, KIND, BN)                                                                          \
    int qgemm_launch_##NAME(const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, int split,           \
                            cudaStream_t stream);                                                                        \
    int qgemm_status_##NAME(unsigned int* out);
MGX_QGEMM_FORMS(MGX_QGEMM_DECLARE)
#undef MGX_QGEMM_DECLARE

// clusters of `split` CTAs with a tile of 128 x 64 each that run at once
int qgemm_split_clusters(int split);

} // namespace mgx
