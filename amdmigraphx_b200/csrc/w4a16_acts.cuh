// Activations of an int4 decode linear as int8 planes: the pre-kernel of w4a16_tc.cu, its launch and the tensor map
// of its result.
#pragma once
#include "common.cuh"
#include "ptx.cuh"
#include <cuda_fp16.h>

namespace mgx {

// ------------------------------------------------------------------ activation pre-kernel
// grid = MB rows (padded) x chunks of 2048 k, 256 threads; a thread owns 8 consecutive k.  (With one
// block of 1024 threads per row a row of 11008 took two trips, each a load from L2: 5.0 us in a decode
// step against 2.7 for 4096.)
// Every activation becomes q = round(a / sa) = 128 h + l.  Two layouts of the int8 rows the
// tensor core multiplies with the weights (K bytes per row, 128 per group):
//   RAW = false (2 rows per activation row m): row 2 m = h, row 2 m + 1 = l; inside every 8 k the
//         evens first, then the odds (the order of the nibbles unpacked to bytes);
//   RAW = true  (4 rows per m), for a weight operand whose first 64 bytes of a group are the LOW
//         nibbles L_j = q[2j] and whose last 64 bytes are the packed bytes B_j = 16 q[2j+1] + L_j
//         themselves: rows [e | 0] and [-o | o] for each of h and l, e_j = a[2j], o_j = a[2j+1], so
//         that  sum_j L_j e_j  and  sum_j (B_j - L_j) o_j = 16 sum_j q[2j+1] o_j  come out.
// Also written: sv (per-group sums of q), sa (per-group scales), zeroed tile counters.
template <int MB, bool RAW>
__global__ void __launch_bounds__(256)
    w4_prepare_acts_kernel(const __half* __restrict__ A, int64_t lda, int64_t M, int64_t K,
                           int8_t* __restrict__ aq, float* __restrict__ sa, int* __restrict__ sv,
                           int* __restrict__ counters, int ncounters)
{
    // The main kernel may start (and stream weights) right away; it waits for this grid's completion before it
    // touches anything written here.  Started as it may be before the kernel in front of this one is complete,
    // it relies on no kernel that writes packed weights letting its successor start early (ptx.cuh): 1.4 us a
    // linear, back to back, against letting it start after the wait.
    grid_launch_dependents();
    // this kernel itself may have been started before the previous kernel of the stream has
    // finished (which may still read the workspace, or be writing A)
    grid_dependency_wait();
    constexpr int RPM = RAW ? 4 : 2; // int8 rows per activation row
    const int m   = blockIdx.x;
    const int tid = threadIdx.x;
    int8_t* rows  = aq + static_cast<int64_t>(RPM * m) * K;
    const int64_t kb = static_cast<int64_t>(blockIdx.y) * 2048;
    for(int i = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + tid; i < ncounters; i += gridDim.x * gridDim.y * 256)
        counters[i] = 0;
    if(m >= M)
    {
        for(int r = 0; r < RPM; ++r)
            if(tid < 128 and kb + tid * 16 < K)
                *reinterpret_cast<uint4*>(rows + r * K + kb + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
        const int64_t g = kb / 128 + tid;
        if(tid < 16 and g < K / 128)
        {
            sv[g * MB + m] = 0;
            sa[g * MB + m] = 0.0f;
        }
        return;
    }
    const __half* row = A + m * lda;
    {
        // 16 consecutive threads hold one group of 128 k
        const int64_t k  = kb + tid * 8;
        const bool valid = k < K;
        const uint4 v    = valid ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0u, 0u, 0u, 0u);
        const __half* vh = reinterpret_cast<const __half*>(&v);
        float mx         = 0.0f;
#pragma unroll
        for(int e = 0; e < 8; ++e)
            mx = fmaxf(mx, fabsf(__half2float(vh[e])));
#pragma unroll
        for(int o = 8; o > 0; o >>= 1)
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        // 128 h + l spans [-16256, 16256] with h in [-127, 127], l in [-64, 63]
        const float scale = mx > 0.0f ? mx / 16256.0f : 1.0f;
        const float inv   = 1.0f / scale;
        int sum           = 0;
        // bytes of the evens (e = 0, 2, 4, 6) and of the odds, for h and for l
        uint32_t he = 0u, ho = 0u, le = 0u, lo = 0u, nho = 0u, nlo = 0u;
#pragma unroll
        for(int e = 0; e < 8; ++e)
        {
            int q = __float2int_rn(__half2float(vh[e]) * inv);
            q     = max(-16256, min(16256, q));
            const int h = (q + 64 + 128 * 256) / 128 - 256; // round(q / 128) for any sign
            const int l = q - 128 * h;
            sum += q;
            const int sh = 8 * (e >> 1);
            if(e & 1)
            {
                ho |= static_cast<uint32_t>(h & 0xFF) << sh;
                lo |= static_cast<uint32_t>(l & 0xFF) << sh;
                nho |= static_cast<uint32_t>(-h & 0xFF) << sh;
                nlo |= static_cast<uint32_t>(-l & 0xFF) << sh;
            }
            else
            {
                he |= static_cast<uint32_t>(h & 0xFF) << sh;
                le |= static_cast<uint32_t>(l & 0xFF) << sh;
            }
        }
        if(valid)
        {
            if constexpr(RAW)
            {
                // byte j = k / 2 of the group's low half, 64 + j of its high half
                const int64_t o = (k & ~int64_t{127}) + ((k & 127) >> 1);
                *reinterpret_cast<uint32_t*>(rows + o)              = he;
                *reinterpret_cast<uint32_t*>(rows + o + 64)         = 0u;
                *reinterpret_cast<uint32_t*>(rows + K + o)          = nho;
                *reinterpret_cast<uint32_t*>(rows + K + o + 64)     = ho;
                *reinterpret_cast<uint32_t*>(rows + 2 * K + o)      = le;
                *reinterpret_cast<uint32_t*>(rows + 2 * K + o + 64) = 0u;
                *reinterpret_cast<uint32_t*>(rows + 3 * K + o)      = nlo;
                *reinterpret_cast<uint32_t*>(rows + 3 * K + o + 64) = lo;
            }
            else
            {
                *reinterpret_cast<uint2*>(rows + k)     = make_uint2(he, ho);
                *reinterpret_cast<uint2*>(rows + K + k) = make_uint2(le, lo);
            }
        }
#pragma unroll
        for(int o = 8; o > 0; o >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if(valid and (tid & 15) == 0)
        {
            sv[(k >> 7) * MB + m] = sum;
            sa[(k >> 7) * MB + m] = scale;
        }
    }
}

namespace {

// [group][row][inner bytes] view of a row-major byte matrix whose rows are `groups` runs of
// `inner` bytes: one request brings `box_groups` runs of `box_rows` rows.
int encode_grouped(CUtensorMap* map, const void* base, uint32_t inner, uint64_t rows, uint64_t pitch,
                   uint64_t groups, uint32_t box_rows, uint32_t box_groups, CUtensorMapSwizzle swz)
{
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[3]    = {inner, rows, groups};
    cuuint64_t strides[2] = {pitch, inner};
    cuuint32_t box[3]     = {inner, box_rows, box_groups};
    cuuint32_t estr[3]    = {1u, 1u, 1u};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides,
                        box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MGX_OK : MGX_E_INVALID_ARG;
}

// mb: padded activation rows (4 and 8: four int8 rows each, 16: two); counters may be null (ncounters 0).
// Chained programmatically to the kernel before it.
int launch_prepare_acts(int mb, const __half* A, int64_t lda, int64_t M, int64_t K, int8_t* aq, float* sa, int* sv,
                        int* counters, int ncounters, cudaStream_t stream)
{
    const dim3 grid(static_cast<unsigned>(mb), static_cast<unsigned>(ceil_div(K, 2048)));
    auto* kernel = mb == 4 ? w4_prepare_acts_kernel<4, true>
                           : (mb == 8 ? w4_prepare_acts_kernel<8, true> : w4_prepare_acts_kernel<16, false>);
    return launch_dependent(kernel, grid, dim3(256), 0, stream, A, lda, M, K, aq, sa, sv, counters, ncounters);
}

} // namespace

} // namespace mgx
