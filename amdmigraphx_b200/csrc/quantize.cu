// HBM-bound element-wise kernels of the quantized path: quantizelinear,
// dequantizelinear, unpack_int4 / pack_int4 and the 8-bit transpose used to make
// quant_dot's [K,N] operand K-contiguous.
//
// Arithmetic follows the MIGraphX operators exactly:
//   quantizelinear   src/include/migraphx/op/quantizelinear.hpp:71-108
//   dequantizelinear src/include/migraphx/op/dequantizelinear.hpp:60-82
//   unpack_int4      src/include/migraphx/op/unpack_int4.hpp:75-120
//   pack_int4        src/include/migraphx/op/pack_int4.hpp:79-123
#include "common.cuh"
#include "ptx.cuh"
#include <cuda_fp16.h>
#include <cuda_fp8.h>

namespace mgx {

// ------------------------------------------------------------------ helpers
template <class T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v)
{
    return v;
}
template <>
__device__ __forceinline__ float to_f32<__half>(__half v)
{
    return __half2float(v);
}

// x / s evaluated in the input type (the reference divides `input[i] / scales[i]`
// in the tensor's own type for integer targets).  migraphx::half divides in fp32 and
// converts the quotient back by shifting the mantissa, i.e. rounding toward zero
// (src/include/migraphx/generic_float.hpp:180-230, 321-329).
template <class T>
__device__ __forceinline__ float div_in_type(float x, float s);
template <>
__device__ __forceinline__ float div_in_type<float>(float x, float s)
{
    return __fdiv_rn(x, s);
}
template <>
__device__ __forceinline__ float div_in_type<__half>(float x, float s)
{
    return __half2float(__float2half_rz(__fdiv_rn(x, s)));
}

struct q_i8
{
    using type = int8_t;
    static __device__ __forceinline__ float zp(int8_t z) { return static_cast<float>(z); }
    template <class In>
    static __device__ __forceinline__ int8_t quant(float x, float s, float z)
    {
        // nearbyint (round-half-even) of the quotient, + zero point, saturate.
        // fminf/fmaxf drop a NaN operand, as std::min/std::max do in the reference's
        // argument order, so NaN saturates to the maximum.
        float q = rintf(div_in_type<In>(x, s)) + z;
        q       = fmaxf(-128.0f, fminf(127.0f, q));
        return static_cast<int8_t>(static_cast<int>(q));
    }
};
struct q_u8
{
    using type = uint8_t;
    static __device__ __forceinline__ float zp(uint8_t z) { return static_cast<float>(z); }
    template <class In>
    static __device__ __forceinline__ uint8_t quant(float x, float s, float z)
    {
        float q = rintf(div_in_type<In>(x, s)) + z;
        q       = fmaxf(0.0f, fminf(255.0f, q));
        return static_cast<uint8_t>(static_cast<int>(q));
    }
};
struct q_fp8
{
    using type = uint8_t; // e4m3fn bit pattern
    static __device__ __forceinline__ float zp(uint8_t z)
    {
        return __half2float(__half(__nv_cvt_fp8_to_halfraw(z, __NV_E4M3)));
    }
    template <class In>
    static __device__ __forceinline__ uint8_t quant(float x, float s, float z)
    {
        // no nearbyint for floating targets: x/s + zp in double, clamp to +-448, then
        // one round-to-nearest-even cast.  fp32 division of fp32 operands equals the
        // double quotient rounded to fp32; the sum with a non-zero zp is done in double.
        float q;
        if(z == 0.0f)
            q = __fdiv_rn(x, s);
        else
            q = static_cast<float>(static_cast<double>(x) / static_cast<double>(s) +
                                   static_cast<double>(z));
        q = fmaxf(-448.0f, fminf(448.0f, q));
        return static_cast<uint8_t>(__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3));
    }
};

struct view2
{
    int64_t s0, s1;
};

// One work item = 16 bytes of one input row (4 fp32 or 8 fp16 columns) -> 4 or 8 output
// bytes.  Index arithmetic is done in IdxT (32-bit whenever the tensor allows it: a 64-bit
// division per item would make the kernel ALU-bound).  UNIFORM: scale and zero point are
// per-tensor (all strides 0) and are read once per thread.
template <class In, class Q, class IdxT, bool UNIFORM>
__global__ void __launch_bounds__(256)
    quantize_vec_kernel(const In* __restrict__ x, int64_t ldx, const In* __restrict__ scale,
                        view2 ss, const typename Q::type* __restrict__ zp, view2 zs,
                        typename Q::type* __restrict__ y, int64_t ldy, IdxT rows, IdxT colsv)
{
    constexpr int VEC = 16 / sizeof(In);
    const IdxT total  = rows * colsv;
    const IdxT stride = static_cast<IdxT>(gridDim.x) * blockDim.x;
    float s0 = 1.0f, z0 = 0.0f;
    if(UNIFORM)
    {
        s0 = to_f32<In>(scale[0]);
        z0 = zp == nullptr ? 0.0f : Q::zp(zp[0]);
    }
    for(IdxT i = static_cast<IdxT>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride)
    {
        const IdxT r = i / colsv;
        const IdxT c = (i - r * colsv) * VEC;
        const uint4 raw = *reinterpret_cast<const uint4*>(x + static_cast<int64_t>(r) * ldx + c);
        float xv[VEC];
        if constexpr(std::is_same<In, float>::value)
        {
            xv[0] = __uint_as_float(raw.x), xv[1] = __uint_as_float(raw.y);
            xv[2] = __uint_as_float(raw.z), xv[3] = __uint_as_float(raw.w);
        }
        else
        {
            const __half* vh = reinterpret_cast<const __half*>(&raw);
#pragma unroll
            for(int j = 0; j < VEC; ++j)
                xv[j] = __half2float(vh[j]);
        }
        uint32_t packed[VEC / 4];
#pragma unroll
        for(int w = 0; w < VEC / 4; ++w)
            packed[w] = 0;
#pragma unroll
        for(int j = 0; j < VEC; ++j)
        {
            float sv = s0, zv = z0;
            if(not UNIFORM)
            {
                sv = to_f32<In>(scale[static_cast<int64_t>(r) * ss.s0 + (c + j) * ss.s1]);
                zv = zp == nullptr ? 0.0f
                                   : Q::zp(zp[static_cast<int64_t>(r) * zs.s0 + (c + j) * zs.s1]);
            }
            const uint32_t q = static_cast<uint8_t>(Q::template quant<In>(xv[j], sv, zv));
            packed[j / 4] |= q << (8 * (j % 4));
        }
        typename Q::type* dst = y + static_cast<int64_t>(r) * ldy + c;
        if constexpr(VEC == 4)
            *reinterpret_cast<uint32_t*>(dst) = packed[0];
        else
            *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
    }
}

// Per-tensor quantizelinear to int8 / fp8: bound by HBM, so the work per element is kept small and U
// 16-byte loads per thread are in flight before the first is used (8192 x 8192 to int8 / fp8, one load
// at a time and two integer clamps per value before: fp32 65 -> 49 us = 6.9 TB/s, fp16 63 -> 39 us).
// Bit-identical to Q::quant:
//  * x / s: quotient from the correctly rounded reciprocal, corrected once with its remainder
//    (P. Markstein's theorem: correctly rounded; where the quotient is subnormal every result is 0);
//    an overflowed or not-a-number quotient is left as it is;
//  * int8, fp16 input: the quotient is cut to 10 mantissa bits (migraphx::half's truncating conversion);
//    saturated against the zero point's bounds, rounded half to even by adding 1.5 * 2^23, whose low
//    byte is the integer;
//  * fp8: saturated, one packed conversion for two values.
// FLAT: rows follow each other without gaps, an item's place needs no division.
template <class In, class Q, int U, bool FLAT>
__global__ void __launch_bounds__(256)
    quantize_uniform_kernel(const In* __restrict__ x, int64_t ldx, const In* __restrict__ scale,
                            const typename Q::type* __restrict__ zp, typename Q::type* __restrict__ y, int64_t ldy,
                            uint32_t total, uint32_t colsv)
{
    constexpr int VEC = 16 / sizeof(In);
    constexpr bool I8 = std::is_same<Q, q_i8>::value;
    if constexpr(not I8) // (packed weights are 8-bit integers: ptx.cuh)
        grid_launch_dependents();
    grid_dependency_wait();
    const float s    = to_f32<In>(scale[0]);
    const float rcp  = static_cast<float>(1.0 / static_cast<double>(s));
    const float z    = zp == nullptr ? 0.0f : Q::zp(zp[0]);
    const bool plain = s > 0.0f and isfinite(rcp) and (I8 or z == 0.0f);
    const float lo   = I8 ? -128.0f - z : -448.0f, hi = I8 ? 127.0f - z : 448.0f;
    const uint32_t z4 = (static_cast<uint32_t>(static_cast<int>(z)) & 0xFFu) * 0x01010101u; // int8: added to four results
    const uint32_t i0 = blockIdx.x * (256u * U) + threadIdx.x;
    uint4 raw[U];
    uint32_t row[U], col[U];
#pragma unroll
    for(int u = 0; u < U; ++u)
    {
        const uint32_t i = i0 + 256u * u;
        row[u]           = FLAT ? 0u : i / colsv;
        col[u]           = FLAT ? i : i - row[u] * colsv;
        if(i < total)
            raw[u] = *reinterpret_cast<const uint4*>(x + row[u] * ldx + static_cast<int64_t>(col[u]) * VEC);
    }
#pragma unroll
    for(int u = 0; u < U; ++u)
    {
        if(i0 + 256u * u >= total)
            break;
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        uint32_t packed[VEC / 4];
#pragma unroll
        for(int p = 0; p < VEC / 4; ++p)
        {
            float q[4];
#pragma unroll
            for(int j = 0; j < 4; ++j)
            {
                if constexpr(VEC == 4)
                    q[j] = __uint_as_float(w[j]);
                else
                {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[2 * p + j / 2]));
                    q[j]           = j & 1 ? f.y : f.x;
                }
            }
            if(plain)
            {
#pragma unroll
                for(int j = 0; j < 4; ++j)
                {
                    const float q0 = __fmul_rn(q[j], rcp);
                    float q1       = __fmaf_rn(__fmaf_rn(-s, q0, q[j]), rcp, q0);
                    if constexpr(not I8)
                        q1 = copysignf(q1, q0); // the correction makes +0 of -0; fp8 keeps the sign, as the other kernels here do
                    q[j] = fabsf(q0) <= 1e30f ? q1 : q0;
                    if constexpr(I8 and VEC == 8)
                        q[j] = __uint_as_float(__float_as_uint(q[j]) & 0xFFFFE000u);
                    q[j] = fmaxf(lo, fminf(hi, q[j]));
                }
                if constexpr(I8)
                {
                    uint32_t b[4];
#pragma unroll
                    for(int j = 0; j < 4; ++j)
                        b[j] = __float_as_uint(__fadd_rn(q[j], 12582912.0f));
                    packed[p] = __vadd4(
                        __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410), z4);
                }
                else
                {
                    const uint32_t b01 = __nv_cvt_float2_to_fp8x2(make_float2(q[0], q[1]), __NV_SATFINITE, __NV_E4M3);
                    const uint32_t b23 = __nv_cvt_float2_to_fp8x2(make_float2(q[2], q[3]), __NV_SATFINITE, __NV_E4M3);
                    packed[p]          = b01 | (b23 << 16);
                }
            }
            else
            {
                packed[p] = 0;
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    packed[p] |= static_cast<uint32_t>(static_cast<uint8_t>(Q::template quant<In>(q[j], s, z))) << (8 * j);
            }
        }
        typename Q::type* dst = y + row[u] * ldy + static_cast<int64_t>(col[u]) * VEC;
        if constexpr(VEC == 4)
            *reinterpret_cast<uint32_t*>(dst) = packed[0];
        else
            *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
    }
}

template <class In, class Q>
__global__ void __launch_bounds__(256)
    quantize_scalar_kernel(const In* __restrict__ x, int64_t ldx, const In* __restrict__ scale,
                           view2 ss, const typename Q::type* __restrict__ zp, view2 zs,
                           typename Q::type* __restrict__ y, int64_t ldy, int64_t rows,
                           int64_t cols)
{
    const int64_t total = rows * cols;
    for(int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
        i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const int64_t r = i / cols;
        const int64_t c = i - r * cols;
        const float s   = to_f32<In>(scale[r * ss.s0 + c * ss.s1]);
        const float z   = zp == nullptr ? 0.0f : Q::zp(zp[r * zs.s0 + c * zs.s1]);
        y[r * ldy + c]  = Q::template quant<In>(to_f32<In>(x[r * ldx + c]), s, z);
    }
}

static int grid_for(int64_t work_items, int threads)
{
    const int64_t blocks = ceil_div(work_items, threads);
    const int64_t cap    = static_cast<int64_t>(device_sm_count()) * 8;
    return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

template <class In, class Q>
static int launch_quantize(const void* x, int64_t ldx, const void* scale, view2 ss, const void* zp,
                           view2 zs, void* y, int64_t ldy, int64_t rows, int64_t cols,
                           cudaStream_t stream)
{
    using Out         = typename Q::type;
    constexpr int VEC = 16 / sizeof(In);
    const bool vec    = cols % VEC == 0 and ldx % VEC == 0 and ldy % VEC == 0 and
                     (reinterpret_cast<uintptr_t>(x) % 16) == 0 and
                     (reinterpret_cast<uintptr_t>(y) % VEC) == 0;
    if(vec)
    {
        const int64_t n    = rows * (cols / VEC);
        const bool uniform = ss.s0 == 0 and ss.s1 == 0 and (zp == nullptr or (zs.s0 == 0 and zs.s1 == 0));
        const bool small   = n < (int64_t{1} << 31) and rows * ldx < (int64_t{1} << 31);
        const int grid     = grid_for(n, 256);
#define MGX_LAUNCH_QV(IDX, UNI)                                                                  \
    quantize_vec_kernel<In, Q, IDX, UNI><<<grid, 256, 0, stream>>>(                              \
        static_cast<const In*>(x), ldx, static_cast<const In*>(scale), ss,                       \
        static_cast<const Out*>(zp), zs, static_cast<Out*>(y), ldy, static_cast<IDX>(rows),      \
        static_cast<IDX>(cols / VEC))
        if constexpr(not std::is_same<Q, q_u8>::value)
        {
            if(small and uniform)
            {
                // four loads per thread where that still gives every SM two blocks
                const bool flat   = ldx == cols and ldy == cols;
                const bool deep   = n >= int64_t{2048} * device_sm_count();
                auto* kernel      = deep ? (flat ? quantize_uniform_kernel<In, Q, 4, true> : quantize_uniform_kernel<In, Q, 4, false>)
                                         : (flat ? quantize_uniform_kernel<In, Q, 1, true> : quantize_uniform_kernel<In, Q, 1, false>);
                const auto blocks = static_cast<unsigned>(ceil_div(n, deep ? 1024 : 256));
                return launch_dependent(kernel, dim3(blocks), dim3(256), 0, stream, static_cast<const In*>(x), ldx,
                                        static_cast<const In*>(scale), static_cast<const Out*>(zp), static_cast<Out*>(y), ldy,
                                        static_cast<uint32_t>(n), static_cast<uint32_t>(cols / VEC));
            }
        }
        if(small and uniform)
            MGX_LAUNCH_QV(uint32_t, true);
        else if(small)
            MGX_LAUNCH_QV(uint32_t, false);
        else if(uniform)
            MGX_LAUNCH_QV(int64_t, true);
        else
            MGX_LAUNCH_QV(int64_t, false);
#undef MGX_LAUNCH_QV
    }
    else
    {
        const int64_t n = rows * cols;
        quantize_scalar_kernel<In, Q><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const In*>(x), ldx, static_cast<const In*>(scale), ss,
            static_cast<const Out*>(zp), zs, static_cast<Out*>(y), ldy, rows, cols);
    }
    return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------ dequantize
template <class X>
__device__ __forceinline__ double x_to_double(X v)
{
    return static_cast<double>(v);
}
struct fp8_bits
{
    uint8_t b;
};
template <>
__device__ __forceinline__ double x_to_double<fp8_bits>(fp8_bits v)
{
    return static_cast<double>(__half2float(__half(__nv_cvt_fp8_to_halfraw(v.b, __NV_E4M3))));
}

template <class X, class S>
__global__ void __launch_bounds__(256)
    dequantize_kernel(const X* __restrict__ x, int64_t ldx, const S* __restrict__ scale, view2 ss,
                      const X* __restrict__ zp, view2 zs, S* __restrict__ y, int64_t ldy,
                      int64_t rows, int64_t cols)
{
    const int64_t total = rows * cols;
    for(int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
        i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const int64_t r = i / cols;
        const int64_t c = i - r * cols;
        const double xv = x_to_double<X>(x[r * ldx + c]);
        const double zv = zp == nullptr ? 0.0 : x_to_double<X>(zp[r * zs.s0 + c * zs.s1]);
        const double sv = static_cast<double>(to_f32<S>(scale[r * ss.s0 + c * ss.s1]));
        const double d  = (xv - zv) * sv;
        if constexpr(std::is_same<S, float>::value)
            y[r * ldy + c] = static_cast<float>(d);
        else
            // double -> float (nearest) -> half (toward zero), as migraphx::half converts
            y[r * ldy + c] = __float2half_rz(static_cast<float>(d));
    }
}

template <class X>
static int launch_dequantize(const void* x, int64_t ldx, const void* scale, int scale_type,
                             view2 ss, const void* zp, view2 zs, void* y, int64_t ldy,
                             int64_t rows, int64_t cols, cudaStream_t stream)
{
    const int64_t n = rows * cols;
    if(scale_type == MGX_F32)
        dequantize_kernel<X, float><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const X*>(x), ldx, static_cast<const float*>(scale), ss,
            static_cast<const X*>(zp), zs, static_cast<float*>(y), ldy, rows, cols);
    else if(scale_type == MGX_F16)
        dequantize_kernel<X, __half><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const X*>(x), ldx, static_cast<const __half*>(scale), ss,
            static_cast<const X*>(zp), zs, static_cast<__half*>(y), ldy, rows, cols);
    else
        return MGX_E_UNSUPPORTED;
    return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------ int4 pack/unpack
template <bool SIGNED>
__global__ void __launch_bounds__(256)
    unpack_int4_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int64_t n)
{
    for(int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
        i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const uint8_t b = in[i];
        uint8_t lo = b & 0xF, hi = b >> 4;
        if(SIGNED)
        {
            lo = static_cast<uint8_t>(static_cast<int8_t>(b << 4) >> 4);
            hi = static_cast<uint8_t>(static_cast<int8_t>(b) >> 4);
        }
        *reinterpret_cast<uchar2*>(out + 2 * i) = make_uchar2(lo, hi);
    }
}

template <bool SIGNED>
__global__ void __launch_bounds__(256)
    pack_int4_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int64_t n)
{
    for(int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
        i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    {
        const uchar2 v = *reinterpret_cast<const uchar2*>(in + 2 * i);
        uint8_t a, b;
        if(SIGNED)
        {
            const int x0 = max(-8, min(7, static_cast<int>(static_cast<int8_t>(v.x))));
            const int x1 = max(-8, min(7, static_cast<int>(static_cast<int8_t>(v.y))));
            a = static_cast<uint8_t>(x0), b = static_cast<uint8_t>(x1);
        }
        else
        {
            a = min(v.x, static_cast<uint8_t>(15));
            b = min(v.y, static_cast<uint8_t>(15));
        }
        out[i] = static_cast<uint8_t>((b << 4) | (a & 0xF));
    }
}

// ------------------------------------------------------------ 8-bit transpose
// 64 x 64 byte tile through shared memory; both the global reads (rows of src)
// and the global writes (rows of dst) are 4-byte per thread, 64 B per 16 lanes.
__global__ void __launch_bounds__(256)
    transpose_8bit_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t rows,
                          int64_t cols, int64_t ld_dst)
{
    __shared__ uint8_t tile[64][64 + 4];
    const int64_t b  = blockIdx.z;
    const uint8_t* s = src + b * rows * cols;
    uint8_t* d       = dst + b * cols * ld_dst;
    const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 64;
    const int64_t c0 = static_cast<int64_t>(blockIdx.x) * 64;
    const int tx     = threadIdx.x & 15; // 16 threads x 4 bytes = 64 columns
    const int ty     = threadIdx.x >> 4; // 16 row slots
    const bool fast_in = (cols % 4 == 0) and ((reinterpret_cast<uintptr_t>(s) & 3u) == 0);
#pragma unroll
    for(int i = 0; i < 4; ++i)
    {
        const int rr    = ty + i * 16;
        const int64_t r = r0 + rr;
        const int64_t c = c0 + tx * 4;
        uint32_t v      = 0;
        if(r < rows)
        {
            if(fast_in and c + 4 <= cols)
                v = *reinterpret_cast<const uint32_t*>(s + r * cols + c);
            else
                for(int j = 0; j < 4; ++j)
                    if(c + j < cols)
                        v |= static_cast<uint32_t>(s[r * cols + c + j]) << (8 * j);
        }
#pragma unroll
        for(int j = 0; j < 4; ++j)
            tile[rr][tx * 4 + j] = static_cast<uint8_t>(v >> (8 * j));
    }
    __syncthreads();
    const bool fast_out = (ld_dst % 4 == 0) and ((reinterpret_cast<uintptr_t>(d) & 3u) == 0);
#pragma unroll
    for(int i = 0; i < 4; ++i)
    {
        const int cc    = ty + i * 16; // column of src = row of dst
        const int64_t c = c0 + cc;
        const int64_t r = r0 + tx * 4;
        if(c >= cols)
            continue;
        uint32_t v = 0;
#pragma unroll
        for(int j = 0; j < 4; ++j)
            v |= static_cast<uint32_t>(tile[tx * 4 + j][cc]) << (8 * j);
        if(fast_out and r + 4 <= rows)
            *reinterpret_cast<uint32_t*>(d + c * ld_dst + r) = v;
        else
            for(int j = 0; j < 4; ++j)
                if(r + j < rows)
                    d[c * ld_dst + r + j] = static_cast<uint8_t>(v >> (8 * j));
    }
}

int transpose_8bit_ld(const void* src, void* dst, int64_t rows, int64_t cols, int64_t batch,
                      int64_t ld_dst, cudaStream_t stream)
{
    if(src == nullptr or dst == nullptr or rows <= 0 or cols <= 0 or batch <= 0 or ld_dst < rows)
        return MGX_E_INVALID_ARG;
    const int64_t gx = ceil_div(cols, 64), gy = ceil_div(rows, 64);
    if(gy > 65535 or batch > 65535)
        return MGX_E_TOO_LARGE;
    dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(batch));
    transpose_8bit_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint8_t*>(src),
                                                    static_cast<uint8_t*>(dst), rows, cols, ld_dst);
    return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------ 16-bit transpose
// 32 x 32 tile of 16-bit elements through shared memory (the [K,N] operand of an fp16 dot
// re-laid out K-contiguous); rows of dst beyond `rows` up to ld_dst are not written.
__global__ void __launch_bounds__(256)
    transpose_16bit_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ dst, int64_t rows,
                           int64_t cols, int64_t ld_dst)
{
    __shared__ uint16_t tile[32][32 + 2];
    const int64_t b   = blockIdx.z;
    const uint16_t* s = src + b * rows * cols;
    uint16_t* d       = dst + b * cols * ld_dst;
    const int64_t r0  = static_cast<int64_t>(blockIdx.y) * 32;
    const int64_t c0  = static_cast<int64_t>(blockIdx.x) * 32;
    const int tx      = threadIdx.x & 31;
    const int ty      = threadIdx.x >> 5; // 8 row slots
#pragma unroll
    for(int i = 0; i < 4; ++i)
    {
        const int rr    = ty + i * 8;
        const int64_t r = r0 + rr, c = c0 + tx;
        tile[rr][tx]    = (r < rows and c < cols) ? s[r * cols + c] : uint16_t{0};
    }
    __syncthreads();
#pragma unroll
    for(int i = 0; i < 4; ++i)
    {
        const int cc    = ty + i * 8; // column of src = row of dst
        const int64_t c = c0 + cc, r = r0 + tx;
        if(c < cols and r < rows)
            d[c * ld_dst + r] = tile[tx][cc];
    }
}

// The same with 16-byte accesses: 64 x 64 elements a block, rows of 72 in shared memory so that the eight elements a
// thread gathers down a column lie in different banks from its neighbours'.  A prompt's values (32 x 512 x 128, 8 MB
// moved) 5.6 us an element at a time, 4.6 so.
// EARLY: launched programmatically, what follows may start early.  For rows as short as a head's (up to 128), the values
// of a prompt's attention: a layer of 512 tokens 268.8 us, launched plainly 272.2, of 1000 536 and 567 - though not for
// such dots directly behind one another (32 x 512 x 128 x 512 14.1 and 12.2 us).  For longer rows plainly: the GEMM behind
// it takes whole SMs, from blocks still to come (8 x 1024 x 1024 x 128 17.5 us, plainly 13.9, 32 x 512 x 512 x 128 17.6 and
// 15.4).
template <bool EARLY>
__global__ void __launch_bounds__(256)
    transpose_16bit_vec_kernel(const uint16_t* src, uint16_t* dst, int64_t rows, int64_t cols,
                               int64_t ld_dst)
{
    __shared__ __align__(16) uint16_t tile[64][72];
    if constexpr(EARLY)
        grid_dependency_wait();
    const uint16_t* s = src + blockIdx.z * rows * cols;
    uint16_t* d       = dst + blockIdx.z * cols * ld_dst;
    const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 64, c0 = static_cast<int64_t>(blockIdx.x) * 64;
#pragma unroll
    for(int i = 0; i < 2; ++i)
    {
        const int u = threadIdx.x + i * 256, rr = u >> 3, cc = (u & 7) * 8;
        if(r0 + rr < rows and c0 + cc < cols)
            *reinterpret_cast<uint4*>(&tile[rr][cc]) = *reinterpret_cast<const uint4*>(s + (r0 + rr) * cols + c0 + cc);
    }
    if constexpr(EARLY)
        grid_launch_dependents();
    __syncthreads();
#pragma unroll
    for(int i = 0; i < 2; ++i)
    {
        // column of src = row of dst; eight of its elements
        const int u = threadIdx.x + i * 256, cc = u >> 3, rr = (u & 7) * 8;
        if(c0 + cc >= cols or r0 + rr >= rows)
            continue;
        uint32_t w[4];
#pragma unroll
        for(int e = 0; e < 4; ++e)
            w[e] = tile[rr + 2 * e][cc] | static_cast<uint32_t>(tile[rr + 2 * e + 1][cc]) << 16;
        uint16_t* at = d + (c0 + cc) * ld_dst + r0 + rr;
        if(r0 + rr + 8 <= rows)
            *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
        else
            for(int e = 0; r0 + rr + e < rows; ++e)
                at[e] = static_cast<uint16_t>(w[e >> 1] >> (16 * (e & 1)));
    }
}

int transpose_16bit_ld(const void* src, void* dst, int64_t rows, int64_t cols, int64_t batch,
                       int64_t ld_dst, cudaStream_t stream)
{
    if(src == nullptr or dst == nullptr or rows <= 0 or cols <= 0 or batch <= 0 or ld_dst < rows)
        return MGX_E_INVALID_ARG;
    const int64_t gx = ceil_div(cols, 32), gy = ceil_div(rows, 32);
    if(gy > 65535 or batch > 65535)
        return MGX_E_TOO_LARGE;
    if(cols % 8 == 0 and ld_dst % 8 == 0 and (reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) % 16 == 0)
    {
        const dim3 vgrid(static_cast<unsigned>(ceil_div(cols, 64)), static_cast<unsigned>(ceil_div(rows, 64)), static_cast<unsigned>(batch));
        const auto* in = static_cast<const uint16_t*>(src);
        auto* out      = static_cast<uint16_t*>(dst);
        if(cols <= 128)
            return launch_dependent(transpose_16bit_vec_kernel<true>, vgrid, dim3(256), 0, stream, in, out, rows, cols, ld_dst);
        transpose_16bit_vec_kernel<false><<<vgrid, 256, 0, stream>>>(in, out, rows, cols, ld_dst);
        return static_cast<int>(cudaGetLastError());
    }
    dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(batch));
    transpose_16bit_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(src),
                                                     static_cast<uint16_t*>(dst), rows, cols, ld_dst);
    return static_cast<int>(cudaGetLastError());
}

} // namespace mgx

using namespace mgx;

extern "C" int mgx_cuda_quantizelinear(const void* x, int x_type, int64_t ldx, const void* scale,
                                       const int64_t scale_strides[2], const void* zp,
                                       const int64_t zp_strides[2], void* y, int y_type,
                                       int64_t ldy, int64_t rows, int64_t cols, void* stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if(rows < 0 or cols < 0)
        return MGX_E_INVALID_ARG;
    if(rows == 0 or cols == 0)
        return MGX_OK; // empty tensors may come with null pointers
    if(x == nullptr or scale == nullptr or y == nullptr or scale_strides == nullptr)
        return MGX_E_INVALID_ARG;
    if(ldx < cols or ldy < cols)
        return MGX_E_INVALID_ARG;
    if(zp != nullptr and zp_strides == nullptr)
        return MGX_E_INVALID_ARG;
    const view2 ss{scale_strides[0], scale_strides[1]};
    const view2 zs = zp != nullptr ? view2{zp_strides[0], zp_strides[1]} : view2{0, 0};
#define MGX_Q_CASE(IN, Q) return launch_quantize<IN, Q>(x, ldx, scale, ss, zp, zs, y, ldy, rows, cols, stream)
    if(x_type == MGX_F32)
    {
        if(y_type == MGX_I8)
            MGX_Q_CASE(float, q_i8);
        if(y_type == MGX_U8)
            MGX_Q_CASE(float, q_u8);
        if(y_type == MGX_FP8_E4M3FN)
            MGX_Q_CASE(float, q_fp8);
    }
    else if(x_type == MGX_F16)
    {
        if(y_type == MGX_I8)
            MGX_Q_CASE(__half, q_i8);
        if(y_type == MGX_U8)
            MGX_Q_CASE(__half, q_u8);
        if(y_type == MGX_FP8_E4M3FN)
            MGX_Q_CASE(__half, q_fp8);
    }
#undef MGX_Q_CASE
    return MGX_E_UNSUPPORTED;
}

extern "C" int mgx_cuda_dequantizelinear(const void* x, int x_type, int64_t ldx, const void* scale,
                                         int scale_type, const int64_t scale_strides[2],
                                         const void* zp, const int64_t zp_strides[2], void* y,
                                         int64_t ldy, int64_t rows, int64_t cols, void* stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if(rows < 0 or cols < 0)
        return MGX_E_INVALID_ARG;
    if(rows == 0 or cols == 0)
        return MGX_OK; // empty tensors may come with null pointers
    if(x == nullptr or scale == nullptr or y == nullptr or scale_strides == nullptr)
        return MGX_E_INVALID_ARG;
    if(ldx < cols or ldy < cols)
        return MGX_E_INVALID_ARG;
    if(zp != nullptr and zp_strides == nullptr)
        return MGX_E_INVALID_ARG;
    const view2 ss{scale_strides[0], scale_strides[1]};
    const view2 zs = zp != nullptr ? view2{zp_strides[0], zp_strides[1]} : view2{0, 0};
    switch(x_type)
    {
    case MGX_I8:
        return launch_dequantize<int8_t>(x, ldx, scale, scale_type, ss, zp, zs, y, ldy, rows, cols, stream);
    case MGX_U8:
        return launch_dequantize<uint8_t>(x, ldx, scale, scale_type, ss, zp, zs, y, ldy, rows, cols, stream);
    case MGX_I32:
        return launch_dequantize<int32_t>(x, ldx, scale, scale_type, ss, zp, zs, y, ldy, rows, cols, stream);
    case MGX_FP8_E4M3FN:
        return launch_dequantize<fp8_bits>(x, ldx, scale, scale_type, ss, zp, zs, y, ldy, rows, cols, stream);
    default: return MGX_E_UNSUPPORTED;
    }
}

extern "C" int mgx_cuda_unpack_int4(const void* in, void* out, int type, int64_t rows,
                                    int64_t packed_cols, void* stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if(in == nullptr or out == nullptr or rows < 0 or packed_cols < 0)
        return MGX_E_INVALID_ARG;
    const int64_t n = rows * packed_cols;
    if(n == 0)
        return MGX_OK;
    if(reinterpret_cast<uintptr_t>(out) & 1u)
        return MGX_E_ALIGNMENT;
    if(type == MGX_U8)
        unpack_int4_kernel<false><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out), n);
    else if(type == MGX_I8)
        unpack_int4_kernel<true><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out), n);
    else
        return MGX_E_UNSUPPORTED;
    return static_cast<int>(cudaGetLastError());
}

extern "C" int mgx_cuda_pack_int4(const void* in, void* out, int type, int64_t rows,
                                  int64_t packed_cols, void* stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if(in == nullptr or out == nullptr or rows < 0 or packed_cols < 0)
        return MGX_E_INVALID_ARG;
    const int64_t n = rows * packed_cols;
    if(n == 0)
        return MGX_OK;
    if(reinterpret_cast<uintptr_t>(in) & 1u)
        return MGX_E_ALIGNMENT;
    if(type == MGX_U8)
        pack_int4_kernel<false><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out), n);
    else if(type == MGX_I8)
        pack_int4_kernel<true><<<grid_for(n, 256), 256, 0, stream>>>(
            static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out), n);
    else
        return MGX_E_UNSUPPORTED;
    return static_cast<int>(cudaGetLastError());
}

extern "C" int mgx_cuda_transpose_8bit(const void* src, void* dst, int64_t rows, int64_t cols,
                                       int64_t batch, void* stream_)
{
    return transpose_8bit_ld(src, dst, rows, cols, batch, rows, static_cast<cudaStream_t>(stream_));
}
