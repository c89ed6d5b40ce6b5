// quant_dot for sm_100a: int8 x int8 -> int32 and fp8(e4m3fn) x fp8 -> fp32 as a
// persistent, warp-specialised, TMA-fed tcgen05 GEMM with the accumulator in
// tensor memory and dequantizelinear / bias / activation / residual fused into
// the epilogue.
//
// Arithmetic contract (MIGraphX `ref` target): src/targets/ref/lowering.cpp:205-249
// -> gemm_naive (src/gemm.cpp:43-63): int8 products summed exactly, stored as
// int32; fp8 products summed in (at least) fp32, stored as fp32.  The fused
// epilogue reproduces dequantizelinear (src/include/migraphx/op/dequantizelinear.hpp:74-77:
// double(x) * scale, one rounding to fp32), then add, then the activation, each
// as a separate fp32 operation like the un-fused instructions.
//
// CTA = 576 threads: warp 0 = TMA producer, warp 1 = tensor-memory owner + MMA issuer (both loop as
// whole warps and elect a lane around the instructions: 384 x 768 x 3072 int8 10.1 -> 8.6 us,
// 8192^3 fp16 888 -> 864 us against loops inside a one-lane branch), warps 2..17 = epilogue (each owns the TMEM lane
// quarter warp_id % 4 and a quarter of the tile's columns).  Two accumulator buffers of BN columns let the epilogue
// of tile i overlap the main loop of tile i+1.
//
// PAIR: the two CTAs of a cluster work on one tile of 256 x BN (cta_group::2).  Each loads its 128 rows of A and half
// of the tile's columns of B, and holds its 128 rows of D; the MMAs, issued by the first CTA, read B from both.
// What a k-block takes out of L2 per SM falls from 128 + BN rows to 128 + BN / 2, which is what bounds a tile of one
// CTA: 8192^3 int8 405 -> 328 us (3.35 POPS, tensor pipe at the clock the power allows), 1000 x 8192 x 8192 fp8 61 -> 54.
//
// SPLIT: the S CTAs of a cluster work on one tile of 128 x 64, each on its share of K; the grid is as many clusters as
// there are tiles.  The partial accumulators are exchanged through shared memory where the stages were, every warp
// adding (in the order of the ranks) and finishing 32 / S rows of 16 columns.  For few tiles and long K:
// one CTA walks a k-block in 0.2 us, 100 x 1000 x 4096 fp8 9.3 -> 6.6 us.
#pragma once
#include "common.cuh"
#include "ptx.cuh"
#include "qgemm_host.cuh"
#include "qgemm_math.cuh"
#include <cuda_fp16.h>
#include <cuda_fp8.h>

namespace mgx {

constexpr int BM        = 128; // rows of D per tile (UMMA M, one TMEM lane per row)
constexpr int BK        = 128; // bytes (= 8-bit elements) of K per pipeline stage
constexpr int UMMA_K    = 32;  // K per tcgen05.mma for 8-bit operands
constexpr int EPI_WARPS = 16;  // four per TMEM lane quarter, each takes a quarter of the columns
constexpr int NTHREADS  = 64 + 32 * EPI_WARPS;
constexpr int EPI_COLS  = 16;  // columns per epilogue chunk (one tcgen05.ld.32x32b.x16)

struct qgemm_params
{
    int64_t M, N, K, batch;
    int64_t ldd, stride_d;
    void* D;
    const float* scale;
    const float* bias;
    const void* residual;
    int tiles_m, tiles_n, group_m;
    int split; // CTAs that share a tile's K: 2, 4 or 8 (SPLIT)
    int64_t num_tiles;
    int num_kb;
    int scale_mode;
    int act;
    void* Dq;          // optional second output: quantizelinear(D) as int8 / fp8 (may be the only one)
    int64_t ldq, stride_q;
    float q_scale;     // per-tensor scale of that quantizelinear, already in D's type
    float q_zp;
    float q_rcp;       // 1 / q_scale refined to full precision
    int q_fp8;         // 0: int8, 1: fp8 e4m3fn
    int write_d;       // D itself is wanted
    int vec_sb; // scale / bias vectors are 16-byte aligned (float4 loads allowed)
    int fast;   // the whole problem takes the epilogue's check-free path (see epi_store_chunk_fast)
    int acc24;  // every accumulator is below 2^24 in magnitude (int8 operands, K < 1024)
    int q_mask; // the fused quantizelinear may take the mantissa-cut value (see launch_qgemm)
    int vec_io; // D (and residual) rows can be accessed with 16-byte (fp32/int32) / 8-byte (fp16) vectors
    // fp16 results whose epilogue operators run in half (MGX_QGEMM_HALF_MATH): 0xFFFFE000, the
    // mantissa cut that truncates an fp32 value in the normal half range to half; else all ones
    uint32_t hmask;
    const uint8_t* lut; // activation + quantizelinear of every half as a table (MGX_QOUT_LUT), or null
    float act_rcp; // erf-GELU: 1 / the constant x is divided by (sqrt 2, or its half value)
};

// v with the mantissa cut by mask (see qgemm_params::hmask); values in the half subnormal range
// keep up to 2^-24 too much, which no later step can see
__device__ __forceinline__ float hcut(float v, uint32_t mask)
{
    return __uint_as_float(__float_as_uint(v) & mask);
}

// the activation with every step rounded by hcut (all ones: the fp32 operator chain)
template <int ACT>
__device__ __forceinline__ float apply_act_cut(float v, uint32_t mask, float act_rcp)
{
    if constexpr(ACT == MGX_ACT_GELU_ERF)
    {
        // (x * 0.5) * (erf(x / c) + 1), operation order of src/op/builder/gelu.cpp:58-74; x * 0.5 is exact
        const float dv = hcut(v * act_rcp, mask);
        const float e1 = hcut(__fadd_rn(hcut(fast_erf(dv), mask), 1.0f), mask);
        return hcut(__fmul_rn(__fmul_rn(v, 0.5f), e1), mask);
    }
    else
        return apply_act<ACT>(v);
}

template <int BN, bool PAIR>
struct qgemm_smem
{
    static constexpr int b_rows      = PAIR ? BN / 2 : BN; // rows of B that this CTA loads
    static constexpr int a_bytes     = BM * BK;
    static constexpr int b_bytes     = b_rows * BK;
    static constexpr int stage_bytes = a_bytes + b_bytes;
    static constexpr int stages      = (b_rows >= 256) ? 4 : (b_rows >= 96 ? 6 : 8);
    static constexpr int epi_bytes   = EPI_WARPS * 32 * EPI_COLS * 4; // 32 rows x 16 words per warp
    static constexpr int bar_bytes   = 256;
    static constexpr int total = stages * stage_bytes + epi_bytes + bar_bytes + 1024; // + alignment slack
    static_assert(b_bytes % 1024 == 0 and total <= 227 * 1024, "operand tiles start on swizzle atoms and fit");
};

// columns of tensor memory between the two accumulators: BN, or the power of two above
template <int BN>
constexpr uint32_t ACC_COLS = BN <= 64 ? 64 : BN <= 128 ? 128 : 256;

// Tile r of one matrix.  Of pairs, groups of group_m rows of tiles, column by column within a group, so that the tiles
// at work at one time share panels of A as well as of B.
template <bool PAIR>
__device__ __forceinline__ void tile_place(const qgemm_params& p, int r, int& m_blk, int& n_blk)
{
    if constexpr(not PAIR)
    {
        m_blk = r % p.tiles_m;
        n_blk = r / p.tiles_m;
        return;
    }
    const int first = r / (p.group_m * p.tiles_n) * p.group_m;
    const int in    = r - first * p.tiles_n;
    const int rows  = min(p.group_m, p.tiles_m - first);
    n_blk           = in / rows;
    m_blk           = first + in - n_blk * rows;
}

struct epi_ctx
{
    const qgemm_params* p;
    uint8_t* box;      // this warp's 32 x 64-byte staging area (16-byte pieces XOR-swizzled by row)
    int rows;          // of it in use
    int lane;
    int64_t row0;      // global row of staging row 0
    int64_t batch_off; // b * stride_d
    int64_t batch_off_q; // b * stride_q
};

// Second half of the epilogue for one 16-column chunk: read the raw accumulators back
// from shared memory so that 4 consecutive lanes cover one 64-byte row segment, apply
// dequantizelinear / bias / activation / residual, convert and store coalesced.
template <bool IS_INT, class OutT, int ACT>
__device__ __forceinline__ void epi_store_chunk(const epi_ctx& e, int64_t col, float4 sc4, float4 bi4)
{
    const qgemm_params& p = *e.p;
    const int pc          = e.lane & 3;  // which 4-column piece of the chunk this lane owns
    const int rsub        = e.lane >> 2; // row within a group of 8
    const int64_t c4      = col + pc * 4;
    const float sc[4]     = {sc4.x, sc4.y, sc4.z, sc4.w};
    const float bi[4]     = {bi4.x, bi4.y, bi4.z, bi4.w};
    const bool full       = p.vec_io and c4 + 4 <= p.N;
    const bool has_bias   = p.bias != nullptr;
#pragma unroll 1
    for(int it = 0; it < 4; ++it)
    {
        const int r       = it * 8 + rsub;
        const int64_t row = e.row0 + r;
        const uint4 w =
            *reinterpret_cast<const uint4*>(e.box + r * 64 + ((pc ^ ((r >> 1) & 3)) * 16));
        if(r >= e.rows or row >= p.M or c4 >= p.N)
            continue;
        const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
        OutT* dst = static_cast<OutT*>(p.D) + e.batch_off + row * p.ldd + c4;
        if constexpr(std::is_same<OutT, int32_t>::value)
        {
            if(full)
                *reinterpret_cast<uint4*>(dst) = w;
            else
                for(int j = 0; j < 4 and c4 + j < p.N; ++j)
                    dst[j] = static_cast<int32_t>(wv[j]);
        }
        else
        {
            float v[4];
            float rs = 1.0f;
            if(p.scale_mode == MGX_SCALE_PER_ROW)
                rs = __ldg(p.scale + row);
#pragma unroll
            for(int j = 0; j < 4; ++j)
            {
                float x;
                const float s = p.scale_mode == MGX_SCALE_PER_ROW ? rs : sc[j];
                if constexpr(IS_INT)
                {
                    const int32_t a = static_cast<int32_t>(wv[j]);
                    x = p.scale_mode == MGX_SCALE_NONE ? (fits_small(a) ? int_to_float_small(a) : __int2float_rn(a)) : dequant_i32(a, s);
                }
                else
                {
                    x = __uint_as_float(wv[j]);
                    if(p.scale_mode != MGX_SCALE_NONE)
                        x = __fmul_rn(x, s);
                }
                if constexpr(std::is_same<OutT, __half>::value)
                {
                    x = hcut(x, p.hmask);
                    if(has_bias)
                        x = hcut(__fadd_rn(x, bi[j]), p.hmask);
                    v[j] = apply_act_cut<ACT>(x, p.hmask, p.act_rcp);
                }
                else
                {
                    if(has_bias)
                        x = __fadd_rn(x, bi[j]);
                    v[j] = apply_act<ACT>(x);
                }
            }
            if(p.residual != nullptr)
            {
                const OutT* res =
                    static_cast<const OutT*>(p.residual) + e.batch_off + row * p.ldd + c4;
                float q[4] = {0.f, 0.f, 0.f, 0.f};
                if(full)
                {
                    if constexpr(std::is_same<OutT, float>::value)
                    {
                        const float4 t = *reinterpret_cast<const float4*>(res);
                        q[0] = t.x, q[1] = t.y, q[2] = t.z, q[3] = t.w;
                    }
                    else
                    {
                        const uint2 t    = *reinterpret_cast<const uint2*>(res);
                        const __half* th = reinterpret_cast<const __half*>(&t);
#pragma unroll
                        for(int j = 0; j < 4; ++j)
                            q[j] = __half2float(th[j]);
                    }
                }
                else
                {
                    for(int j = 0; j < 4 and c4 + j < p.N; ++j)
                    {
                        if constexpr(std::is_same<OutT, float>::value)
                            q[j] = res[j];
                        else
                            q[j] = __half2float(res[j]);
                    }
                }
#pragma unroll
                for(int j = 0; j < 4; ++j)
                {
                    // fp16 model: the reference converts to half by truncating the mantissa
                    // (src/include/migraphx/generic_float.hpp:180-230) before the half add
                    if constexpr(std::is_same<OutT, __half>::value)
                        v[j] = truncate_to_half_precision(v[j]);
                    v[j] = __fadd_rn(v[j], q[j]);
                }
            }
            if constexpr(std::is_same<OutT, __half>::value)
            {
                // the stored value is the truncated half; a fused quantizelinear sees that value
                if(p.Dq != nullptr)
                {
#pragma unroll
                    for(int j = 0; j < 4; ++j)
                        v[j] = truncate_to_half_precision(v[j]);
                }
            }
            if(p.write_d)
            {
                if constexpr(std::is_same<OutT, float>::value)
                {
                    if(full)
                        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                    else
                        for(int j = 0; j < 4 and c4 + j < p.N; ++j)
                            dst[j] = v[j];
                }
                else
                {
                    if(full)
                        *reinterpret_cast<uint2*>(dst) =
                            make_uint2(cvt_rz_f16x2(v[0], v[1]), cvt_rz_f16x2(v[2], v[3]));
                    else
                        for(int j = 0; j < 4 and c4 + j < p.N; ++j)
                            dst[j] = __float2half_rz(v[j]);
                }
            }
            if(p.Dq != nullptr)
            {
                // quantizelinear of the value just produced (per-tensor scale and zero point):
                // x / s in D's type (fp16: fp32 quotient truncated to half, as migraphx::half
                // divides), round half to even, + zero point, saturate
                uint32_t packed = 0;
#pragma unroll
                for(int j = 0; j < 4; ++j)
                {
                    // correctly rounded v / s from the reciprocal computed once per kernel: the quotient is
                    // corrected once with its remainder (P. Markstein's theorem)
                    float qv        = __fmul_rn(v[j], p.q_rcp);
                    const float rem = __fmaf_rn(-p.q_scale, qv, v[j]);
                    qv              = __fmaf_rn(rem, p.q_rcp, qv);
                    uint32_t b;
                    if(p.q_fp8)
                    {
                        qv = fmaxf(-448.0f, fminf(448.0f, qv + p.q_zp));
                        b  = static_cast<uint32_t>(__nv_cvt_float_to_fp8(qv, __NV_SATFINITE, __NV_E4M3));
                    }
                    else
                    {
                        if constexpr(std::is_same<OutT, __half>::value)
                            qv = __uint_as_float(__float_as_uint(qv) & 0xFFFFE000u); // half quotient, truncated
                        // saturate first (keeps the magic-number rounding in range), then round
                        // half to even by adding 1.5 * 2^23; the low mantissa bits are the integer
                        qv = fmaxf(-300.0f, fminf(300.0f, qv));
                        const float r = __fadd_rn(qv, 12582912.0f);
                        int qi        = __float_as_int(r) - 0x4B400000 + static_cast<int>(p.q_zp);
                        qi            = max(-128, min(127, qi));
                        b             = static_cast<uint32_t>(qi) & 0xFFu;
                    }
                    packed |= b << (8 * j);
                }
                uint8_t* qdst = static_cast<uint8_t*>(p.Dq) + e.batch_off_q + row * p.ldq + c4;
                if(c4 + 4 <= p.N and ((reinterpret_cast<uintptr_t>(qdst) & 3u) == 0))
                    *reinterpret_cast<uint32_t*>(qdst) = packed;
                else
                    for(int j = 0; j < 4 and c4 + j < p.N; ++j)
                        qdst[j] = static_cast<uint8_t>(packed >> (8 * j));
            }
        }
    }
}

// float(half_rz(v)) for |v| < 65536 without a conversion and without a branch: normal halves
// keep the top 10 mantissa bits; below 2^-14 a half is a multiple of 2^-24, and |v| + 0.5 rounded
// toward zero keeps exactly those bits (the spacing of fp32 in [0.5, 1) is 2^-24).
__device__ __forceinline__ float half_rz_in_range(float v)
{
    const float av    = fabsf(v);
    const float big   = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
    const float small = copysignf(__fsub_rn(__fadd_rz(av, 0.5f), 0.5f), v);
    return av < 6.103515625e-5f ? small : big;
}

// Four values at once; the real conversion only when one of them is beyond the half range
// (or not a number).
__device__ __forceinline__ void truncate4_to_half_precision(float (&v)[4])
{
    const float hi = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    const float lo = fminf(fminf(fabsf(v[0]), fabsf(v[1])), fminf(fabsf(v[2]), fabsf(v[3])));
    if(hi < 65536.0f and lo >= 6.103515625e-5f)
    {
        // all four are normal halves (the common case): cut the mantissa
#pragma unroll
        for(int j = 0; j < 4; ++j)
            v[j] = __uint_as_float(__float_as_uint(v[j]) & 0xFFFFE000u);
    }
    else if(hi < 65536.0f)
    {
#pragma unroll
        for(int j = 0; j < 4; ++j)
            v[j] = half_rz_in_range(v[j]);
    }
    else
    {
#pragma unroll
        for(int j = 0; j < 4; ++j)
            v[j] = truncate_to_half_precision(v[j]);
    }
}

// The chunk's store phase when little needs checking: every column is in range, all accesses are
// vectors, the scale is per column or per tensor (already in sc4; 1.0 when
// there is none), bi4 is -0.0 without a bias (x + -0.0 == x for every x), an optional
// quantizelinear output is int8 with 4-byte aligned rows.  Same arithmetic as epi_store_chunk.
// MODE 1: residual / quantizelinear / D chosen by the launch's parameters; 2: D only;
// 3: residual, D and quantizelinear; 4: quantizelinear only; 8: residual and D (the combinations
// of an encoder layer's four GEMMs get branch-free loops of their own); 7: the table look-up.
template <bool IS_INT, class OutT, int ACT, int MODE>
__device__ __forceinline__ void epi_store_chunk_fast(const epi_ctx& e, int64_t col, float4 sc4, float4 bi4)
{
    const qgemm_params& p = *e.p;
    const int pc          = e.lane & 3;
    const int rsub        = e.lane >> 2;
    const float sc[4]     = {sc4.x, sc4.y, sc4.z, sc4.w};
    const float bi[4]     = {bi4.x, bi4.y, bi4.z, bi4.w};
    const int64_t off     = e.batch_off + (e.row0 + rsub) * p.ldd + col + pc * 4;
    OutT* dst             = static_cast<OutT*>(p.D) + off;
    const OutT* res       = static_cast<const OutT*>(p.residual) + off;
    uint8_t* qdst = static_cast<uint8_t*>(p.Dq) + e.batch_off_q + (e.row0 + rsub) * p.ldq + col + pc * 4;
    const int64_t dstep = 8 * p.ldd, qstep = 8 * p.ldq;
    // 5 = 2 and 6 = 4 with accumulators below 2^24 (and the mantissa-cut quantizelinear input)
    const bool has_res = MODE == 1 ? p.residual != nullptr : (MODE == 3 or MODE == 8);
    const bool has_q   = MODE == 1 ? p.Dq != nullptr : (MODE == 3 or MODE == 4 or MODE == 6 or MODE == 7);
    const bool wr      = MODE == 1 ? p.write_d != 0 : (MODE != 4 and MODE != 6 and MODE != 7);
    const bool acc24   = (MODE == 5 or MODE == 6) ? true : p.acc24 != 0;
    const bool q_mask  = MODE == 6 ? true : (has_q and p.q_mask != 0);
    // saturation before rounding: bounds are integers, so round-to-nearest stays inside
    const float q_lo = -128.0f - p.q_zp, q_hi = 127.0f - p.q_zp;
    const int q_bias = static_cast<int>(p.q_zp) - 0x4B400000;
    const uint32_t hmask = p.hmask;
    const uint8_t* box = e.box + rsub * 64;
    // (rows beyond M: only in the last row of tiles; one comparison per four values)
    const int rows = static_cast<int>(min(p.M - e.row0, static_cast<int64_t>(e.rows)));
#pragma unroll 2
    for(int it = 0; it < 4; ++it)
    {
        const int r   = it * 8 + rsub;
        if(r >= rows)
            break;
        const uint4 w = *reinterpret_cast<const uint4*>(box + it * 512 + ((pc ^ ((r >> 1) & 3)) * 16));
        const uint32_t wv[4] = {w.x, w.y, w.z, w.w};
        float v[4];
        if constexpr(IS_INT)
        {
            // one uniform branch around all four values, so that only one variant is issued
            if(acc24)
            {
                // |acc| < 2^24: the conversion is exact and the one fp32 multiply rounds like the
                // reference's double product; no range test, no large-accumulator path
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    v[j] = __fmul_rn(__int2float_rn(static_cast<int32_t>(wv[j])), sc[j]);
            }
            else
            {
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    v[j] = dequant_i32(static_cast<int32_t>(wv[j]), sc[j]);
            }
        }
        else
        {
#pragma unroll
            for(int j = 0; j < 4; ++j)
                v[j] = __fmul_rn(__uint_as_float(wv[j]), sc[j]);
        }
        if constexpr(MODE == 7)
        {
            // the half the chain holds after dequantizelinear and bias (the packing conversion
            // truncates, subnormal halves included) indexes the table of activation + quantizelinear
            const uint32_t i01 = cvt_rz_f16x2(__fadd_rn(hcut(v[0], hmask), bi[0]), __fadd_rn(hcut(v[1], hmask), bi[1]));
            const uint32_t i23 = cvt_rz_f16x2(__fadd_rn(hcut(v[2], hmask), bi[2]), __fadd_rn(hcut(v[3], hmask), bi[3]));
            const uint32_t b0 = __ldg(p.lut + (i01 & 0xFFFFu)), b1 = __ldg(p.lut + (i01 >> 16));
            const uint32_t b2 = __ldg(p.lut + (i23 & 0xFFFFu)), b3 = __ldg(p.lut + (i23 >> 16));
            *reinterpret_cast<uint32_t*>(qdst) = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
            qdst += qstep;
            continue;
        }
        if constexpr(std::is_same<OutT, __half>::value)
        {
            // fp16 model: dequantised value, bias sum and the activation's steps each rounded to half
            // when the launch asks for it (hmask), plain fp32 operators otherwise
#pragma unroll
            for(int j = 0; j < 4; ++j)
                v[j] = apply_act_cut<ACT>(hcut(__fadd_rn(hcut(v[j], hmask), bi[j]), hmask), hmask, p.act_rcp);
        }
        else
        {
#pragma unroll
            for(int j = 0; j < 4; ++j)
                v[j] = apply_act<ACT>(__fadd_rn(v[j], bi[j]));
        }
        if(has_res)
        {
            float q[4];
            if constexpr(std::is_same<OutT, float>::value)
            {
                const float4 t = *reinterpret_cast<const float4*>(res);
                q[0] = t.x, q[1] = t.y, q[2] = t.z, q[3] = t.w;
            }
            else
            {
                const uint2 t    = *reinterpret_cast<const uint2*>(res);
                const __half* th = reinterpret_cast<const __half*>(&t);
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    q[j] = __half2float(th[j]);
                truncate4_to_half_precision(v); // the half add works on the truncated half
            }
#pragma unroll
            for(int j = 0; j < 4; ++j)
                v[j] = __fadd_rn(v[j], q[j]);
        }
        if constexpr(std::is_same<OutT, __half>::value)
        {
            // quantizelinear sees the stored half
            if(q_mask)
            {
                // cutting the mantissa is enough: values in the half subnormal range quantise to
                // zero either way, values beyond the half range saturate either way, and the
                // store below truncates by itself
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    v[j] = __uint_as_float(__float_as_uint(v[j]) & 0xFFFFE000u);
            }
            else if(has_q)
                truncate4_to_half_precision(v);
        }
        if(wr)
        {
            if constexpr(std::is_same<OutT, float>::value)
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else
                *reinterpret_cast<uint2*>(dst) =
                    make_uint2(cvt_rz_f16x2(v[0], v[1]), cvt_rz_f16x2(v[2], v[3]));
        }
        if(has_q)
        {
            uint32_t b[4];
#pragma unroll
            for(int j = 0; j < 4; ++j)
            {
                float qv        = __fmul_rn(v[j], p.q_rcp);
                const float rem = __fmaf_rn(-p.q_scale, qv, v[j]);
                qv              = __fmaf_rn(rem, p.q_rcp, qv);
                if constexpr(std::is_same<OutT, __half>::value)
                    qv = __uint_as_float(__float_as_uint(qv) & 0xFFFFE000u); // half quotient, truncated
                qv   = fmaxf(q_lo, fminf(q_hi, qv));
                b[j] = static_cast<uint32_t>(__float_as_int(__fadd_rn(qv, 12582912.0f)) + q_bias);
            }
            *reinterpret_cast<uint32_t*>(qdst) =
                __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
        }
        dst += dstep;
        res += dstep;
        qdst += qstep;
    }
}

// The epilogue role, one instantiation per activation so that the code a warp executes is
// one contiguous region (the activation is chosen once per kernel, not per element).
// Each warp owns TMEM lane quarter (warp % 4) = 32 rows of the tile, and a quarter of the
// tile's columns.  Per 16-column chunk: tcgen05.ld (one row per thread) -> swizzled shared
// memory -> read back with 4 lanes per 64-byte row segment -> dequantizelinear / bias /
// activation / residual -> coalesced global stores.
template <int BN, bool IS_INT, class OutT, int ACT, int MODE, bool PAIR, bool SPLIT>
__device__ __forceinline__ void epilogue_role(const qgemm_params& p, uint8_t* epi_base, uint8_t* part, uint64_t* peer_bar,
                                              uint64_t* accf_bar, uint64_t* acce_bar,
                                              volatile uint32_t* abort_flag, uint32_t tmem_base,
                                              int warp, int lane, int64_t first_tile,
                                              int64_t tile_step, int64_t tiles_mn)
{
    const int ew      = warp - 2;
    const int quarter = warp & 3;
    const int slice   = ew >> 2;
    // this warp's chunks of the tile's columns: a quarter of them, or as near to it as whole chunks allow
    constexpr int CHUNKS = BN / EPI_COLS;
    // (the first case apart: one more register, and the int8 kernel of 128 columns spills)
    const int col_lo     = CHUNKS % 4 == 0 ? slice * (BN / 4) : slice * CHUNKS / 4 * EPI_COLS;
    const int nchunk     = CHUNKS % 4 == 0 ? CHUNKS / 4 : (slice + 1) * CHUNKS / 4 - slice * CHUNKS / 4;
    constexpr int ROWS   = PAIR ? 2 * BM : BM; // of a tile
    const int row_cta    = PAIR ? static_cast<int>(blockIdx.x & 1) * BM : 0;
    epi_ctx e;
    e.p    = &p;
    e.box  = epi_base + ew * (32 * EPI_COLS * 4);
    e.lane = lane;
    e.rows = 32;
    uint8_t* my_row    = e.box + lane * 64;
    const int my_swz   = (lane >> 1) & 3;
    const bool per_col = p.scale_mode == MGX_SCALE_PER_COL;
    const float tensor_scale = p.scale_mode == MGX_SCALE_PER_TENSOR ? __ldg(p.scale) : 1.0f;
    uint32_t lt = 0;
    for(int64_t t = first_tile; t < p.num_tiles; t += tile_step, ++lt)
    {
        const int b     = static_cast<int>(t / tiles_mn);
        const int r     = static_cast<int>(t % tiles_mn);
        int m_blk, n_blk;
        tile_place<PAIR>(p, r, m_blk, n_blk);
        const uint32_t buf = lt & 1u;
        int64_t col0 = static_cast<int64_t>(n_blk) * BN + col_lo;
        e.row0       = static_cast<int64_t>(m_blk) * ROWS + row_cta + quarter * 32;
        // SPLIT: unit u = 4 x chunk + quarter of the tile is finished by CTA u / units, S warps to a unit
        const int units = SPLIT ? EPI_WARPS / p.split : 1;
        const int unit  = SPLIT ? static_cast<int>(blockIdx.x) % p.split * units + ew / p.split : 0;
        if constexpr(SPLIT)
        {
            e.rows = 32 / p.split;
            col0   = static_cast<int64_t>(n_blk) * BN + (unit >> 2) * EPI_COLS;
            e.row0 = static_cast<int64_t>(m_blk) * BM + (unit & 3) * 32 + ew % p.split * e.rows;
        }
        e.batch_off = b * p.stride_d;
        e.batch_off_q = b * p.stride_q;

        // this lane's 4 columns of a chunk: scale and bias.  The first chunk's are fetched
        // before the wait for the accumulator (latency hidden behind the main loop), the
        // next chunk's while the current one is processed.  The loops below are deliberately
        // not unrolled: a tile's epilogue runs only a few times per launch, so straight-line
        // code would be bound by instruction fetch.
        auto load_sb = [&](int ch, float4& sc, float4& bi) {
            sc = make_float4(tensor_scale, tensor_scale, tensor_scale, tensor_scale);
            bi = MODE != 0 ? make_float4(-0.f, -0.f, -0.f, -0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr(not std::is_same<OutT, int32_t>::value)
            {
                const int64_t c4 = col0 + ch * EPI_COLS + (lane & 3) * 4;
                if(c4 + 4 <= p.N and p.vec_sb)
                {
                    if(per_col)
                        sc = __ldg(reinterpret_cast<const float4*>(p.scale + c4));
                    if(p.bias != nullptr)
                        bi = __ldg(reinterpret_cast<const float4*>(p.bias + c4));
                }
                else
                {
                    float* sp = reinterpret_cast<float*>(&sc);
                    float* bp = reinterpret_cast<float*>(&bi);
                    for(int j = 0; j < 4; ++j)
                    {
                        if(c4 + j < p.N)
                        {
                            if(per_col)
                                sp[j] = __ldg(p.scale + c4 + j);
                            if(p.bias != nullptr)
                                bp[j] = __ldg(p.bias + c4 + j);
                        }
                    }
                }
            }
        };
        // The residual is read inside the store loop; asking for its lines a chunk ahead turns
        // those reads into L1 hits (the loop is not unrolled, so their latency would be exposed).
        auto prefetch_res = [&](int ch) {
            if constexpr(not std::is_same<OutT, int32_t>::value)
            {
                const int64_t c4 = col0 + ch * EPI_COLS + (lane & 3) * 4;
                if(p.residual == nullptr or c4 >= p.N)
                    return;
#pragma unroll
                for(int it = 0; it < 4; ++it)
                {
                    const int64_t row = e.row0 + it * 8 + (lane >> 2);
                    if(row < p.M)
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(
                            static_cast<const OutT*>(p.residual) + e.batch_off + row * p.ldd + c4));
                }
            }
        };
        float4 sc_next, bi_next;
        load_sb(0, sc_next, bi_next);
        prefetch_res(0);

        if(not mbar_wait_bounded(&accf_bar[buf], (lt >> 1) & 1u, abort_flag, 3))
            break;
        tc_fence_after_sync();

        if constexpr(SPLIT)
        {
            static_assert(BN == 4 * EPI_COLS and not PAIR, "one chunk per warp");
            uint32_t acc[EPI_COLS];
            __syncwarp();
            tmem_ld_32x32b_x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + slice * EPI_COLS, acc);
            tmem_ld_wait();
            // (the accumulator being complete, the MMAs have read all that was in the stages)
            const int mine = slice * 4 + quarter;
            uint8_t* row   = part + mine * 2048 + lane * 64;
#pragma unroll
            for(int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(row + ((q ^ my_swz) * 16)) =
                    make_uint4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
            __syncwarp();
            if(lane == 0)
                cluster_arrive(peer_bar, mine / units);
            // units x S = 16 arrivals: all this CTA's units are in place in all CTAs
            if(not __all_sync(0xffffffffu, mbar_wait_cluster_bounded(peer_bar, 0, abort_flag, 6)))
                break;
            for(int i = lane; i < e.rows * 4; i += 32)
            {
                const int r = i >> 2, pc = i & 3, from = ew % p.split * e.rows + r;
                const uint8_t* src = part + unit * 2048 + from * 64 + ((pc ^ ((from >> 1) & 3)) * 16);
                uint4 v[8];
#pragma unroll
                for(int k = 0; k < 8; ++k)
                    if(k < p.split)
                        v[k] = cluster_load_uint4(src, k);
                uint4 sum = v[0];
#pragma unroll
                for(int k = 1; k < 8; ++k)
                    if(k < p.split)
                    {
                        if constexpr(IS_INT)
                            sum.x += v[k].x, sum.y += v[k].y, sum.z += v[k].z, sum.w += v[k].w;
                        else
                        {
                            sum.x = __float_as_uint(__uint_as_float(sum.x) + __uint_as_float(v[k].x));
                            sum.y = __float_as_uint(__uint_as_float(sum.y) + __uint_as_float(v[k].y));
                            sum.z = __float_as_uint(__uint_as_float(sum.z) + __uint_as_float(v[k].z));
                            sum.w = __float_as_uint(__uint_as_float(sum.w) + __uint_as_float(v[k].w));
                        }
                    }
                *reinterpret_cast<uint4*>(e.box + r * 64 + ((pc ^ ((r >> 1) & 3)) * 16)) = sum;
            }
            __syncwarp();
            if(col0 < p.N)
            {
                if constexpr(MODE != 0 and not std::is_same<OutT, int32_t>::value)
                    epi_store_chunk_fast<IS_INT, OutT, ACT, MODE>(e, col0, sc_next, bi_next);
                else
                    epi_store_chunk<IS_INT, OutT, ACT>(e, col0, sc_next, bi_next);
            }
            break; // one tile per cluster
        }

#pragma unroll 1
        for(int ch = 0; ch < nchunk; ++ch)
        {
            const int64_t col = col0 + ch * EPI_COLS;
            const float4 sc_cur = sc_next, bi_cur = bi_next;
            if(ch + 1 < nchunk)
            {
                load_sb(ch + 1, sc_next, bi_next);
                prefetch_res(ch + 1);
            }
            uint32_t acc[EPI_COLS];
            __syncwarp(); // tcgen05.ld is warp-collective; also orders reuse of the box
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   buf * ACC_COLS<BN> + col_lo + ch * EPI_COLS;
            tmem_ld_32x32b_x16(taddr, acc);
            tmem_ld_wait();
            if(col < p.N)
            {
#pragma unroll
                for(int q = 0; q < 4; ++q)
                    *reinterpret_cast<uint4*>(my_row + ((q ^ my_swz) * 16)) =
                        make_uint4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
                __syncwarp();
                if constexpr(MODE != 0 and not std::is_same<OutT, int32_t>::value)
                    epi_store_chunk_fast<IS_INT, OutT, ACT, MODE>(e, col, sc_cur, bi_cur);
                else
                    epi_store_chunk<IS_INT, OutT, ACT>(e, col, sc_cur, bi_cur);
            }
        }
        // all TMEM reads of this buffer are complete (wait::ld above)
        tc_fence_before_sync();
        __syncwarp();
        if(lane == 0)
        {
            if constexpr(PAIR)
                cluster_arrive(&acce_bar[buf], 0); // the CTA that issues the MMAs
            else
                mbar_arrive(&acce_bar[buf]);
        }
    }
}

// IS_INT: accumulator registers hold int32 (kind::i8) else fp32 bit patterns.
// OutT: int32_t (raw accumulator), float or __half.
// F16: the operands are fp16 (kind::f16, 64 elements of K per 128-byte stage row); the byte
// layout of the pipeline is the one of the 8-bit kinds.
template <int BN, bool IS_INT, class OutT, bool F16, bool PAIR, bool SPLIT>
__global__ void __launch_bounds__(NTHREADS, 1)
    qgemm_kernel(const __grid_constant__ CUtensorMap tmap_a,
                 const __grid_constant__ CUtensorMap tmap_b,
                 const qgemm_params p)
{
    using S = qgemm_smem<BN, PAIR>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem           = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);

    uint8_t* epi_base   = smem + S::stages * S::stage_bytes;
    uint8_t* bar_base   = epi_base + S::epi_bytes;
    uint64_t* full_bar  = reinterpret_cast<uint64_t*>(bar_base);
    uint64_t* empty_bar = full_bar + S::stages;
    uint64_t* accf_bar  = empty_bar + S::stages; // [2] accumulator ready
    uint64_t* acce_bar  = accf_bar + 2;          // [2] accumulator drained
    uint64_t* peer_bar  = acce_bar + 2;          // SPLIT: the cluster's partial sums are in place
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(peer_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    constexpr uint32_t TMEM_COLS = 2 * ACC_COLS<BN>;
    const uint32_t rank = PAIR ? blockIdx.x & 1u : 0u; // in the pair

    // the next kernel of the stream may set itself up while this one runs
    grid_launch_dependents();

    if(threadIdx.x == 0)
    {
        for(int s = 0; s < S::stages; ++s)
        {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for(int b = 0; b < 2; ++b)
        {
            mbar_init(&accf_bar[b], 1);
            mbar_init(&acce_bar[b], PAIR ? 2 * EPI_WARPS : EPI_WARPS); // one arrival per epilogue warp
        }
        mbar_init(peer_bar, EPI_WARPS);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_a);
        prefetch_tensormap(&tmap_b);
    }
    if(warp == 1)
    {
        if constexpr(PAIR)
        {
            tmem_alloc_pair(tmem_slot, TMEM_COLS);
            tmem_relinquish_pair();
        }
        else
        {
            tmem_alloc(tmem_slot, TMEM_COLS);
            tmem_relinquish();
        }
    }
    tc_fence_before_sync();
    if constexpr(PAIR or SPLIT)
        cluster_barrier(); // all its CTAs' barriers exist, a pair's tensor memory is allocated
    else
        __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    const int64_t first_tile = SPLIT ? blockIdx.x / p.split : PAIR ? blockIdx.x >> 1 : blockIdx.x;
    const int64_t tile_step  = SPLIT ? p.num_tiles : PAIR ? gridDim.x >> 1 : gridDim.x;
    // this CTA's blocks of K
    const int share = SPLIT ? static_cast<int>(blockIdx.x) % p.split : 0;
    const int kb_lo = SPLIT ? p.num_kb * share / p.split : 0;
    const int kb_hi = SPLIT ? p.num_kb * (share + 1) / p.split : p.num_kb;
    const int64_t tiles_mn   = static_cast<int64_t>(p.tiles_m) * p.tiles_n;

    if(warp == 0)
    {
        // ---------------------------------------------------- TMA producer
        // everything up to here overlapped the previous kernel of the stream; its results
        // (this kernel's operands) are complete after the wait
        grid_dependency_wait();
        uint32_t s = 0, ph = 1;
        bool ok    = true;
        for(int64_t t = first_tile; ok and t < p.num_tiles; t += tile_step)
        {
            const int b     = static_cast<int>(t / tiles_mn);
            const int r     = static_cast<int>(t % tiles_mn);
            int m_blk, n_blk;
            tile_place<PAIR>(p, r, m_blk, n_blk);
            for(int kb = kb_lo; kb < kb_hi; ++kb)
            {
                if(not mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2))
                {
                    ok = false;
                    break;
                }
                if(elect_one())
                {
                    uint8_t* sa = smem + s * S::stage_bytes;
                    if constexpr(PAIR)
                    {
                        // the first CTA's barrier counts both CTAs' bytes.  The second cannot get a phase
                        // ahead: its place is free again only when the MMAs that follow that phase are done
                        if(rank == 0)
                            mbar_expect_tx(&full_bar[s], 2 * S::stage_bytes);
                        tma_load_3d_pair(sa, &tmap_a, &full_bar[s], kb * BK, (2 * m_blk + static_cast<int>(rank)) * BM, b);
                        tma_load_3d_pair(sa + S::a_bytes, &tmap_b, &full_bar[s], kb * BK,
                                         n_blk * BN + static_cast<int>(rank) * S::b_rows, b);
                    }
                    else
                    {
                        mbar_expect_tx(&full_bar[s], S::stage_bytes);
                        tma_load_3d(sa, &tmap_a, &full_bar[s], kb * BK, m_blk * BM, b);
                        tma_load_3d(sa + S::a_bytes, &tmap_b, &full_bar[s], kb * BK, n_blk * BN, b);
                    }
                }
                if(++s == S::stages)
                    s = 0, ph ^= 1u;
            }
        }
        if constexpr(PAIR)
        {
            // The first CTA's MMAs release the stages of both.  The last release of each is waited for here too, so that
            // none arrives at a CTA that has left (a stage that was never filled is free).
            for(int i = 0; ok and i < S::stages; ++i)
            {
                ok = mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2);
                if(++s == S::stages)
                    s = 0, ph ^= 1u;
            }
        }
    }
    else if(warp == 1)
    {
        // ---------------------------------------------------- MMA issuer
        constexpr uint32_t UMMA_M = PAIR ? 2 * BM : BM;
        constexpr uint32_t idesc  = IS_INT ? make_idesc(2u, 1u, 1u, UMMA_M, BN)  // s32 += s8*s8
                                           : make_idesc(1u, 0u, 0u, UMMA_M, BN); // f32 += e4m3*e4m3 (f16*f16)
        // the operands arrive only after the previous kernel of the stream is done: the
        // bounded waits below must not count that time
        grid_dependency_wait();
        const uint64_t desc0 = make_smem_desc_sw128(smem_u32(smem));
        uint32_t s = 0, ph = 0;
        uint32_t lt = 0; // local tile counter
        bool ok     = rank == 0; // of a pair, the first CTA issues for both
        for(int64_t t = first_tile; ok and t < p.num_tiles; t += tile_step, ++lt)
        {
            const uint32_t buf = lt & 1u;
            if constexpr(PAIR)
            {
                if(not __all_sync(0xffffffffu, mbar_wait_cluster_bounded(&acce_bar[buf], ((lt >> 1) & 1u) ^ 1u, abort_flag, 4)))
                    break;
            }
            else if(not mbar_wait_warp(&acce_bar[buf], ((lt >> 1) & 1u) ^ 1u, abort_flag, 4))
                break;
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + buf * ACC_COLS<BN>;
            for(int kb = kb_lo; kb < kb_hi; ++kb)
            {
                if(not mbar_wait_warp(&full_bar[s], ph, abort_flag, 1))
                {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if(elect_one())
                {
                    const uint64_t adesc = desc0 + static_cast<uint64_t>((s * S::stage_bytes) >> 4);
                    const uint64_t bdesc = adesc + static_cast<uint64_t>(S::a_bytes >> 4);
#pragma unroll
                    for(int k = 0; k < BK / UMMA_K; ++k)
                    {
                        // advancing K inside the 128-byte swizzle row: +32 B on the start address
                        const uint64_t koff = static_cast<uint64_t>((k * UMMA_K) >> 4);
                        if constexpr(PAIR and IS_INT)
                            mma_i8_pair(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                        else if constexpr(PAIR and F16)
                            mma_f16_pair(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                        else if constexpr(PAIR)
                            mma_f8_pair(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                        else if constexpr(IS_INT)
                            mma_i8(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                        else if constexpr(F16)
                            mma_f16(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                        else
                            mma_f8(d_tmem, adesc + koff, bdesc + koff, idesc, ((kb - kb_lo) | k) != 0);
                    }
                    // the stage is reusable once these MMAs have read it; after the last, the accumulator complete
                    if constexpr(PAIR)
                    {
                        tc_commit_pair(&empty_bar[s]);
                        if(kb == kb_hi - 1)
                            tc_commit_pair(&accf_bar[buf]);
                    }
                    else
                    {
                        tc_commit(&empty_bar[s]);
                        if(kb == kb_hi - 1)
                            tc_commit(&accf_bar[buf]);
                    }
                }
                if(++s == S::stages)
                    s = 0, ph ^= 1u;
            }
        }
    }
    else
    {
        // ---------------------------------------------------- epilogue
        // (reads residual / scale / bias and writes D: only after the previous kernel is done)
        grid_dependency_wait();
        // the check-free variant is chosen once per launch: the tile loop a warp runs holds
        // only the store path it takes
#define MGX_EPI_MODE(ACT, MODE)                                                                           \
    epilogue_role<BN, IS_INT, OutT, ACT, MODE, PAIR, SPLIT>(p, epi_base, smem, peer_bar, accf_bar, acce_bar, abort_flag, \
                                                            tmem_base, warp, lane, first_tile, tile_step, tiles_mn)
// (fp16 operands have no quantised result, and only int32 accumulators a mode of their own below 2^24)
#define MGX_EPI_IF(COND, ACT, MODE) \
    if constexpr(COND)              \
    MGX_EPI_MODE(ACT, MODE)
#define MGX_EPILOGUE(ACT)                    \
    switch(mode)                             \
    {                                        \
    case 0: MGX_EPI_MODE(ACT, 0); break;     \
    case 2: MGX_EPI_MODE(ACT, 2); break;     \
    case 3: MGX_EPI_IF(not F16, ACT, 3); break; \
    case 4: MGX_EPI_IF(not F16, ACT, 4); break; \
    case 5: MGX_EPI_IF(IS_INT, ACT, 5); break; \
    case 6: MGX_EPI_IF(IS_INT, ACT, 6); break; \
    case 8: MGX_EPI_MODE(ACT, 8); break;     \
    default: MGX_EPI_IF(not F16, ACT, 1); break; \
    }
        const bool m_res = p.residual != nullptr, m_q = p.Dq != nullptr, m_wr = p.write_d != 0;
        const bool m_24  = IS_INT and p.acc24 != 0;
        const int mode   = p.fast == 0 ? 0
                           : (not m_res and not m_q and m_wr) ? (m_24 ? 5 : 2)
                           : (m_res and m_q and m_wr)         ? 3
                           : (m_res and not m_q and m_wr)     ? 8
                           : (not m_res and m_q and not m_wr) ? ((m_24 and p.q_mask != 0) ? 6 : 4)
                                                              : 1;
        if constexpr(std::is_same<OutT, int32_t>::value)
            MGX_EPI_MODE(MGX_ACT_NONE, 0);
        else if(std::is_same<OutT, __half>::value and not F16 and p.lut != nullptr and p.fast != 0 and not m_res and m_q and not m_wr)
        {
            if constexpr(std::is_same<OutT, __half>::value and not F16)
                MGX_EPI_MODE(MGX_ACT_NONE, 7);
        }
        else
            switch(p.act)
            {
            // (by itself and first: as the default behind the others its general path for fp32 results of int8 was 5 to
            // 9 % slower, 900 x 1500 x 512 6.3 -> 6.9 us)
            case MGX_ACT_NONE: MGX_EPILOGUE(MGX_ACT_NONE); break;
            case MGX_ACT_RELU: MGX_EPILOGUE(MGX_ACT_RELU); break;
            case MGX_ACT_GELU_ERF: MGX_EPILOGUE(MGX_ACT_GELU_ERF); break;
            case MGX_ACT_GELU_TANH: MGX_EPILOGUE(MGX_ACT_GELU_TANH); break;
            default: MGX_EPILOGUE(MGX_ACT_SILU); break;
            }
#undef MGX_EPILOGUE
#undef MGX_EPI_IF
#undef MGX_EPI_MODE
    }

    // ---------------------------------------------------------- teardown
    if(*abort_flag != 0)
    {
        // give copies that may still be in flight time to land before the CTA's
        // shared memory is released
        for(int i = 0; i < 1000; ++i)
            __nanosleep(1000);
    }
    tc_fence_before_sync();
    if constexpr(PAIR or SPLIT)
    {
        // no CTA leaves, or frees a pair's tensor memory, while another may still read its operands or partial sums or
        // arrive on its barriers
        cluster_barrier();
    }
    else
        __syncthreads();
    if(warp == 1)
    {
        tc_fence_after_sync();
        if constexpr(PAIR)
            tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else
            tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------ host

static int encode_operand_map(CUtensorMap* map, const void* base, int64_t k, int64_t rows,
                              int64_t batch, int64_t ld, int64_t batch_stride, int box_rows)
{
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[3]    = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows),
                             static_cast<cuuint64_t>(batch)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld),
                             static_cast<cuuint64_t>(batch > 1 ? batch_stride : ld * rows)};
    cuuint32_t box[3]     = {static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(box_rows), 1u};
    cuuint32_t estr[3]    = {1u, 1u, 1u};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MGX_OK : MGX_E_INVALID_ARG;
}

template <int BN, bool IS_INT, class OutT, bool F16, bool PAIR, bool SPLIT>
static int launch_qgemm(const mgx_qgemm_desc& d, const void* A, const void* B, void* D,
                        const float* scale, const float* bias, const void* residual,
                        int64_t ldb, int64_t stride_b, const qout_args& qo, int split, cudaStream_t stream)
{
    using S = qgemm_smem<BN, PAIR>;
    CUtensorMap ta, tb;
    constexpr int64_t ab = F16 ? 2 : 1; // bytes per operand element: the maps address bytes
    int rc = encode_operand_map(&ta, A, d.K * ab, d.M, d.batch, d.lda * ab, d.stride_a * ab, BM);
    if(rc != MGX_OK)
        return rc;
    rc = encode_operand_map(&tb, B, d.K * ab, d.N, d.batch, ldb * ab, stride_b * ab, S::b_rows);
    if(rc != MGX_OK)
        return rc;
    qgemm_params p{};
    constexpr int es = sizeof(OutT);
    p.vec_sb = ((reinterpret_cast<uintptr_t>(scale) & 15u) == 0 and (reinterpret_cast<uintptr_t>(bias) & 15u) == 0) ? 1 : 0;
    const int64_t valign = es == 4 ? 16 : 8; // bytes per lane in the coalesced store
    p.vec_io = ((reinterpret_cast<uintptr_t>(D) % valign) == 0 and (d.ldd * es) % valign == 0 and
                (d.batch == 1 or (d.stride_d * es) % valign == 0) and
                (residual == nullptr or (reinterpret_cast<uintptr_t>(residual) % valign) == 0))
                   ? 1
                   : 0;
    p.M          = d.M;
    p.N          = d.N;
    p.K          = d.K;
    p.batch      = d.batch;
    p.ldd        = d.ldd;
    p.stride_d   = d.stride_d;
    p.D          = D;
    p.scale      = scale;
    p.bias       = bias;
    p.residual   = residual;
    p.tiles_m    = static_cast<int>(ceil_div(d.M, PAIR ? 2 * BM : BM));
    p.tiles_n    = static_cast<int>((d.N + BN - 1) / BN);
    p.split      = split;
    p.group_m    = PAIR ? (p.tiles_m < 8 ? p.tiles_m : 8) : p.tiles_m;
    p.num_tiles  = static_cast<int64_t>(p.tiles_m) * p.tiles_n * d.batch;
    p.num_kb     = static_cast<int>((d.K * ab + BK - 1) / BK);
    p.scale_mode = d.scale_mode;
    p.act        = d.act;
    p.Dq         = qo.Dq;
    p.ldq        = qo.ldq;
    p.stride_q   = qo.stride_q;
    p.q_scale    = qo.scale;
    p.q_rcp      = static_cast<float>(1.0 / static_cast<double>(qo.scale));
    p.q_zp       = qo.zp;
    p.q_fp8      = qo.fp8;
    p.write_d    = qo.write_d;
    // the epilogue's check-free path: whole 16-column chunks in N, vector access everywhere
    // (a ragged last row of tiles costs it one comparison: 985 x 3072 x 768 took 20.8 us on the
    // general path, more than 3072 rows on this one), no per-row scale, quantizelinear output (if any) int8 in aligned words.
    // The residual shares D's leading dimension and must allow the same vector width.
    {
        const size_t es     = std::is_same<OutT, __half>::value ? 2 : 4;
        const size_t valign = es * 4;
        const bool res_ok   = residual == nullptr or (reinterpret_cast<uintptr_t>(residual) % valign) == 0;
        const bool q_ok     = qo.Dq == nullptr or
                          (qo.fp8 == 0 and (reinterpret_cast<uintptr_t>(qo.Dq) & 3u) == 0 and
                           qo.ldq % 4 == 0 and qo.stride_q % 4 == 0);
        p.fast = (not std::is_same<OutT, int32_t>::value and p.vec_io and p.vec_sb and res_ok and q_ok and
                  d.scale_mode != MGX_SCALE_PER_ROW and d.N % EPI_COLS == 0)
                     ? 1
                     : 0;
    }
    p.hmask      = (std::is_same<OutT, __half>::value and (d.flags & MGX_QGEMM_HALF_MATH) != 0) ? 0xFFFFE000u
                                                                                                 : 0xFFFFFFFFu;
    p.act_rcp    = p.hmask != 0xFFFFFFFFu ? 1.0f / 1.4140625f : 0.70710678118654752440f;
    // the table stands for activation + quantizelinear of a half: only where the chain holds one
    p.lut        = (p.hmask != 0xFFFFFFFFu and qo.fp8 == 0) ? static_cast<const uint8_t*>(qo.lut) : nullptr;
    p.acc24      = (IS_INT and d.K < 1024) ? 1 : 0; // |a b| <= 2^14 for int8 operands
    // |v| < 2^-14 (half subnormals) divided by a scale >= 2^-12 stays below 1/4: quantises to zero
    // whatever its low bits; no zero point may shift the rounding boundary
    p.q_mask     = (qo.Dq != nullptr and qo.fp8 == 0 and qo.scale >= 0.000244140625f and
                    qo.zp == static_cast<float>(static_cast<int>(qo.zp))) ? 1 : 0;
    auto kernel  = qgemm_kernel<BN, IS_INT, OutT, F16, PAIR, SPLIT>;
    int rc2 = ensure_smem_optin(reinterpret_cast<const void*>(kernel), S::total);
    if(rc2 != MGX_OK)
        return rc2;
    // (every group of SMs that clusters are placed in has an even number of them)
    const int sms  = PAIR ? device_sm_count() / 2 : device_sm_count();
    const int grid = SPLIT ? static_cast<int>(p.num_tiles) * split
                           : static_cast<int>(p.num_tiles < sms ? p.num_tiles : sms) * (PAIR ? 2 : 1);
    // programmatic dependent launch: set-up (tensor-memory allocation, barriers, descriptor
    // prefetch) overlaps the tail of the previous kernel of the stream
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = dim3(static_cast<unsigned>(grid));
    cfg.blockDim         = dim3(NTHREADS);
    cfg.dynamicSmemBytes = S::total;
    cfg.stream           = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id               = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(PAIR ? 2 : split);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = PAIR or SPLIT ? 2 : 1;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, ta, tb, p));
}

template <int BN, bool IS_INT, bool F16, bool PAIR, bool SPLIT = false>
static int dispatch_out(const mgx_qgemm_desc& d, const qgemm_operands& o, const qout_args& qo, cudaStream_t stream, int split = 1)
{
    switch(d.out_type)
    {
    case MGX_I32:
        if constexpr(IS_INT)
            return launch_qgemm<BN, true, int32_t, false, PAIR, SPLIT>(d, o.A, o.B, o.D, o.scale, o.bias, o.residual, o.ldb, o.stride_b, qo, split, stream);
        else
            return MGX_E_UNSUPPORTED;
    case MGX_F32:
        return launch_qgemm<BN, IS_INT, float, F16, PAIR, SPLIT>(d, o.A, o.B, o.D, o.scale, o.bias, o.residual, o.ldb, o.stride_b, qo, split, stream);
    case MGX_F16:
        return launch_qgemm<BN, IS_INT, __half, F16, PAIR, SPLIT>(d, o.A, o.B, o.D, o.scale, o.bias, o.residual, o.ldb, o.stride_b, qo, split, stream);
    default: return MGX_E_UNSUPPORTED;
    }
}

} // namespace mgx
