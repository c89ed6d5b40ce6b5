// What the two int4 decode kernels share (w4a16_tc.cu: work items dealt out evenly; w4a16_cluster.cu: a cluster
// splits K): shapes, the unpacking of packed weights, the staging of scales and zero points, the fold of the
// integer sums, and the host's tensor map, workspace head and choice of a form by the number of rows.
#pragma once
#include "common.cuh"
#include "ptx.cuh"
#include "w4a16_acts.cuh"
#include <cuda_fp16.h>

namespace mgx {

constexpr int TC_ROWS     = 128; // output columns (weight rows) per CTA tile = UMMA M
constexpr int TC_GROUP_K  = 128; // k per group
constexpr int TC_SUPER    = 4;   // groups per work item (each row gives 256 contiguous bytes)
constexpr int TC_PACKED   = TC_ROWS * TC_GROUP_K / 2; // 8192 bytes of packed weights per group
constexpr int TC_WSTAGE   = TC_SUPER * TC_PACKED;     // 32768
constexpr int TC_TSTAGES  = 2;   // A operand buffers in tensor memory
constexpr int TC_THREADS  = 480;
constexpr int TC_ISSUERS  = 4;   // MMA-issuing threads, one per group of a work item
constexpr int TC_ACC_COLS = 128; // accumulator columns per buffer (two buffers)
constexpr int TC_A_COL0   = 256; // first tensor-memory column of the A operand buffers
constexpr int TC_A_COLS   = TC_GROUP_K / 4; // 32 columns per group
constexpr int TC_EPI      = 3 * 128 * (5 + 3 + 2) * 4 + 64; // epilogue metadata

// NB: int8 activation rows of a group in the B operand.
// MR: activation rows folded by the epilogue (M <= MR <= MB).
// RAW: the weight operand of a group is [64 bytes of low nibbles | the 64 packed bytes] and every
// activation row has 4 rows in the B operand (see the pre-kernel); otherwise it is the 128
// nibbles unpacked to bytes and 2 rows.  RAW costs one logic operation per eight weights
// instead of three, and twice the accumulator columns per activation row.
// ESETS: sets of four epilogue warps; with two, each set folds half of the MR rows (the second
// set is warps 15..18).
template <int NB_, int MR_, bool RAW_, int ESETS_>
struct tc_form
{
    static constexpr int NB = NB_, MR = MR_, ESETS = ESETS_;
    static constexpr bool RAW   = RAW_;
    static constexpr int CPM    = RAW ? 4 : 2;      // accumulator columns per activation row
    static constexpr int MB     = NB / CPM;         // padded activation rows
    static constexpr int GPP    = TC_ACC_COLS / NB; // groups per pass (one accumulator buffer): 8 or 4
    static constexpr int ABYTES = NB * TC_GROUP_K;  // activation rows of one group
    static constexpr int MRW    = MR / ESETS;       // rows an epilogue warp folds
    static constexpr int C      = CPM * MRW;        // accumulator columns it reads per group
    static constexpr int THREADS = TC_THREADS + (ESETS - 1) * 128;
};

// f(form) with the form for M <= 16 rows
template <class F>
int tc_by_rows(int64_t M, F f)
{
    if(M == 1)
        return f(tc_form<16, 1, true, 1>{});
    if(M == 2)
        return f(tc_form<16, 2, true, 1>{});
    if(M <= 4)
        return f(tc_form<16, 4, true, 1>{});
    if(M <= 8)
        return f(tc_form<32, 8, true, 2>{});
    return f(tc_form<32, 16, false, 2>{});
}

// kernel arguments of both
struct tc_operands
{
    const __half* scales;
    const uint8_t* zp; // may be null
    const float* sa;   // [K/128][MB] activation scale of every (group, row)
    const int* sv;     // [K/128][MB] per-group sums of the quantised activations
    __half* D;
    int64_t N, K, ldd;
    int M, group, groups_per_row, zp_const;
};

// Epilogue metadata in shared memory, three buffers each: per output column the aligned 32-bit words that
// hold the scales (at most 5) and zero points (at most 3) of a pass, GPP x MB activation group sums and
// group scales.
struct tc_meta
{
    uint32_t* sw; // [3][128][5]
    uint32_t* zw; // [3][128][3]
    int* sv;      // [3][128]
    float* sa;    // [3][128]
    __device__ explicit tc_meta(uint8_t* base)
        : sw(reinterpret_cast<uint32_t*>(base)),
          zw(sw + 3 * 128 * 5),
          sv(reinterpret_cast<int*>(zw + 3 * 128 * 3)),
          sa(reinterpret_cast<float*>(sv + 3 * 128))
    {
    }
};

// cp.async copies of the words around the scales and zero points of a pass (consecutive lanes copy
// consecutive words of a column's run, so a request touches few sectors) and of the activation group sums,
// into buffer vb; `half` of two warps serves 64 output columns.
template <int MB>
__device__ __forceinline__ void tc_stage_metadata(const tc_operands& p, const tc_meta& meta, uint32_t vb, int half, int lane,
                                                  int tile, int g0, int count)
{
    const int rshift = 31 - __clz(p.group / TC_GROUP_K); // groups are powers of two
    const uint32_t sbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.scales) & 3u);
    const uint32_t zbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.zp) & 3u);
    const char* sptr = reinterpret_cast<const char*>(p.scales) - sbase0; // 4-byte aligned
    const char* zptr = reinterpret_cast<const char*>(p.zp) - zbase0;
    auto cp_async4 = [](const void* dst, const void* src) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    };
    const int gi0 = g0 >> rshift;
    const int ng  = ((g0 + count - 1) >> rshift) - gi0 + 1;
    const int n0  = tile * TC_ROWS + half * 64;
    // scales: up to 5 words per column
#pragma unroll 2
    for(int idx = lane; idx < 64 * 5; idx += 32)
    {
        const int r = idx / 5, w = idx - r * 5;
        const int n = min(n0 + r, static_cast<int>(p.N) - 1);
        // byte offsets from the aligned base: first scale, end of the run
        const uint32_t s = sbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0) * 2u;
        const uint32_t a = s & ~3u;
        const int nw     = static_cast<int>((((s + ng * 2 + 3u) & ~3u) - a) >> 2);
        if(w < nw)
            cp_async4(meta.sw + (vb * 128 + half * 64 + r) * 5 + w, sptr + a + 4 * w);
    }
    if(p.zp != nullptr)
    {
#pragma unroll 2
        for(int idx = lane; idx < 64 * 3; idx += 32)
        {
            const int r = idx / 3, w = idx - r * 3;
            const int n = min(n0 + r, static_cast<int>(p.N) - 1);
            const uint32_t z = zbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0);
            const uint32_t a = z & ~3u;
            const int nw     = static_cast<int>((((z + ng + 3u) & ~3u) - a) >> 2);
            if(w < nw)
                cp_async4(meta.zw + (vb * 128 + half * 64 + r) * 3 + w, zptr + a + 4 * w);
        }
    }
    // group sums and group scales: count x MB words each, half of them per warp
    for(int i = half * 64 + lane; i < count * MB; i += 32)
        if(i < half * 64 + 64)
        {
            cp_async4(meta.sv + vb * 128 + i, p.sv + static_cast<int64_t>(g0) * MB + i);
            cp_async4(meta.sa + vb * 128 + i, p.sa + static_cast<int64_t>(g0) * MB + i);
        }
}

// The `cnt` groups of a work item for one weight row: 64 packed bytes per group from shared memory (128-byte
// swizzle, so a quarter warp's 16-byte reads fall in eight different bank groups), 32 words to this row's lane
// of tensor memory: either the nibbles as bytes (inside every 8 k the evens first, then the odds; the
// activation rows are stored in the same order) or the low nibbles followed by the packed bytes as they are
// (RAW).  stage: [pair of groups][row][128 bytes], 16-byte chunks swizzled by the row.
template <bool RAW>
__device__ __forceinline__ void tc_unpack_item(const uint8_t* stage, int row, int cnt, uint32_t taddr)
{
    const int sw = row & 7;
#pragma unroll
    for(int q = 0; q < TC_SUPER; ++q)
    {
        if(q < cnt)
        {
            const uint8_t* pk = stage + (q >> 1) * (2 * TC_PACKED) + row * 128;
            uint32_t u[32];
#pragma unroll
            for(int c = 0; c < 4; ++c)
            {
                const uint4 w = *reinterpret_cast<const uint4*>(pk + ((((q & 1) * 4 + c) ^ sw) << 4));
                if constexpr(RAW)
                {
                    u[4 * c + 0] = w.x & 0x0F0F0F0Fu, u[16 + 4 * c + 0] = w.x;
                    u[4 * c + 1] = w.y & 0x0F0F0F0Fu, u[16 + 4 * c + 1] = w.y;
                    u[4 * c + 2] = w.z & 0x0F0F0F0Fu, u[16 + 4 * c + 2] = w.z;
                    u[4 * c + 3] = w.w & 0x0F0F0F0Fu, u[16 + 4 * c + 3] = w.w;
                }
                else
                {
                    u[8 * c + 0] = w.x & 0x0F0F0F0Fu, u[8 * c + 1] = (w.x >> 4) & 0x0F0F0F0Fu;
                    u[8 * c + 2] = w.y & 0x0F0F0F0Fu, u[8 * c + 3] = (w.y >> 4) & 0x0F0F0F0Fu;
                    u[8 * c + 4] = w.z & 0x0F0F0F0Fu, u[8 * c + 5] = (w.z >> 4) & 0x0F0F0F0Fu;
                    u[8 * c + 6] = w.w & 0x0F0F0F0Fu, u[8 * c + 7] = (w.w >> 4) & 0x0F0F0F0Fu;
                }
            }
            tmem_st_32x32b_x32(taddr + q * TC_A_COLS, u);
        }
    }
}

// The groups of a pass for one output column `col` of the tile (= lane of tensor memory) and the MRW
// activation rows from m0: out[m] += sc sa[m] (Q[m] - z Sv[m]) with Q = sum_k q a_int, in exact integer
// arithmetic up to the one conversion.  Scale, zero point and activation group sums are in shared memory
// (buffer vb).  All arithmetic stays off the conversion pipe except one half -> float per group.
// acc_addr: accumulator buffer, this warp's lanes, first column.
template <class FORM>
__device__ __forceinline__ void tc_fold_pass(const tc_operands& p, const tc_meta& meta, uint32_t vb, int col, int m0, int tile,
                                             int g0, int count, uint32_t acc_addr, float (&out)[FORM::MRW])
{
    constexpr int C = FORM::C, MB = FORM::MB;
    // groups read from tensor memory per trip (all loads in flight before the first fold)
    constexpr int TR      = C <= 4 ? 8 : (C <= 8 ? 4 : 2);
    const bool has_zp     = p.zp != nullptr;
    const int rshift      = 31 - __clz(p.group / TC_GROUP_K); // groups are powers of two
    const uint32_t sbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.scales) & 3u);
    const uint32_t zbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.zp) & 3u);
    const int gi0         = g0 >> rshift;
    const int n           = min(tile * TC_ROWS + col, static_cast<int>(p.N) - 1);
    // this column's first scale / zero point inside its staged words, in bytes
    const uint32_t sbyte = (sbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0) * 2u) & 3u;
    const uint32_t zbyte = (zbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0)) & 3u;
    auto fold = [&](const uint32_t(&acc)[C], int gl) {
        // quantisation group of group gl, relative to gi0
        const uint32_t grel = static_cast<uint32_t>(((g0 + gl) >> rshift) - gi0);
        const uint32_t soff = sbyte + 2u * grel, zoff = zbyte + grel;
        const uint32_t sw   = meta.sw[(vb * 128 + col) * 5 + (soff >> 2)];
        const uint32_t sh   = (soff & 2u) ? sw >> 16 : sw & 0xFFFFu;
        float sc            = __half2float(__ushort_as_half(static_cast<unsigned short>(sh)));
        // without zero points the staged word is not meaningful and not used
        const uint32_t zw = meta.zw[(vb * 128 + col) * 3 + (has_zp ? zoff >> 2 : 0u)];
        int z = has_zp ? static_cast<int>((zw >> (8u * (zoff & 3u))) & 0xFFu) : p.zp_const;
        if constexpr(FORM::RAW)
        {
            sc *= 0.0625f; // Q is computed times 16
            z *= 16;
        }
        const int* svb   = meta.sv + vb * 128 + gl * MB + m0;
        const float* sab = meta.sa + vb * 128 + gl * MB + m0;
#pragma unroll
        for(int m = 0; m < FORM::MRW; ++m)
        {
            int q;
            if constexpr(FORM::RAW)
            {
                // columns: sum L e_h, 16 sum q_odd o_h, sum L e_l, 16 sum q_odd o_l;
                // 16 Q = 2048 E_h + 128 O_h + 16 E_l + O_l
                q = static_cast<int>(acc[4 * m]) * 2048 + static_cast<int>(acc[4 * m + 3]);
                q = static_cast<int>(acc[4 * m + 1]) * 128 + q;
                q = static_cast<int>(acc[4 * m + 2]) * 16 + q;
            }
            else // columns: P_hi, P_lo, below 2^18 in magnitude
                q = static_cast<int>(acc[2 * m]) * 128 + static_cast<int>(acc[2 * m + 1]);
            q      = q - z * svb[m];
            out[m] = fmaf(sc * sab[m], static_cast<float>(q), out[m]);
        }
    };
#pragma unroll 1
    for(int gl = 0; gl < count; gl += TR)
    {
        uint32_t acc[TR][C];
        if(gl + TR <= count)
        {
            // full trip: straight-line code, the folds interleave
#pragma unroll
            for(int t = 0; t < TR; ++t)
                tmem_ld_32x32b<C>(acc_addr + (gl + t) * FORM::NB, acc[t]);
            tmem_ld_wait();
#pragma unroll
            for(int t = 0; t < TR; ++t)
                fold(acc[t], gl + t);
        }
        else
        {
#pragma unroll
            for(int t = 0; t < TR; ++t)
                if(gl + t < count) // the same for the whole warp
                    tmem_ld_32x32b<C>(acc_addr + (gl + t) * FORM::NB, acc[t]);
            tmem_ld_wait();
#pragma unroll
            for(int t = 0; t < TR; ++t)
                if(gl + t < count)
                    fold(acc[t], gl + t);
        }
    }
}

// ------------------------------------------------------------------ host
namespace {

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Sizes of a problem and the head of the workspace: activation planes, group scales, group sums.
struct tc_layout
{
    int nb, mb, tiles, groups, blocks; // blocks: work items of a tile
    size_t off_sa, off_sv, end;
    explicit tc_layout(const mgx_w4_desc& d)
    {
        // up to 8 rows: 4 int8 rows per activation row (RAW operand); up to 16: 2 rows
        nb     = d.M <= 4 ? 16 : 32;
        mb     = d.M <= 4 ? 4 : (d.M <= 8 ? 8 : 16);
        tiles  = static_cast<int>(ceil_div(d.N, TC_ROWS));
        groups = static_cast<int>(d.K / TC_GROUP_K);
        blocks = (groups + TC_SUPER - 1) / TC_SUPER;
        off_sa = align_up(static_cast<size_t>(nb) * d.K, 256);
        off_sv = align_up(off_sa + static_cast<size_t>(groups) * mb * sizeof(float), 256);
        end    = off_sv + static_cast<size_t>(groups) * mb * sizeof(int);
    }
};

// Tensor maps of the packed weights (rows of K / 2 bytes; one request = 128 rows x 128 bytes, two groups) and
// of the planes at the head of the workspace, the pre-kernel that fills it, and the kernel's operands.
int tc_prepare(const mgx_w4_desc& d, const tc_layout& lay, const void* A, const void* Bp, const void* scales, const void* zp,
               void* D, uint8_t* ws, int* counters, int ncounters, cudaStream_t stream, CUtensorMap& tw, CUtensorMap& ta,
               tc_operands& p)
{
    auto* aq = reinterpret_cast<int8_t*>(ws);
    auto* sa = reinterpret_cast<float*>(ws + lay.off_sa);
    auto* sv = reinterpret_cast<int*>(ws + lay.off_sv);
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[2]    = {static_cast<cuuint64_t>(d.K / 2), static_cast<cuuint64_t>(d.N)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(d.K / 2)};
    cuuint32_t box[2]     = {128u, TC_ROWS};
    cuuint32_t estr[2]    = {1u, 1u};
    if(encode(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(Bp), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return MGX_E_INVALID_ARG;
    int rc = encode_grouped(&ta, aq, TC_GROUP_K, static_cast<uint64_t>(lay.nb), static_cast<uint64_t>(d.K),
                            static_cast<uint64_t>(lay.groups), static_cast<uint32_t>(lay.nb), TC_SUPER,
                            CU_TENSOR_MAP_SWIZZLE_128B);
    if(rc != MGX_OK)
        return rc;
    rc = launch_prepare_acts(lay.mb, static_cast<const __half*>(A), d.lda, d.M, d.K, aq, sa, sv, counters, ncounters, stream);
    if(rc != MGX_OK)
        return rc;
    p.scales         = static_cast<const __half*>(scales);
    p.zp             = static_cast<const uint8_t*>(zp);
    p.sa             = sa;
    p.sv             = sv;
    p.D              = static_cast<__half*>(D);
    p.M              = static_cast<int>(d.M);
    p.N              = d.N;
    p.K              = d.K;
    p.ldd            = d.ldd;
    p.group          = d.group;
    p.groups_per_row = static_cast<int>(d.K / d.group);
    p.zp_const       = d.zp_const;
    return MGX_OK;
}

} // namespace

} // namespace mgx
