// Decode-step attention of a grouped-query decoder layer against the fp16 KV cache, one launch.
//
// Stands in for the operator chain the GroupQueryAttention parser emits after concat_past_present
// (src/onnx/parse_group_query_attention.cpp:184-262): the KV heads broadcast to the query heads,
// dot(Q, K^T) over the whole cache length, mul by the scale, where(position > seqlens_k, -inf),
// softmax, dot(P, V).  With one query row per head this is a stream over the valid part of the
// cache: HBM-bound, 2 * (seqlens_k + 1) * head * 2 bytes per (batch entry, KV head), read once for
// all the query heads that share the KV head.  Positions beyond seqlens_k (up to the end of a tile of
// 64) take no part: their probabilities are exactly zero in the chain.
//
// One or two persistent CTAs per SM; a job is a (batch entry, KV head), taken by a cluster of CTAs, each
// with a consecutive range of the valid positions.  Row maximum, sum of exponentials and the partial
// outputs are exchanged through distributed shared memory, so there is no second launch and no scratch
// in global memory.  A CTA's share goes through a ring of tiles of 64 positions, filled by TMA (128-byte
// swizzle) with all the keys of a job and then all its values: values travel while the scores are still
// being turned into probabilities, the keys of the next job while this one's result is added up.
// (With 16-byte loads by the threads themselves between the barriers, one job per CTA: 512 jobs of up
// to 2048 positions 86 us; so 69 us = 5.5 TB/s.)
//
// The chain's fp16 roundings are kept (migraphx::half truncates, src/include/migraphx/generic_float.hpp):
// the score is cut to half after the dot and after the scaling, exp(x - max) is cut to half, the
// sum runs over those halves in fp32, the quotient is cut to half before P V (ref_softmax,
// src/targets/ref/lowering.cpp:282-313).  Dots accumulate in fp32 (the reference: double).
#include "common.cuh"
#include "ptx.cuh"
#include "qgemm_math.cuh"
#include <algorithm>
#include <cuda_fp16.h>
#include <mutex>

namespace mgx {

constexpr int GD_WARPS      = 8;
constexpr int GD_THREADS    = 32 * GD_WARPS; // consumers; one more warp requests tiles
constexpr int GD_TILE       = 64;            // positions
constexpr int GD_HEADS      = 8;             // query heads per KV head, padded
constexpr int GD_MAX_STAGES = 12;
constexpr int GD_MAX_SPLIT  = 8;

struct gqa_decode_params
{
    const __half* q; // [batch][heads] rows of `head` contiguous halves
    int64_t q_sb, q_sh;
    int q_vec; // query rows can be read as 16-byte vectors
    const void* seqlens;
    int seqlens_i64;
    __half* out; // [batch, heads * head]
    float scale;
    int cache_seq, kv_heads, fact;
    int jobs, split; // (batch entry, KV head) pairs; CTAs of a cluster
    int cap, pitch, stages; // score columns a CTA holds in shared memory; tiles of its ring
};

__device__ __forceinline__ float gd_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// v >= 0 cut to half precision, subnormal halves included
__device__ __forceinline__ float gd_trunc_nonneg(float v)
{
    const float big   = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
    const float small = __fsub_rn(__fadd_rz(v, 0.5f), 0.5f);
    return v < 6.103515625e-5f ? small : big;
}

__device__ __forceinline__ void gd_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void gd_ldmatrix_trans(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void gd_consumer_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(GD_THREADS) : "memory"); }

// D: head size (64 or 128).  Both products are mma.sync m16n8k16 with the query heads of the KV head as
// the 8 columns, 16 positions (scores) or 16 output columns (P V) as the rows:
//  * Q K^T: the order of the contraction index inside a fragment is free, so lane (g, t) takes the 8
//    consecutive halves at 32 b + 8 t of its two positions as 16-byte reads for the two 16-wide steps of
//    block b, and of its query head once per job;
//  * P V: A = V^T by transposing ldmatrix, B = the probabilities, made from the stored exponentials
//    where they are used.
template <int D>
__global__ void __launch_bounds__(GD_THREADS + 32, 2)
    gqa_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const gqa_decode_params p)
{
    constexpr int NB      = D / 32;          // 32-wide blocks of the head dimension
    constexpr int HALVES  = D / 64;          // 128-byte halves of a row
    constexpr int TBYTES  = GD_TILE * D * 2; // bytes of a tile: [half][position][128 bytes]
    constexpr float log2e = 1.4426950408889634f;
    extern __shared__ uint8_t gd_raw[];
    __shared__ float red_m[GD_HEADS], red_s[GD_HEADS]; // this CTA's maxima / sums, read by the cluster
    __shared__ float wred[GD_WARPS][GD_HEADS];         // per-warp partials
    __shared__ float cta_out[GD_HEADS * D];            // this CTA's partial output, read by the cluster
    __shared__ float tot_m[GD_HEADS], tot_s[GD_HEADS];
    __shared__ uint64_t full_bar[GD_MAX_STAGES], empty_bar[GD_MAX_STAGES], peer_bar;
    __shared__ uint32_t abort_word;
    volatile uint32_t* abort_flag = &abort_word;
    uint8_t* ring = gd_raw + ((1024u - (smem_u32(gd_raw) & 1023u)) & 1023u);
    __half* sc    = reinterpret_cast<__half*>(ring + p.stages * TBYTES); // [heads][cap] scores, then exponentials
    float* part   = reinterpret_cast<float*>(sc);                        // [warps][heads][D], after the exponentials

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    grid_launch_dependents();
    if(tid == 0)
    {
        for(int s = 0; s < p.stages; ++s)
        {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], GD_TILE / 16); // one warp per 16 positions
        }
        mbar_init(&peer_bar, p.split);
        abort_word = 0;
        fence_barrier_init();
    }
    __syncthreads();
    // the other CTAs' barriers exist before anyone arrives on them: waited for at the first exchange
    if(p.split > 1)
        cluster_barrier_arrive();
    const int rank  = static_cast<int>(blockIdx.x) % p.split;
    const int first = static_cast<int>(blockIdx.x) / p.split, step = static_cast<int>(gridDim.x) / p.split;
    grid_dependency_wait(); // caches, queries and lengths may come from the previous kernel

    // Positions k0 .. k0 + n - 1 of job (batch entry, KV head) are this CTA's.  Positions 0 .. seqlens_k
    // take part; a length outside the cache is clamped (the chain would mask nothing beyond the cache).
    auto share = [&](int job, int& k0) {
        const int b        = job / p.kv_heads;
        const int64_t last = p.seqlens_i64 ? static_cast<const int64_t*>(p.seqlens)[b]
                                           : static_cast<int64_t>(static_cast<const int32_t*>(p.seqlens)[b]);
        const int len   = last < 0 ? 1 : (last + 1 > p.cache_seq ? p.cache_seq : static_cast<int>(last + 1));
        const int chunk = min((len + p.split - 1) / p.split, p.cap);
        k0              = rank * chunk;
        return max(min(len, k0 + chunk) - k0, 0);
    };

    if(warp == GD_WARPS)
    {
        // ---------------------------------------------------- producer
        int s = 0, ph = 1;
        bool ok = true;
        for(int job = first; ok and job < p.jobs; job += step)
        {
            int k0;
            const int tiles = (share(job, k0) + GD_TILE - 1) / GD_TILE;
            for(int i = 0; ok and i < 2 * tiles; ++i)
            {
                ok = mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2);
                if(ok and elect_one())
                {
                    mbar_expect_tx(&full_bar[s], TBYTES);
                    const int pos = k0 + (i < tiles ? i : i - tiles) * GD_TILE;
                    for(int h = 0; h < HALVES; ++h)
                        tma_load_3d(ring + s * TBYTES + h * GD_TILE * 128, i < tiles ? &tmap_k : &tmap_v, &full_bar[s], h * 64,
                                    pos, job);
                }
                if(++s == p.stages)
                    s = 0, ph ^= 1;
            }
        }
        if(p.split > 1)
            cluster_barrier_wait();
    }
    else
    {
        // ---------------------------------------------------- consumers
        const int g = lane >> 2, t = lane & 3; // fragment coordinates
        // position (of eight) that stands for MMA row g: rows four apart are in different halves of the
        // swizzled 128 bytes, so that lanes 8 i .. 8 i + 7 read all banks
        const int prow = (g >> 1) | ((g & 1) << 2);
        bool dead      = false; // a wait gave up: go on without waiting
        int tile0      = 0;     // tiles of earlier jobs
        int xch        = 0;     // exchanges so far
        // every CTA of the cluster has written what it announces
        auto exchange = [&]() {
            gd_consumer_barrier();
            if(p.split > 1)
            {
                if(xch == 0)
                    cluster_barrier_wait();
                if(tid < p.split)
                    cluster_arrive(&peer_bar, tid);
                if(not dead and not __all_sync(0xffffffffu, mbar_wait_cluster_bounded(&peer_bar, xch & 1, abort_flag, 6)))
                    dead = true;
            }
            ++xch;
        };
        // what the CTAs of the cluster hold at `at`, added in their order, or the largest: all under way together (one
        // after another 0.2 us each; eight reads for two CTAs: 32 heads, 128 positions 6.1 -> 6.4 us)
        auto of_cluster = [&](const float* at, bool largest) {
            float v[GD_MAX_SPLIT];
#pragma unroll
            for(int r = 0; r < GD_MAX_SPLIT; ++r)
                if(r < p.split)
                    v[r] = __uint_as_float(cluster_load(at, r));
            float x = v[0];
#pragma unroll
            for(int r = 1; r < GD_MAX_SPLIT; ++r)
                if(r < p.split)
                    x = largest ? fmaxf(x, v[r]) : x + v[r];
            return x;
        };
        auto wait_tile = [&](int tile) {
            if(not dead and not mbar_wait_warp(&full_bar[tile % p.stages], (tile / p.stages) & 1, abort_flag, 1))
                dead = true;
            return ring + (tile % p.stages) * TBYTES;
        };
        auto release_tile = [&](int tile) {
            __syncwarp();
            if(lane == 0)
                mbar_arrive(&empty_bar[tile % p.stages]);
        };
        for(int job = first; job < p.jobs; job += step)
        {
            int k0;
            const int n      = share(job, k0);
            const int tiles  = (n + GD_TILE - 1) / GD_TILE;
            const int b      = job / p.kv_heads;
            const int64_t h0 = static_cast<int64_t>(job % p.kv_heads) * p.fact;
            // query head g, halves 32 b + 8 t .. + 7 (zero for the padding heads)
            uint32_t qb[NB][4];
#pragma unroll
            for(int blk = 0; blk < NB; ++blk)
            {
                qb[blk][0] = qb[blk][1] = qb[blk][2] = qb[blk][3] = 0u;
                if(g < p.fact)
                {
                    const __half* src = p.q + b * p.q_sb + (h0 + g) * p.q_sh + blk * 32 + t * 8;
                    if(p.q_vec)
                    {
                        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(src));
                        qb[blk][0] = v.x, qb[blk][1] = v.y, qb[blk][2] = v.z, qb[blk][3] = v.w;
                    }
                    else
#pragma unroll
                        for(int e = 0; e < 4; ++e)
                            qb[blk][e] = static_cast<uint32_t>(__half_as_ushort(src[2 * e])) |
                                         (static_cast<uint32_t>(__half_as_ushort(src[2 * e + 1])) << 16);
                }
            }
            // ---- scores of this CTA's positions, cut to half after the dot and after the scaling
            float mx[2] = {-INFINITY, -INFINITY}; // heads 2 t, 2 t + 1
            for(int grp = warp; grp < tiles * (GD_TILE / 16); grp += GD_WARPS)
            {
                const int tile    = grp / (GD_TILE / 16);
                const uint8_t* kt = wait_tile(tile0 + tile);
                const int r0      = grp % (GD_TILE / 16) * 16 + prow;
                if(grp * 16 >= n)
                {
                    release_tile(tile0 + tile);
                    continue;
                }
                // a sum of its own per block of 32, added in fp32: the tensor core's running sum loses a little
                // at every step, and the score is cut to half next.  (Of the results 0.4 to 2.8 % are not the half
                // that the chain with 64-bit dots gives, over 14 shapes of 200 to 4096 positions; with scalar fp32
                // sums 0.5 to 3.8 %.)
                float cb[NB][4];
#pragma unroll
                for(int blk = 0; blk < NB; ++blk)
                {
                    const uint8_t* at = kt + (blk / 2) * GD_TILE * 128 + r0 * 128 + ((((blk & 1) * 4 + t) ^ prow) << 4);
                    const uint4 lo = *reinterpret_cast<const uint4*>(at), hi = *reinterpret_cast<const uint4*>(at + 1024);
                    cb[blk][0] = cb[blk][1] = cb[blk][2] = cb[blk][3] = 0.0f;
                    gd_mma(cb[blk], lo.x, hi.x, lo.y, hi.y, qb[blk][0], qb[blk][1]);
                    gd_mma(cb[blk], lo.z, hi.z, lo.w, hi.w, qb[blk][2], qb[blk][3]);
                }
                release_tile(tile0 + tile);
                // element e: position prow + 8 (e >> 1) of the group, head 2 t + (e & 1)
#pragma unroll
                for(int e = 0; e < 4; ++e)
                {
                    float c = cb[0][e] + cb[1][e];
                    if constexpr(NB == 4)
                        c += cb[2][e] + cb[3][e];
                    const int h = 2 * t + (e & 1), j = grp * 16 + prow + 8 * (e >> 1);
                    if(h < p.fact and j < n)
                    {
                        float sv = truncate_to_half_precision(c);
                        sv       = truncate_to_half_precision(__fmul_rn(sv, p.scale));
                        mx[e & 1]          = fmaxf(mx[e & 1], sv);
                        sc[h * p.pitch + j] = __float2half_rz(sv);
                    }
                }
            }
#pragma unroll
            for(int e = 0; e < 2; ++e)
            {
#pragma unroll
                for(int o = 4; o < 32; o <<= 1)
                    mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], o));
                if(g == 0)
                    wred[warp][2 * t + e] = mx[e];
            }
            gd_consumer_barrier();
            if(tid < GD_HEADS)
            {
                float m = wred[0][tid];
#pragma unroll
                for(int w = 1; w < GD_WARPS; ++w)
                    m = fmaxf(m, wred[w][tid]);
                red_m[tid] = m;
            }
            exchange();
            if(p.split > 1)
            {
                if(tid < GD_HEADS)
                    tot_m[tid] = of_cluster(red_m + tid, true);
                gd_consumer_barrier();
            }
            const float* gmax = p.split > 1 ? tot_m : red_m;
            // ---- e = half(exp(x - max)) in place, the sum over the stored halves in fp32; 8 / fact warps a head
            {
                const int parts = GD_WARPS / p.fact, h = warp / parts;
                const float gm  = gmax[h];
                float s         = 0.0f;
                for(int j = (warp - h * parts) * 32 + lane; j < n; j += 32 * parts)
                {
                    const float x = __half2float(sc[h * p.pitch + j]);
                    const float e = gd_trunc_nonneg(gd_exp2((x - gm) * log2e));
                    sc[h * p.pitch + j] = __float2half_rz(e);
                    s += e;
                }
#pragma unroll
                for(int o = 16; o > 0; o >>= 1)
                    s += __shfl_xor_sync(0xffffffffu, s, o);
                if(lane == 0)
                    wred[warp][0] = s; // (the maxima in wred were read before the exchange)
            }
            gd_consumer_barrier();
            if(tid < p.fact)
            {
                const int parts = GD_WARPS / p.fact;
                float s         = 0.0f;
                for(int w = 0; w < parts; ++w)
                    s += wred[tid * parts + w][0];
                red_s[tid] = s;
            }
            exchange();
            if(p.split > 1)
            {
                if(tid < p.fact)
                    tot_s[tid] = of_cluster(red_s + tid, false);
                gd_consumer_barrier();
            }
            // ---- partial P V: p = half(e / sum) where it is used (one reciprocal per head, the quotient
            // corrected once with its remainder: P. Markstein's theorem)
            const float total = g < p.fact ? (p.split > 1 ? tot_s : red_s)[g] : 1.0f;
            const float rcp   = __frcp_rn(total);
            float o[D / 16][4];
#pragma unroll
            for(int i = 0; i < D / 16; ++i)
                o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
            for(int grp = warp; grp < tiles * (GD_TILE / 16); grp += GD_WARPS)
            {
                const int tile = grp / (GD_TILE / 16), j0 = grp * 16;
                if(j0 >= n)
                {
                    wait_tile(tile0 + tiles + tile);
                    release_tile(tile0 + tiles + tile);
                    continue;
                }
                // probabilities of positions 2 t, 2 t + 1 and 8 + 2 t, 9 + 2 t for head g
                uint32_t pb[2] = {0u, 0u};
                if(g < p.fact)
                {
#pragma unroll
                    for(int i = 0; i < 2; ++i)
                    {
                        const int j      = j0 + 8 * i + 2 * t;
                        const uint32_t w = *reinterpret_cast<const uint32_t*>(sc + g * p.pitch + j);
                        const float2 e2  = __half22float2(*reinterpret_cast<const __half2*>(&w));
                        float a0 = e2.x * rcp, a1 = e2.y * rcp;
                        a0 = __fmaf_rn(__fmaf_rn(-a0, total, e2.x), rcp, a0);
                        a1 = __fmaf_rn(__fmaf_rn(-a1, total, e2.y), rcp, a1);
                        pb[i] = cvt_rz_f16x2(j < n ? a0 : 0.0f, j + 1 < n ? a1 : 0.0f);
                    }
                }
                const uint8_t* vt = wait_tile(tile0 + tiles + tile);
                // ldmatrix addresses: matrix m = lane / 8 holds positions 8 (m >> 1) .. + 7, columns 8 (m & 1) .. + 7
                const int r         = grp % (GD_TILE / 16) * 16 + (lane >> 4) * 8 + (lane & 7);
                const uint32_t vrow = smem_u32(vt) + r * 128;
                // positions past the end hold anything, not-a-numbers included: cleared in the fragments
                const uint32_t m0 = (j0 + 2 * t < n ? 0x0000FFFFu : 0u) | (j0 + 2 * t + 1 < n ? 0xFFFF0000u : 0u);
                const uint32_t m1 = (j0 + 8 + 2 * t < n ? 0x0000FFFFu : 0u) | (j0 + 9 + 2 * t < n ? 0xFFFF0000u : 0u);
#pragma unroll
                for(int i = 0; i < D / 16; ++i)
                {
                    uint32_t a[4];
                    const int chunk = (i & 3) * 2 + ((lane >> 3) & 1);
                    gd_ldmatrix_trans(a, vrow + (i / 4) * GD_TILE * 128 + ((chunk ^ (lane & 7)) << 4));
                    gd_mma(o[i], a[0] & m0, a[1] & m0, a[2] & m1, a[3] & m1, pb[0], pb[1]);
                }
                release_tile(tile0 + tiles + tile);
            }
            tile0 += 2 * tiles;
            gd_consumer_barrier(); // every warp is done with the exponentials: their place takes the partials
            // o[i][e]: column 16 i + g + 8 (e >> 1), head 2 t + (e & 1)
#pragma unroll
            for(int i = 0; i < D / 16; ++i)
#pragma unroll
                for(int e = 0; e < 4; ++e)
                    if(2 * t + (e & 1) < p.fact)
                        part[(warp * p.fact + 2 * t + (e & 1)) * D + 16 * i + g + 8 * (e >> 1)] = o[i][e];
            gd_consumer_barrier();
            __half* dst = p.out + (static_cast<int64_t>(b) * p.kv_heads * p.fact + h0) * D;
            for(int i = tid; i < p.fact * D; i += GD_THREADS)
            {
                float s = 0.0f;
#pragma unroll
                for(int w = 0; w < GD_WARPS; ++w)
                    s += part[w * p.fact * D + i];
                if(p.split > 1)
                    cta_out[i] = s;
                else
                    dst[i] = __float2half_rz(s);
            }
            // (cta_out is written again two exchanges later, red_m and red_s three)
            exchange();
            if(p.split > 1)
                for(int i = tid + rank * GD_THREADS; i < p.fact * D; i += p.split * GD_THREADS)
                    dst[i] = __float2half_rz(of_cluster(cta_out + i, false));
        }
    }
    // ---------------------------------------------------------- teardown
    if(*abort_flag != 0)
        for(int i = 0; i < 1000; ++i)
            __nanosleep(1000); // copies in flight land before shared memory is released
    if(p.split > 1)
        cluster_barrier(); // no CTA leaves while another may read its shared memory
}

// ------------------------------------------------------------------ host
namespace {

// dynamic shared memory of a CTA when `resident` of them share an SM (beside the static arrays)
constexpr size_t smem_max(int resident) { return (resident == 1 ? 220 : 106) * 1024 + 128; }

// Bytes of the score / partial-result region for a share of `cap` positions (a multiple of 16).  The heads' rows are
// cap + 8 halves apart: an odd multiple of 16 bytes, so that eight heads' words lie in different banks.
size_t region_bytes(int64_t fact, int64_t head, int64_t cap)
{
    return std::max<size_t>(sizeof(__half) * fact * (cap + 8), sizeof(float) * GD_WARPS * fact * head);
}

int64_t share_cap(int64_t cache_seq, int split) { return (ceil_div(cache_seq, split) + 15) / 16 * 16; }

bool share_fits(int64_t fact, int64_t head, int64_t cap, int resident)
{
    return region_bytes(fact, head, cap) + (resident == 1 ? 1 : 4) * GD_TILE * head * 2 + 1024 <= smem_max(resident);
}

template <int D>
void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, size_t smem, cudaStream_t stream)
{
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(GD_THREADS + 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = stream;
    attr[0].id               = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs    = attr;
    cfg.numAttrs = 2;
}

// Clusters of `split` CTAs that fit the device at once, `resident` CTAs to an SM.
template <int D>
int max_clusters(int split, int resident)
{
    static std::mutex m;
    static int cached[64][2][4] = {};
    int dev                     = 0;
    if(split == 1)
        return device_sm_count() * resident;
    if(cudaGetDevice(&dev) != cudaSuccess or dev < 0 or dev >= 64)
        return device_sm_count() / (2 * split);
    std::lock_guard<std::mutex> lock(m);
    int& n = cached[dev][resident - 1][split == 2 ? 1 : (split == 4 ? 2 : 3)];
    if(n == 0)
    {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        configure<D>(cfg, attr, device_sm_count() * resident / split, split, smem_max(resident), nullptr);
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, gqa_decode_kernel<D>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

template <int D>
int launch_gqa_decode(gqa_decode_params p, const void* k_cache, const void* v_cache, cudaStream_t stream)
{
    const int rc = ensure_smem_optin(reinterpret_cast<const void*>(gqa_decode_kernel<D>), smem_max(1));
    if(rc != MGX_OK)
        return rc;
    // One CTA per SM or two, and the split of a job's positions over a cluster, with the smallest estimated
    // time.  Jobs go round the clusters.  A share streams at 44 bytes per ns with the SM to itself and
    // keeps its CTA in barriers and exchanges for about 6 us, which a second CTA of the SM fills.
    // Measured, 512 jobs of 1024 - 2047 positions, 128 wide (403 MB): two per SM, whole jobs 72 us,
    // half jobs 81; one per SM, whole jobs 93, half jobs 109.  32 such jobs: two per SM, eighths 11.9 us,
    // one per SM, quarters 12.4.
    double best  = 0.0;
    int clusters = 0, per_sm = 1;
    for(int resident : {1, 2})
        for(int split : {1, 2, 4, 8})
        {
            const int64_t cap = share_cap(p.cache_seq, split);
            if(not share_fits(p.fact, D, cap, resident) or (split > 1 and cap < GD_TILE))
                continue;
            const int c     = std::min(max_clusters<D>(split, resident), p.jobs);
            const double s  = cap * (D * 4) / 44.0;
            const double ns = static_cast<double>(ceil_div(p.jobs, c)) * (resident == 1 ? s + 6000.0 : std::max(2.0 * s, s + 6000.0));
            if(best == 0.0 or ns < best)
                best = ns, p.split = split, clusters = c, p.cap = static_cast<int>(cap), per_sm = resident;
        }
    if(best == 0.0)
        return MGX_E_TOO_LARGE;
    const size_t region = region_bytes(p.fact, D, p.cap);
    p.pitch             = p.cap + 8;
    p.stages = static_cast<int>(std::min<size_t>(GD_MAX_STAGES, (smem_max(per_sm) - 1024 - region) / (GD_TILE * D * 2)));
    CUtensorMap tk, tv;
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[3]    = {D, static_cast<cuuint64_t>(p.cache_seq), static_cast<cuuint64_t>(p.jobs)};
    cuuint64_t strides[2] = {D * 2, static_cast<cuuint64_t>(p.cache_seq) * D * 2};
    cuuint32_t box[3]     = {64u, GD_TILE, 1u};
    cuuint32_t estr[3]    = {1u, 1u, 1u};
    for(auto [map, base] : {std::pair(&tk, k_cache), std::pair(&tv, v_cache)})
        if(encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return MGX_E_INVALID_ARG;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure<D>(cfg, attr, clusters, p.split, 1024 + region + p.stages * (GD_TILE * D * 2), stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, gqa_decode_kernel<D>, tk, tv, p));
}

} // namespace

int gqa_decode_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx

extern "C" int mgx_cuda_gqa_decode_supported(int64_t batch, int64_t heads, int64_t kv_heads, int64_t head,
                                             int64_t cache_seq)
{
    using namespace mgx;
    if(batch <= 0 or heads <= 0 or kv_heads <= 0 or cache_seq <= 0 or heads % kv_heads != 0)
        return 0;
    const int64_t fact = heads / kv_heads;
    if((head != 64 and head != 128) or (fact != 1 and fact != 2 and fact != 4 and fact != 8))
        return 0;
    if(batch > 65535 or kv_heads > 65535 or batch * kv_heads > (int64_t{1} << 30) or cache_seq > (int64_t{1} << 30))
        return 0;
    return share_fits(fact, head, share_cap(cache_seq, 8), 1) ? 1 : 0;
}

extern "C" int mgx_cuda_gqa_decode_attention(const mgx_gqa_decode_desc* d, const void* q, const void* k_cache,
                                             const void* v_cache, const void* seqlens, void* out, void* stream_)
{
    using namespace mgx;
    if(d == nullptr or q == nullptr or k_cache == nullptr or v_cache == nullptr or seqlens == nullptr or out == nullptr)
        return MGX_E_INVALID_ARG;
    if(d->batch <= 0 or d->heads <= 0 or d->kv_heads <= 0 or d->cache_seq <= 0 or d->heads % d->kv_heads != 0)
        return MGX_E_INVALID_ARG;
    if(d->seqlens_type != MGX_I32 and d->seqlens_type != MGX_I64)
        return MGX_E_UNSUPPORTED;
    if(d->head != 64 and d->head != 128)
        return MGX_E_UNSUPPORTED;
    const int64_t fact = d->heads / d->kv_heads;
    if(fact != 1 and fact != 2 and fact != 4 and fact != 8)
        return MGX_E_UNSUPPORTED;
    if(d->batch > 65535 or d->kv_heads > 65535 or d->batch * d->kv_heads > (int64_t{1} << 30) or d->cache_seq > (int64_t{1} << 30))
        return MGX_E_TOO_LARGE;
    // rows are read as 16-byte vectors
    if((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) % 16 != 0 or
       reinterpret_cast<uintptr_t>(q) % 2 != 0 or reinterpret_cast<uintptr_t>(out) % 2 != 0)
        return MGX_E_ALIGNMENT;
    gqa_decode_params p{};
    p.q    = static_cast<const __half*>(q);
    p.q_sb = d->q_batch_stride, p.q_sh = d->q_head_stride;
    p.q_vec = reinterpret_cast<uintptr_t>(q) % 16 == 0 and d->q_batch_stride % 8 == 0 and d->q_head_stride % 8 == 0 ? 1 : 0;
    p.seqlens     = seqlens;
    p.seqlens_i64 = d->seqlens_type == MGX_I64 ? 1 : 0;
    p.out         = static_cast<__half*>(out);
    p.scale       = d->scale;
    p.cache_seq   = static_cast<int>(d->cache_seq);
    p.kv_heads    = static_cast<int>(d->kv_heads);
    p.fact        = static_cast<int>(fact);
    p.jobs        = static_cast<int>(d->batch * d->kv_heads);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    return d->head == 128 ? launch_gqa_decode<128>(p, k_cache, v_cache, stream)
                          : launch_gqa_decode<64>(p, k_cache, v_cache, stream);
}
