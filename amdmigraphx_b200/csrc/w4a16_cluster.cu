// Weight-only int4 linear for decode (M <= 16 rows of activations) on the tcgen05 tensor core,
// built to be bound by the HBM stream of packed weights:
//
//   D[m,n] = sum_g  s[n,g] * sum_{k in g} (q[n,k] - zp[n,g]) * a[m,k]
//
// is evaluated with INTEGER tensor-core arithmetic.  A small pre-kernel writes every
// activation row as int8 rows (a ~ sa[g,m] * (128 h + l), |error| <= sa/2, i.e. 15 bits of the
// range of the row's own group g of 128 k: an outlier costs only the 127 other values of its
// group precision, not the whole row) and the per-group sums Sv[g,m] = sum_k (128 h + l).  The main kernel computes,
// per group g of 128 k and per 128 output columns, with kind::i8 MMAs whose A operand are the
// UNSIGNED weights and whose B operand are the activation rows, exact int32 sums
// Q[n,m] = sum_k q[n,k] a_int[m,k] (spread over 2 or 4 accumulator columns per activation row,
// see RAW below), and the epilogue folds  s[n,g] * sa[g,m] * (Q - zp[n,g] * Sv[g,m])  into fp32
// registers.
// The only inexact steps are the 15-bit activation rounding and the fp32 sum over groups; the
// reference (src/onnx/parse_matmulnbits.cpp:85-158 IR on the ref target) rounds every
// dequantised weight to fp16 instead, which is the coarser of the two.
//
// CTA = 480 threads (608 with a second set of epilogue warps), one CTA per SM:
//   warp 0        TMA producer: per work item (4 groups) two requests of 128 rows x 128 bytes of
//                 packed weights and one of the activation rows of the same groups
//   warps 2..5    unpack: one thread per weight row, shared memory -> registers -> the row's lane
//                 of TENSOR MEMORY (tcgen05.st); the MMA reads its A operand from there, so the
//                 unpacked bytes never cross shared memory
//   warps 1, 10..12  MMA issuers: group i of every work item
//   warps 13, 14  cp.async copies of the epilogue's scales / zero points / group sums, up to
//                 three passes ahead
//   warps 6..9 (and 15..18)  epilogue fold out of two accumulator buffers; the partial sums of a
//                 tile are added through distributed shared memory in rank order, an exchange being
//                 waited for only at the next one
// Work: a cluster of S CTAs takes tiles of 128 output columns in turn, CTA r of it the r-th share of K,
// whose activation planes stay in its shared memory for the whole kernel.  What surrounds the stream of a
// smaller matrix bounds it: with the items dealt out evenly (w4a16_tc.cu) tiles are completed through
// partial sums and counters in global memory and the planes are fetched again for every tile.  One row /
// 16 rows, that form and this: 4096 x 4096 7.2 -> 6.4 us / 10.7 -> 8.2; 4096 x 11008 13.6 -> 9.8 /
// 19.6 -> 17.0; 8192 x 1024 7.1 -> 4.4 / 8.8 -> 5.8; 7168 x 8192 11.8 -> 10.4 / 18.7 -> 17.1.
// Launches are chained programmatically: the main kernel streams weights while the pre-kernel still runs
// - and not while what precedes that does, which may be what writes them (the pre-kernel lets it start only
// after its own wait; with weights requested behind that kernel's back a decoder layer took 75.0 us, 76.5 so).
// Only plain TMA loads; every wait is bounded.
#include "common.cuh"
#include "ptx.cuh"
#include "w4a16_acts.cuh"
#include <algorithm>
#include <cuda_fp16.h>
#include <mutex>

namespace mgx {
namespace { // (names shared with w4a16_tc.cu)

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

constexpr int TC_MAX_SPLIT  = 8; // CTAs of a cluster; divides TC_ROWS
constexpr int TC_MAX_STAGES = 5;
constexpr int TC_XBUFS      = 3; // partial results of a tile: [buffer][row][column]
constexpr size_t TC_SMEM    = 226 * 1024;

// shared memory beside the ring of weights: planes of `items` work items, metadata, partial results
template <int NB>
constexpr size_t tc_fixed(int items, int rows)
{
    return static_cast<size_t>(items) * TC_SUPER * NB * TC_GROUP_K + 512 + TC_EPI + TC_XBUFS * rows * TC_ROWS * 4 + 1024;
}

struct tc_params
{
    const __half* scales;
    const uint8_t* zp; // may be null
    const float* sa;   // [K/128][MB] activation scale of every (group, row)
    const int* sv;     // [K/128][MB] per-group sums of the quantised activations
    __half* D;
    int64_t N, K, ldd;
    int M;
    int group, groups_per_row, zp_const;
    int tiles, clusters, split; // tiles of 128 columns; clusters; CTAs of a cluster
    int items, stages;          // most work items of a share of K; stages of the ring
};

// ------------------------------------------------------------------ main kernel
// A work item is TC_SUPER consecutive groups of a tile (the last of a tile may hold fewer): the walk over a
// CTA's tiles and, within each, its items lo .. hi - 1.
struct tc_walk
{
    int tile, sg, lo, hi, step, ntiles, G;
    __device__ tc_walk(int first, int tile_step, int tiles, int item_lo, int item_hi, int groups)
        : tile(first), sg(item_lo), lo(item_lo), hi(item_hi), step(tile_step), ntiles(tiles), G(groups)
    {
    }
    // next pass: at most `cap` (a multiple of TC_SUPER) groups of one tile
    __device__ bool next(int cap, int& tile_out, int& g0, int& count, bool& last)
    {
        if(tile >= ntiles or lo >= hi)
            return false;
        tile_out       = tile;
        g0             = sg * TC_SUPER;
        const int nblk = min(cap / TC_SUPER, hi - sg);
        count          = min(G, (sg + nblk) * TC_SUPER) - g0;
        sg += nblk;
        last = sg == hi;
        if(last)
        {
            sg = lo;
            tile += step;
        }
        return true;
    }
};

// MR: activation rows folded by the epilogue (M <= MR <= MB).
// RAW: the weight operand of a group is [64 bytes of low nibbles | the 64 packed bytes] and every
// activation row has 4 rows in the B operand (see the pre-kernel); otherwise it is the 128
// nibbles unpacked to bytes and 2 rows.  RAW costs one logic operation per eight weights
// instead of three, and twice the accumulator columns per activation row.
// ESETS: sets of four epilogue warps; with two, each set folds half of the MR rows (the second
// set is warps 15..18).
template <int NB, int MR, bool RAW, int ESETS>
__global__ void __launch_bounds__(TC_THREADS + (ESETS - 1) * 128, 1)
    w4a16_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w,
                    const __grid_constant__ CUtensorMap tmap_a,
                    const tc_params p)
{
    constexpr int CPM    = RAW ? 4 : 2;      // accumulator columns per activation row
    constexpr int MB     = NB / CPM;         // padded activation rows
    constexpr int GPP    = TC_ACC_COLS / NB; // groups per pass (one accumulator buffer): 8 or 4
    constexpr int XROWS  = MB;               // rows of a partial result
    constexpr int ABYTES = NB * TC_GROUP_K;  // activation rows of one group
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem           = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    const int WST           = p.stages;
    uint8_t* acts           = smem + WST * TC_WSTAGE; // planes of this CTA's share of K: [group][row][128 bytes]
    uint8_t* bar_base       = acts + p.items * TC_SUPER * ABYTES;
    uint64_t* full_bar      = reinterpret_cast<uint64_t*>(bar_base); // weights landed
    uint64_t* empty_bar     = full_bar + TC_MAX_STAGES;  // weights read by all rows
    uint64_t* unp_bar       = empty_bar + TC_MAX_STAGES; // A operand in tensor memory
    uint64_t* tfree_bar     = unp_bar + TC_TSTAGES; // MMAs that read it retired
    uint64_t* accf_bar      = tfree_bar + TC_TSTAGES;
    uint64_t* acce_bar      = accf_bar + 2;
    uint64_t* meta_bar      = acce_bar + 2;     // [3] epilogue metadata of a pass staged
    uint64_t* mfree_bar     = meta_bar + 3;     // [3] ... and folded
    uint64_t* acts_bar      = mfree_bar + 3;    // planes landed
    uint64_t* peer_bar      = acts_bar + 1;     // the whole cluster's partial results are in place
    uint32_t* tmem_slot     = reinterpret_cast<uint32_t*>(peer_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    // epilogue metadata, three buffers each: per output column the aligned 32-bit words that
    // hold the scales (at most 5) and zero points (at most 3) of a pass, GPP x MB activation
    // group sums and group scales
    uint32_t* epi_sw = reinterpret_cast<uint32_t*>(bar_base + 512);     // [3][128][5]
    uint32_t* epi_zw = epi_sw + 3 * 128 * 5;                            // [3][128][3]
    int* epi_sv      = reinterpret_cast<int*>(epi_zw + 3 * 128 * 3);    // [3][128]
    float* epi_sa    = reinterpret_cast<float*>(epi_sv + 3 * 128);      // [3][128]
    float* part      = reinterpret_cast<float*>(bar_base + 512 + TC_EPI); // [TC_XBUFS][XROWS][128]

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    // the next kernel of the stream may be started early if it asks for it (the pre-kernel of
    // the next linear does: it waits for this grid's completion before it reads or writes)
    grid_launch_dependents();
    if(threadIdx.x == 0)
    {
        for(int s = 0; s < WST; ++s)
        {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 128);
        }
        for(int b = 0; b < 2; ++b)
        {
            mbar_init(&unp_bar[b], 128);
            mbar_init(&tfree_bar[b], TC_ISSUERS);
            mbar_init(&accf_bar[b], TC_ISSUERS);
            mbar_init(&acce_bar[b], 4 * ESETS);
        }
        for(int b = 0; b < 3; ++b)
        {
            mbar_init(&meta_bar[b], 64);
            mbar_init(&mfree_bar[b], 4 * ESETS);
        }
        mbar_init(acts_bar, 1);
        mbar_init(peer_bar, p.split);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_w);
        prefetch_tensormap(&tmap_a);
    }
    if(warp == 1)
    {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if(p.split > 1)
        cluster_barrier(); // the other CTAs' barriers exist before anyone arrives on them
    const int G       = static_cast<int>(p.K / TC_GROUP_K);
    const int SG      = (G + TC_SUPER - 1) / TC_SUPER;
    const int rank    = static_cast<int>(blockIdx.x) % p.split;
    const int cluster = static_cast<int>(blockIdx.x) / p.split;
    const int sg_lo   = SG * rank / p.split; // this CTA's items of every tile
    const int sg_hi   = SG * (rank + 1) / p.split;
    const int nsuper  = (sg_hi - sg_lo) * ((p.tiles - cluster + p.clusters - 1) / p.clusters);
    const tc_walk walk0(cluster, p.clusters, p.tiles, sg_lo, sg_hi, G);
    // MMA issuers: warps 1, 10, 11, 12 -> group 0..3 of every work item
    const int issuer = warp == 1 ? 0 : (warp >= 10 and warp <= 12 ? warp - 9 : -1);

    if(warp == 0)
    {
        // ---------------------------------------------------- TMA producer
        // A stage = 4 groups of packed weights (two requests of 128 rows x 128 bytes).  The weights
        // are requested at once: whatever wrote them is complete, the pre-kernel having waited for it
        // before it let this kernel start.  The activation planes are written by the pre-kernel, whose
        // completion is awaited before they are requested.
        int tile = cluster, sg = sg_lo;
        const int head = min(nsuper, WST);
        int s = 0;
        uint32_t ph = 1;
        for(int j = 0; j < nsuper; ++j)
        {
            if(not mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2))
                break;
            if(elect_one())
            {
                uint8_t* st = smem + s * TC_WSTAGE;
                // groups past the end of K are zero-filled and still counted
                mbar_expect_tx(&full_bar[s], TC_WSTAGE);
                tma_load_2d(st, &tmap_w, &full_bar[s], sg * (TC_WSTAGE / TC_ROWS), tile * TC_ROWS);
                tma_load_2d(st + TC_WSTAGE / 2, &tmap_w, &full_bar[s],
                            sg * (TC_WSTAGE / TC_ROWS) + 128, tile * TC_ROWS);
            }
            if(++s == WST)
                s = 0, ph ^= 1u;
            if(++sg == sg_hi)
            {
                sg = sg_lo;
                tile += p.clusters;
            }
            if(j == head - 1)
            {
                grid_dependency_wait();
                if(elect_one())
                {
                    mbar_expect_tx(acts_bar, static_cast<uint32_t>((sg_hi - sg_lo) * TC_SUPER * ABYTES));
                    for(int i = sg_lo; i < sg_hi; ++i)
                        tma_load_3d(acts + (i - sg_lo) * TC_SUPER * ABYTES, &tmap_a, acts_bar, 0, 0, i * TC_SUPER);
                }
            }
        }
    }
    else if(issuer >= 0)
    {
        // ---------------------------------------------------- MMA issuers
        // Each of four warps issues the four k-steps of "its" group of every work item.
        // D s32 += A u8 (weights, tensor memory) * B s8 (activation rows, K-major shared
        // memory); M = 128, N = NB
        constexpr uint32_t idesc = make_idesc(2u, 0u, 1u, TC_ROWS, NB);
        const uint64_t bdesc0    = make_smem_desc_sw128(smem_u32(acts + issuer * ABYTES));
        tc_walk walk             = walk0;
        int tile, g0, count;
        bool seg_last;
        bool ok    = true;
        int j      = 0;
        // the activation planes come from the previous kernel of the stream: the bounded
        // waits below must not count its run time
        grid_dependency_wait();
        if(nsuper > 0)
            ok = mbar_wait_warp(acts_bar, 0u, abort_flag, 7);
        for(uint32_t pc = 0; ok and walk.next(GPP, tile, g0, count, seg_last); ++pc)
        {
            const uint32_t buf = pc & 1u;
            if(not mbar_wait_warp(&acce_bar[buf], ((pc >> 1) & 1u) ^ 1u, abort_flag, 4))
                break;
            tc_fence_after_sync();
            for(int gl = 0; gl < count; gl += TC_SUPER, ++j)
            {
                const uint32_t t  = j & 1u;
                const uint32_t tp = (j >> 1) & 1u;
                // implies that the stage's TMA requests have landed
                if(not mbar_wait_warp(&unp_bar[t], tp, abort_flag, 5))
                {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if(elect_one())
                {
                    if(gl + issuer < count)
                    {
                        const uint64_t bdesc  = bdesc0 + static_cast<uint64_t>(((g0 + gl - sg_lo * TC_SUPER) * ABYTES) >> 4);
                        const uint32_t a_tmem = tmem_base + TC_A_COL0 + (t * TC_SUPER + issuer) * TC_A_COLS;
                        const uint32_t d_tmem = tmem_base + buf * TC_ACC_COLS + (gl + issuer) * NB;
#pragma unroll
                        for(int k = 0; k < 4; ++k)
                            mma_i8_tmem_a(d_tmem, a_tmem + k * 8,
                                          bdesc + static_cast<uint64_t>((k * 32) >> 4), idesc, k != 0);
                    }
                    tc_commit(&tfree_bar[t]);
                    if(gl + TC_SUPER >= count)
                        tc_commit(&accf_bar[buf]);
                }
            }
        }
    }
    else if(warp == 13 or warp == 14)
    {
        // ---------------------------------------------------- epilogue metadata, up to 3 passes ahead
        // cp.async copies of the aligned words around the scales and zero points of a pass
        // (consecutive lanes copy consecutive words of a column's run, so a request touches
        // few sectors) and of the activation group sums.  Each of the two warps serves 64
        // output columns.
        grid_dependency_wait(); // sv and sa come from the pre-kernel
        const int half  = warp - 13;
        const int rshift = 31 - __clz(p.group / TC_GROUP_K); // groups are powers of two
        const uint32_t sbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.scales) & 3u);
        const uint32_t zbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.zp) & 3u);
        const char* sptr = reinterpret_cast<const char*>(p.scales) - sbase0; // 4-byte aligned
        const char* zptr = reinterpret_cast<const char*>(p.zp) - zbase0;
        auto cp_async4 = [](const void* dst, const void* src) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src)
                         : "memory");
        };
        tc_walk walk = walk0;
        int tile, g0, count;
        bool seg_last;
        for(uint32_t pc = 0; walk.next(GPP, tile, g0, count, seg_last); ++pc)
        {
            const uint32_t vb = pc % 3u;
            if(not mbar_wait_bounded(&mfree_bar[vb], ((pc / 3u) & 1u) ^ 1u, abort_flag, 9))
                break;
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
                    cp_async4(epi_sw + (vb * 128 + half * 64 + r) * 5 + w, sptr + a + 4 * w);
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
                        cp_async4(epi_zw + (vb * 128 + half * 64 + r) * 3 + w, zptr + a + 4 * w);
                }
            }
            // group sums and group scales: count x MB words each, half of them per warp
            for(int i = half * 64 + lane; i < count * MB; i += 32)
                if(i < half * 64 + 64)
                {
                    cp_async4(epi_sv + vb * 128 + i, p.sv + static_cast<int64_t>(g0) * MB + i);
                    cp_async4(epi_sa + vb * 128 + i, p.sa + static_cast<int64_t>(g0) * MB + i);
                }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(
                             smem_u32(&meta_bar[vb]))
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    else if(warp < 6)
    {
        // ---------------------------------------------------- unpack: nibbles -> bytes
        // One thread per weight row: 64 packed bytes per group from shared memory (128-byte
        // swizzle, so a quarter warp's 16-byte reads fall in eight different bank groups), 32
        // words to this row's lane of tensor memory: either the nibbles as bytes (inside every
        // 8 k the evens first, then the odds; the activation rows are stored in the same order)
        // or the low nibbles followed by the packed bytes as they are (RAW).
        const int row            = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const int sw             = row & 7;
        int sg                   = sg_lo;
        int s                    = 0;
        uint32_t ph              = 0;
        for(int j = 0; j < nsuper; ++j)
        {
            const uint32_t t  = j & 1u;
            const uint32_t tp = (j >> 1) & 1u;
            // the tensor-memory stores below are warp-wide: leave only as a whole warp
            if(not __all_sync(0xffffffffu, mbar_wait_bounded(&full_bar[s], ph, abort_flag, 1)))
                break;
            if(not __all_sync(0xffffffffu, mbar_wait_bounded(&tfree_bar[t], tp ^ 1u, abort_flag, 8)))
                break;
            tc_fence_after_sync();
            const int cnt = min(TC_SUPER, G - sg * TC_SUPER);
#pragma unroll
            for(int q = 0; q < TC_SUPER; ++q)
            {
                if(q < cnt)
                {
                    // [pair of groups][row][128 bytes], 16-byte chunks swizzled by the row
                    const uint8_t* pk = smem + s * TC_WSTAGE + (q >> 1) * (2 * TC_PACKED) + row * 128;
                    uint32_t u[32];
#pragma unroll
                    for(int c = 0; c < 4; ++c)
                    {
                        const uint4 w =
                            *reinterpret_cast<const uint4*>(pk + ((((q & 1) * 4 + c) ^ sw) << 4));
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
                    tmem_st_32x32b_x32(tmem_base + lane_addr + TC_A_COL0 +
                                           (t * TC_SUPER + q) * TC_A_COLS,
                                       u);
                }
            }
            mbar_arrive(&empty_bar[s]); // the packed blocks are in registers
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&unp_bar[t]);
            if(++s == WST)
                s = 0, ph ^= 1u;
            if(++sg == sg_hi)
                sg = sg_lo;
        }
    }
    else
    {
        // ---------------------------------------------------- epilogue: fold the groups
        // Scale, zero point and activation group sums of a pass are already in shared memory
        // (metadata warps).  Column 2 m of a group's accumulator is P_hi, column 2 m + 1 P_lo
        // of activation row m; only the MR rows in use are read.  All arithmetic stays off
        // the conversion pipe except one half -> float per group: |P_hi|, |P_lo| < 2^18.
        grid_dependency_wait(); // sa comes from the pre-kernel, D may still be read by an earlier one
        constexpr int MRW = MR / ESETS;          // rows this warp folds ...
        const int eset    = warp >= 15 ? 1 : 0;
        const int m0      = eset * MRW;          // ... starting at this one
        const int quarter = warp & 3;
        const int col     = quarter * 32 + lane; // output column inside the tile = TMEM lane
        const int rshift  = 31 - __clz(p.group / TC_GROUP_K); // groups are powers of two
        const uint32_t sbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.scales) & 3u);
        const uint32_t zbase0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p.zp) & 3u);
        float out[MRW];
#pragma unroll
        for(int m = 0; m < MRW; ++m)
            out[m] = 0.0f;
        tc_walk walk = walk0;
        // one group: out[m] += sc sa[m] (Q[m] - z Sv[m]) with Q = sum_k q a_int, in exact integer
        // arithmetic up to the one conversion.  soff / zoff: byte offset of the group's scale /
        // zero point inside this column's staged words
        constexpr int C  = CPM * MRW; // accumulator columns read per group
        const bool has_zp = p.zp != nullptr;
        auto fold = [&](const uint32_t(&acc)[C], int gl, uint32_t vb, uint32_t soff, uint32_t zoff) {
            const uint32_t sw = epi_sw[(vb * 128 + col) * 5 + (soff >> 2)];
            const uint32_t sh = (soff & 2u) ? sw >> 16 : sw & 0xFFFFu;
            float sc          = __half2float(__ushort_as_half(static_cast<unsigned short>(sh)));
            // without zero points the staged word is not meaningful and not used
            const uint32_t zw = epi_zw[(vb * 128 + col) * 3 + (has_zp ? zoff >> 2 : 0u)];
            int z = has_zp ? static_cast<int>((zw >> (8u * (zoff & 3u))) & 0xFFu) : p.zp_const;
            if constexpr(RAW)
            {
                sc *= 0.0625f; // Q is computed times 16
                z *= 16;
            }
            const int* svb   = epi_sv + vb * 128 + gl * MB + m0;
            const float* sab = epi_sa + vb * 128 + gl * MB + m0;
#pragma unroll
            for(int m = 0; m < MRW; ++m)
            {
                int q;
                if constexpr(RAW)
                {
                    // columns: sum L e_h, 16 sum q_odd o_h, sum L e_l, 16 sum q_odd o_l;
                    // 16 Q = 2048 E_h + 128 O_h + 16 E_l + O_l
                    q = static_cast<int>(acc[4 * m]) * 2048 + static_cast<int>(acc[4 * m + 3]);
                    q = static_cast<int>(acc[4 * m + 1]) * 128 + q;
                    q = static_cast<int>(acc[4 * m + 2]) * 16 + q;
                }
                else
                    q = static_cast<int>(acc[2 * m]) * 128 + static_cast<int>(acc[2 * m + 1]);
                q      = q - z * svb[m];
                out[m] = fmaf(sc * sab[m], static_cast<float>(q), out[m]);
            }
        };
        // groups read from tensor memory per trip (all loads in flight before the first fold)
        constexpr int TR = C <= 4 ? 8 : (C <= 8 ? 4 : 2);
        constexpr int ETHREADS = 128 * ESETS;
        const int et           = (eset == 1 ? warp - 15 : warp - 6) * 32 + lane + eset * 128;
        bool dead              = false; // a wait gave up: go on without waiting, the barriers need every thread
        // tile number x of this cluster: the sum over its CTAs, each a share of the columns, is written to D
        auto finish = [&](int x) {
            if(not dead and not __all_sync(0xffffffffu, mbar_wait_cluster_bounded(peer_bar, x & 1, abort_flag, 6)))
                dead = true;
            const float* from = part + (x % TC_XBUFS) * XROWS * TC_ROWS;
            const int share   = TC_ROWS / p.split;
            const int c       = rank * share + et % share;
            const int64_t nc  = static_cast<int64_t>(cluster + x * p.clusters) * TC_ROWS + c;
            if(nc < p.N and not dead)
                for(int m = et / share; m < p.M; m += ETHREADS / share)
                {
                    float v[TC_MAX_SPLIT], sum = 0.0f;
#pragma unroll
                    for(int r = 0; r < TC_MAX_SPLIT; ++r)
                        v[r] = r < p.split ? __uint_as_float(cluster_load(from + m * TC_ROWS + c, r)) : 0.0f;
#pragma unroll
                    for(int r = 0; r < TC_MAX_SPLIT; ++r)
                        sum += v[r];
                    p.D[m * p.ldd + nc] = __float2half_rn(sum);
                }
        };
        int done = 0; // tiles exchanged so far
        int tile, g0, count;
        bool seg_last;
        for(uint32_t pc = 0; walk.next(GPP, tile, g0, count, seg_last); ++pc)
        {
            const uint32_t buf = pc & 1u;
            const uint32_t vb  = pc % 3u;
            if(not dead and (not mbar_wait_warp(&meta_bar[vb], (pc / 3u) & 1u, abort_flag, 10) or
                             not mbar_wait_warp(&accf_bar[buf], (pc >> 1) & 1u, abort_flag, 3)))
                dead = true;
            tc_fence_after_sync();
            const int gi0 = g0 >> rshift;
            const int n   = min(tile * TC_ROWS + col, static_cast<int>(p.N) - 1);
            const uint32_t sbyte =
                (sbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0) * 2u) & 3u;
            const uint32_t zbyte = (zbase0 + static_cast<uint32_t>(n * p.groups_per_row + gi0)) & 3u;
            // quantisation group of group gl, relative to gi0
            auto grel = [&](int gl) { return static_cast<uint32_t>(((g0 + gl) >> rshift) - gi0); };
            const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   buf * TC_ACC_COLS + CPM * m0;
#pragma unroll 1
            for(int gl = 0; gl < count; gl += TR)
            {
                uint32_t acc[TR][C];
                if(gl + TR <= count)
                {
                    // full trip: straight-line code, the folds interleave
#pragma unroll
                    for(int t = 0; t < TR; ++t)
                        tmem_ld_32x32b<C>(tbase + (gl + t) * NB, acc[t]);
                    tmem_ld_wait();
#pragma unroll
                    for(int t = 0; t < TR; ++t)
                        fold(acc[t], gl + t, vb, sbyte + 2u * grel(gl + t), zbyte + grel(gl + t));
                }
                else
                {
#pragma unroll
                    for(int t = 0; t < TR; ++t)
                        if(gl + t < count) // the same for the whole warp
                            tmem_ld_32x32b<C>(tbase + (gl + t) * NB, acc[t]);
                    tmem_ld_wait();
#pragma unroll
                    for(int t = 0; t < TR; ++t)
                        if(gl + t < count)
                            fold(acc[t], gl + t, vb, sbyte + 2u * grel(gl + t), zbyte + grel(gl + t));
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if(lane == 0)
            {
                mbar_arrive(&acce_bar[buf]);
                mbar_arrive(&mfree_bar[vb]);
            }
            if(seg_last)
            {
                // this CTA's share of the tile is complete
                const int64_t nc = static_cast<int64_t>(tile) * TC_ROWS + col;
                if(p.split == 1)
                {
#pragma unroll
                    for(int m = 0; m < MRW; ++m)
                        if(m0 + m < p.M and nc < p.N and not dead)
                            p.D[(m0 + m) * p.ldd + nc] = __float2half_rn(out[m]);
                }
                else
                {
                    // announced here, summed at the next tile.  The buffer is written again three tiles
                    // later, after this CTA has seen all of the next tile announced, which every CTA does
                    // only when it has read this one.
#pragma unroll
                    for(int m = 0; m < MRW; ++m)
                        part[((done % TC_XBUFS) * XROWS + m0 + m) * TC_ROWS + col] = out[m];
                    if(done > 0)
                        finish(done - 1);
                    asm volatile("bar.sync 1, %0;" ::"n"(ETHREADS) : "memory");
                    if(et < p.split)
                        cluster_arrive(peer_bar, et);
                    ++done;
                }
#pragma unroll
                for(int m = 0; m < MRW; ++m)
                    out[m] = 0.0f;
            }
        }
        if(done > 0)
            finish(done - 1);
    }

    // ---------------------------------------------------------- teardown
    if(*abort_flag != 0)
    {
        for(int i = 0; i < 1000; ++i)
            __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if(warp == 1)
    {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
    if(p.split > 1)
    {
        __syncwarp();
        cluster_barrier(); // no CTA leaves while another may read its partial results
    }
}

} // namespace

// ------------------------------------------------------------------ host
namespace {

struct tc_plan
{
    int nb, mb, tiles, groups, blocks;
    size_t off_sa, off_sv, total;
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

tc_plan make_plan(const mgx_w4_desc& d)
{
    tc_plan pl{};
    // up to 8 rows: 4 int8 rows per activation row (RAW operand); up to 16: 2 rows
    pl.nb     = d.M <= 4 ? 16 : 32;
    pl.mb     = d.M <= 4 ? 4 : (d.M <= 8 ? 8 : 16);
    pl.tiles  = static_cast<int>(ceil_div(d.N, TC_ROWS));
    pl.groups = static_cast<int>(d.K / TC_GROUP_K);
    pl.blocks = (pl.groups + TC_SUPER - 1) / TC_SUPER;
    pl.off_sa = align_up(static_cast<size_t>(pl.nb) * d.K, 256);
    pl.off_sv = align_up(pl.off_sa + static_cast<size_t>(pl.groups) * pl.mb * sizeof(float), 256);
    pl.total  = pl.off_sv + static_cast<size_t>(pl.groups) * pl.mb * sizeof(int);
    return pl;
}

// stages of the weight ring beside the planes of `items` work items
template <int NB>
int ring_stages(int items, int rows)
{
    const size_t fixed = tc_fixed<NB>(items, rows);
    return fixed >= TC_SMEM ? 0 : static_cast<int>(std::min<size_t>(TC_MAX_STAGES, (TC_SMEM - fixed) / TC_WSTAGE));
}

template <int ESETS>
void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, size_t smem, cudaStream_t stream)
{
    // programmatic dependent launch: the kernel may start while the pre-kernel still runs
    // and waits for it (griddepcontrol.wait) only where it reads what the pre-kernel wrote
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(TC_THREADS + (ESETS - 1) * 128);
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = stream;
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id               = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(split);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs    = attr;
    cfg.numAttrs = split > 1 ? 2 : 1;
}

// Clusters of `split` CTAs that fit the device at once, one CTA per SM (asked once per kernel and device).
template <int NB, int MR, bool RAW, int ESETS>
int max_clusters(int split)
{
    static std::mutex m;
    static int cached[64][TC_MAX_SPLIT + 1] = {};
    if(split == 1)
        return device_sm_count();
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess or dev < 0 or dev >= 64)
        return device_sm_count() / (2 * split);
    std::lock_guard<std::mutex> lock(m);
    int& n = cached[dev][split];
    if(n == 0)
    {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        configure<ESETS>(cfg, attr, device_sm_count() / split, split, TC_SMEM, nullptr);
        attr[0]      = attr[1];
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, w4a16_cluster_kernel<NB, MR, RAW, ESETS>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

template <int NB, int MR, bool RAW, int ESETS>
int launch_main(int blocks, const CUtensorMap& tw, const CUtensorMap& ta, tc_params p, cudaStream_t stream)
{
    constexpr int rows = NB / (RAW ? 4 : 2);
    int rc = ensure_smem_optin(reinterpret_cast<const void*>(w4a16_cluster_kernel<NB, MR, RAW, ESETS>), TC_SMEM);
    if(rc != MGX_OK)
        return rc;
    // The split of K with the smallest estimated time: a CTA takes 32 KB per item at its share of the HBM
    // stream (44 bytes per ns with all SMs at it, at most 100), at least 600 ns per item with fewer than
    // three stages in its ring; a tile costs a pass of the exchange, the last one 1 us.
    double best = 0.0;
    for(int split = 1; split <= TC_MAX_SPLIT and split <= blocks; split *= 2)
    {
        const int items  = static_cast<int>(ceil_div(blocks, split));
        const int stages = ring_stages<NB>(items, rows);
        if(stages < 2)
            continue;
        const int clusters = std::min(max_clusters<NB, MR, RAW, ESETS>(split), p.tiles);
        const int64_t mine = ceil_div(p.tiles, clusters);
        const double rate  = std::min(100.0, 6500.0 / (clusters * split));
        const double ns    = mine * items * std::max(TC_WSTAGE / rate, stages < 3 ? 1000.0 : 600.0) +
                          (split > 1 ? mine * 150.0 + 1000.0 : 0.0);
        if(best == 0.0 or ns < best)
            best = ns, p.split = split, p.clusters = clusters, p.items = items, p.stages = stages;
    }
    if(best == 0.0)
        return MGX_E_UNSUPPORTED; // (w4a16_tc_applicable says so beforehand)
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure<ESETS>(cfg, attr, p.clusters, p.split, tc_fixed<NB>(p.items, rows) + p.stages * TC_WSTAGE, stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, w4a16_cluster_kernel<NB, MR, RAW, ESETS>, tw, ta, p));
}

} // namespace

// Up to seven 32 KB work items per SM: there what surrounds the stream counts, beyond it the even dealing
// of items in w4a16_tc.cu is faster (one row: 12288 x 4096, 5.2 items, 8.7 us here and 10.4 there;
// 22016 x 4096, 9.3 items, 16.3 and 12.9).  An eighth of K's planes has to fit beside two stages of the ring.
bool w4a16_cluster_applicable(const mgx_w4_desc& d)
{
    const int64_t items = ceil_div(d.N, TC_ROWS) * ceil_div(d.K, TC_SUPER * TC_GROUP_K);
    return w4a16_tc_applicable(d) and items <= 7 * static_cast<int64_t>(device_sm_count()) and
           d.K <= (d.M <= 4 ? 65536 : 28672);
}

size_t w4a16_cluster_workspace(const mgx_w4_desc& d) { return make_plan(d).total; }

int w4a16_cluster_launch(const mgx_w4_desc& d, const void* A, const void* Bp, const void* scales,
                    const void* zp, void* D, void* workspace, size_t workspace_bytes,
                    cudaStream_t stream)
{
    const tc_plan pl = make_plan(d);
    if(workspace == nullptr or workspace_bytes < pl.total)
        return MGX_E_WORKSPACE;
    if((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0 or
       not w4a16_tc_pointers_ok(d, A, Bp, scales, zp))
        return MGX_E_ALIGNMENT;
    auto* ws       = static_cast<uint8_t*>(workspace);
    auto* aq       = reinterpret_cast<int8_t*>(ws);
    auto* sa       = reinterpret_cast<float*>(ws + pl.off_sa);
    auto* sv       = reinterpret_cast<int*>(ws + pl.off_sv);
    CUtensorMap tw, ta;
    // packed weights: rows of K / 2 bytes; one request = 128 rows x 128 bytes (two groups)
    int rc = MGX_OK;
    {
        cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
        if(encode == nullptr)
            return MGX_E_DRIVER;
        cuuint64_t dims[2]    = {static_cast<cuuint64_t>(d.K / 2), static_cast<cuuint64_t>(d.N)};
        cuuint64_t strides[1] = {static_cast<cuuint64_t>(d.K / 2)};
        cuuint32_t box[2]     = {128u, TC_ROWS};
        cuuint32_t estr[2]    = {1u, 1u};
        if(encode(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(Bp), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            rc = MGX_E_INVALID_ARG;
    }
    if(rc != MGX_OK)
        return rc;
    rc = encode_grouped(&ta, aq, TC_GROUP_K, static_cast<uint64_t>(pl.nb), static_cast<uint64_t>(d.K),
                        static_cast<uint64_t>(pl.groups), static_cast<uint32_t>(pl.nb), TC_SUPER,
                        CU_TENSOR_MAP_SWIZZLE_128B);
    if(rc != MGX_OK)
        return rc;
    rc = launch_prepare_acts(pl.mb, static_cast<const __half*>(A), d.lda, d.M, d.K, aq, sa, sv, nullptr, 0, stream);
    if(rc != MGX_OK)
        return rc;
    tc_params p{};
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
    p.tiles          = pl.tiles;
    if(d.M == 1)
        return launch_main<16, 1, true, 1>(pl.blocks, tw, ta, p, stream);
    if(d.M == 2)
        return launch_main<16, 2, true, 1>(pl.blocks, tw, ta, p, stream);
    if(d.M <= 4)
        return launch_main<16, 4, true, 1>(pl.blocks, tw, ta, p, stream);
    if(d.M <= 8)
        return launch_main<32, 8, true, 2>(pl.blocks, tw, ta, p, stream);
    return launch_main<32, 16, false, 2>(pl.blocks, tw, ta, p, stream);
}

int w4a16_cluster_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
