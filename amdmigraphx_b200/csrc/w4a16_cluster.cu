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
// The fp32 sum over groups is made per share and the shares are added: against 64-bit sums the relative error
// of a result is 1.6e-4 to 2.5e-4 (its rounding to half and the 15-bit activations), the same as with all groups
// in one sum to four digits, at 40 shapes of 1 to 16 rows, terms of both signs and of one.
// Launches are chained programmatically: the main kernel streams weights while the pre-kernel (and the tail
// of the previous kernel of the stream, which does not write packed weights: ptx.cuh) still runs.
// Only plain TMA loads; every wait is bounded.
#include "w4a16_decode.cuh"
#include <algorithm>
#include <mutex>

namespace mgx {
namespace { // (names that w4a16_tc.cu has too)

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

struct tc_params : tc_operands
{
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

template <class FORM>
__global__ void __launch_bounds__(FORM::THREADS, 1)
    w4a16_cluster_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const tc_params p)
{
    constexpr int NB = FORM::NB, CPM = FORM::CPM, GPP = FORM::GPP, ABYTES = FORM::ABYTES, MRW = FORM::MRW, ESETS = FORM::ESETS;
    constexpr int XROWS = FORM::MB; // rows of a partial result
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
    const tc_meta meta(bar_base + 512);
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
        // are requested at once: whatever wrote them is complete (ptx.cuh).  The activation planes are
        // written by the pre-kernel, whose completion is awaited before they are requested.
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
        // Each of the two warps serves 64 output columns.
        grid_dependency_wait(); // sv and sa come from the pre-kernel
        tc_walk walk = walk0;
        int tile, g0, count;
        bool seg_last;
        for(uint32_t pc = 0; walk.next(GPP, tile, g0, count, seg_last); ++pc)
        {
            const uint32_t vb = pc % 3u;
            if(not mbar_wait_bounded(&mfree_bar[vb], ((pc / 3u) & 1u) ^ 1u, abort_flag, 9))
                break;
            tc_stage_metadata<FORM::MB>(p, meta, vb, warp - 13, lane, tile, g0, count);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&meta_bar[vb])) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    else if(warp < 6)
    {
        // ---------------------------------------------------- unpack: nibbles -> bytes
        // one thread per weight row
        const int row            = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
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
            tc_unpack_item<FORM::RAW>(smem + s * TC_WSTAGE, row, cnt, tmem_base + lane_addr + TC_A_COL0 + t * TC_SUPER * TC_A_COLS);
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
        grid_dependency_wait(); // sa comes from the pre-kernel, D may still be read by an earlier one
        const int eset    = warp >= 15 ? 1 : 0;
        const int m0      = eset * MRW;          // first of the rows this warp folds
        const int quarter = warp & 3;
        const int col     = quarter * 32 + lane; // output column inside the tile = TMEM lane
        float out[MRW];
#pragma unroll
        for(int m = 0; m < MRW; ++m)
            out[m] = 0.0f;
        tc_walk walk = walk0;
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
            tc_fold_pass<FORM>(p, meta, vb, col, m0, tile, g0, count,
                               tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * TC_ACC_COLS + CPM * m0, out);
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

// stages of the weight ring beside the planes of `items` work items
template <int NB>
int ring_stages(int items, int rows)
{
    const size_t fixed = tc_fixed<NB>(items, rows);
    return fixed >= TC_SMEM ? 0 : static_cast<int>(std::min<size_t>(TC_MAX_STAGES, (TC_SMEM - fixed) / TC_WSTAGE));
}

template <class FORM>
void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, size_t smem, cudaStream_t stream)
{
    // programmatic dependent launch: the kernel may start while the pre-kernel still runs
    // and waits for it (griddepcontrol.wait) only where it reads what the pre-kernel wrote
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(FORM::THREADS);
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
template <class FORM>
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
        configure<FORM>(cfg, attr, device_sm_count() / split, split, TC_SMEM, nullptr);
        attr[0]      = attr[1];
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, w4a16_cluster_kernel<FORM>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

template <class FORM>
int launch_main(int blocks, const CUtensorMap& tw, const CUtensorMap& ta, tc_params p, cudaStream_t stream)
{
    constexpr int rows = FORM::MB;
    int rc = ensure_smem_optin(reinterpret_cast<const void*>(w4a16_cluster_kernel<FORM>), TC_SMEM);
    if(rc != MGX_OK)
        return rc;
    // The split of K with the smallest estimated time: a CTA takes 32 KB per item at its share of the HBM
    // stream (44 bytes per ns with all SMs at it, at most 100), at least 600 ns per item with fewer than
    // three stages in its ring; a tile costs a pass of the exchange, the last one 1 us.
    double best = 0.0;
    for(int split = 1; split <= TC_MAX_SPLIT and split <= blocks; split *= 2)
    {
        const int items  = static_cast<int>(ceil_div(blocks, split));
        const int stages = ring_stages<FORM::NB>(items, rows);
        if(stages < 2)
            continue;
        const int clusters = std::min(max_clusters<FORM>(split), p.tiles);
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
    configure<FORM>(cfg, attr, p.clusters, p.split, tc_fixed<FORM::NB>(p.items, rows) + p.stages * TC_WSTAGE, stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, w4a16_cluster_kernel<FORM>, tw, ta, p));
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

size_t w4a16_cluster_workspace(const mgx_w4_desc& d) { return tc_layout(d).end; }

int w4a16_cluster_launch(const mgx_w4_desc& d, const void* A, const void* Bp, const void* scales,
                    const void* zp, void* D, void* workspace, size_t workspace_bytes,
                    cudaStream_t stream)
{
    const tc_layout lay(d);
    if(workspace == nullptr or workspace_bytes < lay.end)
        return MGX_E_WORKSPACE;
    if((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0 or
       not w4a16_tc_pointers_ok(d, A, Bp, scales, zp))
        return MGX_E_ALIGNMENT;
    CUtensorMap tw, ta;
    tc_params p{};
    const int rc = tc_prepare(d, lay, A, Bp, scales, zp, D, static_cast<uint8_t*>(workspace), nullptr, 0, stream, tw, ta, p);
    if(rc != MGX_OK)
        return rc;
    p.tiles = lay.tiles;
    return tc_by_rows(d.M, [&](auto form) { return launch_main<decltype(form)>(lay.blocks, tw, ta, p, stream); });
}

int w4a16_cluster_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
