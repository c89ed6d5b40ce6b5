// quant_dot for at most 16 rows of A (decode-sized batches) with the weights [N, K]
// K-contiguous: bound by the HBM stream of the weights, so the roles of the operands are
// swapped with respect to the tiled GEMM.  The WEIGHTS are the tcgen05 A operand (128 output
// columns per MMA, straight from the TMA-filled shared memory), the few activation rows are
// the B operand (N = 16), and the accumulator holds D transposed: TMEM lane = output column,
// TMEM column = row of A.
// Work: a cluster of S CTAs owns a range of output columns in whole sixteens, so that ranges differ by at
// most 16 columns, and CTA r of it the r-th share of K.  The range goes by in blocks of at most 128
// columns; the S partial sums of a block are added through distributed shared memory in rank order
// (int32: exact; fp32: fixed order).  No partial sums, counters or second kernel in global memory: with
// the (128-column tile, k-block) items dealt out evenly and tiles completed by the last CTA to arrive,
// half of a small linear's time was that exchange (one row, 4096 x 4096 fp8: 10.7 us, now 7.6; 16 rows,
// 14336 x 4096: 23.4 us, then 15.0).
// The epilogue is the tiled GEMM's arithmetic (dequantizelinear, bias, activation, fp32 / fp16 /
// raw int32 output; op::quant_dot + dequantizelinear.hpp:60-82 + the fused pointwise module).
//
// CTA = 192 to 576 threads: warp 0 TMA producer, warp 1 MMA issuer + tensor-memory owner, the others
// epilogue, for every four rows one to each quarter of the columns.  The last block's epilogue is not hidden:
// with one warp to a quarter for all rows a lane's sixteen GELUs in turn were 2 us (16 rows, fp8 with GELU,
// 14336 x 4096 14.1 -> 12.3 us, 4096 x 4096 9.2 -> 7.9, int8 8192 x 1024 8.2 -> 5.5); with 576 threads for
// few rows the larger block starts later (one row, 4096 x 4096 7.35 -> 7.7).  Only plain TMA loads; every wait
// is bounded.
#include "common.cuh"
#include "ptx.cuh"
#include "qgemm_math.cuh"
#include <algorithm>
#include <cuda_fp16.h>
#include <mutex>
#include <type_traits>

namespace mgx {

constexpr int GV_ROWS    = 128; // output columns (weight rows) per tile = UMMA M
constexpr int GV_MB      = 16;  // padded rows of A = UMMA N
constexpr int GV_BK      = 128; // bytes of K per item
constexpr int GV_BOX     = 32;  // weight rows per TMA request
constexpr int GV_STAGES  = 10;
constexpr int GV_W_BYTES = GV_ROWS * GV_BK; // 16384
constexpr int GV_A_BYTES = GV_MB * GV_BK;   // 2048
constexpr int GV_STAGE   = GV_W_BYTES + GV_A_BYTES;
constexpr int GV_PART    = GV_MB * GV_ROWS * 4; // a block's raw accumulators: [row of A][column]
constexpr int GV_SMEM    = GV_STAGES * GV_STAGE + 2 * GV_PART + 256 + 1024;
constexpr int GV_RPW     = 4; // rows of A that an epilogue warp takes
constexpr int GV_THREADS = 64 + GV_MB / GV_RPW * GV_ROWS; // at most
constexpr int GV_MAX_SPLIT = 8; // CTAs of a cluster; divides GV_ROWS

struct gv_params
{
    void* D;
    const float* scale;
    const float* bias;
    int64_t N, ldd;
    int M;
    int scale_mode, act;
    int kblocks;                   // 128-byte blocks of K
    int col_units, clusters, split; // sixteens of output columns; clusters; CTAs of a cluster
};

template <bool IS_INT, class OutT>
__global__ void __launch_bounds__(GV_THREADS, 1)
    qgemv_kernel(const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_a,
                 const gv_params p)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem           = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    uint8_t* bar_base       = smem + GV_STAGES * GV_STAGE;
    uint64_t* full_bar      = reinterpret_cast<uint64_t*>(bar_base);
    uint64_t* empty_bar     = full_bar + GV_STAGES;
    uint64_t* accf_bar      = empty_bar + GV_STAGES; // [2]
    uint64_t* acce_bar      = accf_bar + 2;          // [2]
    uint64_t* peer_bar      = acce_bar + 2;          // the whole cluster's partial sums are in place
    uint32_t* tmem_slot     = reinterpret_cast<uint32_t*>(peer_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    uint32_t* part          = reinterpret_cast<uint32_t*>(bar_base + 256); // [2][row of A][column]

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    grid_launch_dependents();
    if(threadIdx.x == 0)
    {
        for(int s = 0; s < GV_STAGES; ++s)
        {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for(int b = 0; b < 2; ++b)
        {
            mbar_init(&accf_bar[b], 1);
            mbar_init(&acce_bar[b], (blockDim.x - 64) / 32);
        }
        mbar_init(peer_bar, p.split);
        *abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&tmap_w);
        prefetch_tensormap(&tmap_a);
    }
    if(warp == 1)
    {
        tmem_alloc(tmem_slot, 32);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if(p.split > 1)
        cluster_barrier(); // the other CTAs' barriers exist before anyone arrives on them
    const int rank    = static_cast<int>(blockIdx.x) % p.split;
    const int cluster = static_cast<int>(blockIdx.x) / p.split;
    // this cluster's columns and this CTA's blocks of K
    const int n_lo   = static_cast<int>(static_cast<int64_t>(p.col_units) * cluster / p.clusters) * 16;
    const int n_hi   = static_cast<int>(static_cast<int64_t>(p.col_units) * (cluster + 1) / p.clusters) * 16;
    const int kb_lo  = static_cast<int>(static_cast<int64_t>(p.kblocks) * rank / p.split);
    const int kb_hi  = static_cast<int>(static_cast<int64_t>(p.kblocks) * (rank + 1) / p.split);
    const int blocks = (n_hi - n_lo + GV_ROWS - 1) / GV_ROWS;

    if(warp == 0)
    {
        // ---------------------------------------------------- TMA producer
        grid_dependency_wait(); // A is the previous kernel's output
        uint32_t s = 0, ph = 1;
        bool ok    = true;
        for(int blk = 0; ok and blk < blocks; ++blk)
        {
            const int n0    = n_lo + blk * GV_ROWS;
            const int boxes = (min(GV_ROWS, n_hi - n0) + GV_BOX - 1) / GV_BOX;
            for(int kb = kb_lo; kb < kb_hi; ++kb)
            {
                if(not mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2))
                {
                    ok = false;
                    break;
                }
                if(elect_one())
                {
                    uint8_t* st = smem + s * GV_STAGE;
                    // bytes past the end of K or N are zero-filled and still counted; columns of the tile
                    // past the range keep what an earlier item left there and are not stored
                    mbar_expect_tx(&full_bar[s], static_cast<uint32_t>(boxes * GV_BOX * GV_BK + GV_A_BYTES));
                    for(int i = 0; i < boxes; ++i)
                        tma_load_2d(st + i * GV_BOX * GV_BK, &tmap_w, &full_bar[s], kb * GV_BK, n0 + i * GV_BOX);
                    tma_load_2d(st + GV_W_BYTES, &tmap_a, &full_bar[s], kb * GV_BK, 0);
                }
                if(++s == GV_STAGES)
                    s = 0, ph ^= 1u;
            }
        }
    }
    else if(warp == 1)
    {
        // ---------------------------------------------------- MMA issuer
        // D (s32 | f32) += A (weights) * B (rows of A); M = 128, N = 16, K = 32 bytes
        constexpr uint32_t idesc = IS_INT ? make_idesc(2u, 1u, 1u, GV_ROWS, GV_MB)
                                          : make_idesc(1u, 0u, 0u, GV_ROWS, GV_MB);
        const uint64_t desc0 = make_smem_desc_sw128(smem_u32(smem));
        bool ok    = true;
        uint32_t s = 0, ph = 0;
        grid_dependency_wait(); // the bounded waits below must not count the previous kernel's time
        for(int blk = 0; ok and blk < blocks; ++blk)
        {
            const uint32_t buf = blk & 1u;
            if(not mbar_wait_warp(&acce_bar[buf], ((blk >> 1) & 1u) ^ 1u, abort_flag, 4))
                break;
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + buf * GV_MB;
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
                    const uint64_t adesc = desc0 + static_cast<uint64_t>((s * GV_STAGE) >> 4);
                    const uint64_t bdesc = adesc + static_cast<uint64_t>(GV_W_BYTES >> 4);
#pragma unroll
                    for(int k = 0; k < 4; ++k)
                    {
                        const uint64_t koff = static_cast<uint64_t>((k * 32) >> 4);
                        if constexpr(IS_INT)
                            mma_i8(d_tmem, adesc + koff, bdesc + koff, idesc, (kb != kb_lo or k != 0) ? 1u : 0u);
                        else
                            mma_f8(d_tmem, adesc + koff, bdesc + koff, idesc, (kb != kb_lo or k != 0) ? 1u : 0u);
                    }
                    tc_commit(&empty_bar[s]);
                    if(kb == kb_hi - 1)
                        tc_commit(&accf_bar[buf]);
                }
                if(++s == GV_STAGES)
                    s = 0, ph ^= 1u;
            }
        }
    }
    else
    {
        // ---------------------------------------------------- epilogue
        grid_dependency_wait(); // D free to overwrite
        const int quarter = warp & 3;
        const int row0    = (warp - 2) / 4 * GV_RPW;
        const int epi     = static_cast<int>(blockDim.x) - 64; // threads
        const float tensor_scale = p.scale_mode == MGX_SCALE_PER_TENSOR ? __ldg(p.scale) : 1.0f;
        // raw accumulator -> output value, as in the tiled GEMM's epilogue
        auto finish = [&](uint32_t raw, float s, float b) {
            float x;
            if constexpr(IS_INT)
            {
                const int32_t a = static_cast<int32_t>(raw);
                x = p.scale_mode == MGX_SCALE_NONE ? (fits_small(a) ? int_to_float_small(a) : __int2float_rn(a))
                                                   : dequant_i32(a, s);
            }
            else
            {
                x = __uint_as_float(raw);
                if(p.scale_mode != MGX_SCALE_NONE)
                    x = __fmul_rn(x, s);
            }
            if(p.bias != nullptr)
                x = __fadd_rn(x, b);
            switch(p.act)
            {
            case MGX_ACT_RELU: return apply_act<MGX_ACT_RELU>(x);
            case MGX_ACT_GELU_ERF: return apply_act<MGX_ACT_GELU_ERF>(x);
            case MGX_ACT_GELU_TANH: return apply_act<MGX_ACT_GELU_TANH>(x);
            case MGX_ACT_SILU: return apply_act<MGX_ACT_SILU>(x);
            default: return x;
            }
        };
        auto store = [&](int64_t m, int64_t n, uint32_t raw, float s, float b) {
            if constexpr(std::is_same<OutT, int32_t>::value)
                static_cast<int32_t*>(p.D)[m * p.ldd + n] = static_cast<int32_t>(raw);
            else if constexpr(std::is_same<OutT, float>::value)
                static_cast<float*>(p.D)[m * p.ldd + n] = finish(raw, s, b);
            else
                static_cast<__half*>(p.D)[m * p.ldd + n] = __float2half_rz(finish(raw, s, b));
        };
        auto column = [&](int64_t n, float& s, float& b) {
            s = tensor_scale, b = 0.0f;
            if(n < p.N)
            {
                if(p.scale_mode == MGX_SCALE_PER_COL)
                    s = __ldg(p.scale + n);
                if(p.bias != nullptr)
                    b = __ldg(p.bias + n);
            }
        };
        bool dead = false; // a wait gave up: go on without waiting, the barriers need every thread
        const int et = threadIdx.x - 64;
        for(int blk = 0; blk < blocks; ++blk)
        {
            const uint32_t buf = blk & 1u;
            const int n0       = n_lo + blk * GV_ROWS;
            const int cols     = static_cast<int>(min(static_cast<int64_t>(min(GV_ROWS, n_hi - n0)), p.N - n0)); // of this block
            const int col      = quarter * 32 + lane;
            float s = 1.0f, b = 0.0f;
            if(p.split == 1)
                column(n0 + col, s, b); // (latency hidden behind the main loop)
            if(not dead and not mbar_wait_warp(&accf_bar[buf], (blk >> 1) & 1u, abort_flag, 3))
                dead = true;
            tc_fence_after_sync();
            uint32_t acc[GV_RPW];
            tmem_ld_32x32b_x4(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * GV_MB + row0, acc);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if(lane == 0)
                mbar_arrive(&acce_bar[buf]);
            if(p.split == 1)
            {
                if(col < cols and not dead)
                {
#pragma unroll
                    for(int m = 0; m < GV_RPW; ++m)
                        if(row0 + m < p.M)
                            store(row0 + m, n0 + col, acc[m], s, b);
                }
                continue;
            }
            uint32_t* mine = part + buf * (GV_MB * GV_ROWS);
#pragma unroll
            for(int m = 0; m < GV_RPW; ++m)
                if(row0 + m < p.M)
                    mine[(row0 + m) * GV_ROWS + col] = acc[m];
            // CTA r finishes the r-th share of the columns.  A buffer is written again two blocks later,
            // after the exchange of the next block, which every thread reaches after it has read this one.
            const int share = GV_ROWS / p.split;
            const int c     = rank * share + et % share;
            column(n0 + c, s, b);
            asm volatile("bar.sync 1, %0;" ::"r"(epi) : "memory");
            if(et < p.split)
                cluster_arrive(peer_bar, et);
            if(not dead and not __all_sync(0xffffffffu, mbar_wait_cluster_bounded(peer_bar, blk & 1, abort_flag, 6)))
                dead = true;
            if(c < cols and not dead)
                for(int m = et / share; m < p.M; m += epi / share)
                {
                    uint32_t tot = IS_INT ? 0u : __float_as_uint(0.0f);
#pragma unroll
                    for(int r = 0; r < GV_MAX_SPLIT; ++r)
                    {
                        if(r >= p.split)
                            break;
                        const uint32_t v = cluster_load(mine + m * GV_ROWS + c, r);
                        if constexpr(IS_INT)
                            tot += v;
                        else
                            tot = __float_as_uint(__uint_as_float(tot) + __uint_as_float(v));
                    }
                    store(m, n0 + c, tot, s, b);
                }
        }
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
        tmem_dealloc(tmem_base, 32);
    }
    if(p.split > 1)
        cluster_barrier(); // no CTA leaves while another may read its partial sums
}

// ------------------------------------------------------------------ host
namespace {

int encode_k_major(CUtensorMap* map, const void* base, uint64_t k, uint64_t rows, uint64_t pitch,
                   uint32_t box_rows)
{
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[2]    = {k, rows};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2]     = {GV_BK, box_rows};
    cuuint32_t estr[2]    = {1u, 1u};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides,
                        box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MGX_OK : MGX_E_INVALID_ARG;
}

void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, int threads, cudaStream_t stream)
{
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = GV_SMEM;
    cfg.stream           = stream;
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id               = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(split);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs    = attr;
    cfg.numAttrs = split > 1 ? 2 : 1;
}

// Clusters of `split` CTAs that fit the device at once (asked once per device).
template <bool IS_INT, class OutT>
int max_clusters(int split)
{
    static std::mutex m;
    static int cached[64][GV_MAX_SPLIT + 1] = {};
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
        configure(cfg, attr, device_sm_count() / split, split, GV_THREADS, nullptr);
        attr[0]      = attr[1];
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, qgemv_kernel<IS_INT, OutT>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

template <bool IS_INT, class OutT>
int launch_gv(const CUtensorMap& tw, const CUtensorMap& ta, gv_params p, cudaStream_t stream)
{
    auto kernel = qgemv_kernel<IS_INT, OutT>;
    int rc      = ensure_smem_optin(reinterpret_cast<const void*>(kernel), GV_SMEM);
    if(rc != MGX_OK)
        return rc;
    // The split of K with the smallest estimated time: a CTA takes its share of the HBM stream (6.5 KB
    // per ns over the CTAs, at most 100 bytes per ns), at least 190 ns per 128-byte block of K (ten
    // requests in flight, however narrow the block, against HBM's latency), and an exchange through the
    // cluster costs about 1 us, hidden but for the last.
    double best = 0.0;
    for(int split = 1; split <= GV_MAX_SPLIT and split <= p.kblocks; split *= 2)
    {
        const int clusters = std::min(max_clusters<IS_INT, OutT>(split), p.col_units);
        const int64_t cols = ceil_div(p.col_units, clusters) * 16;
        const int64_t kb   = ceil_div(p.kblocks, split);
        const double rate  = std::min(100.0, 6500.0 / (clusters * split));
        const double ns    = std::max(cols * kb * GV_BK / rate, ceil_div(cols, GV_ROWS) * kb * 190.0) +
                          ceil_div(cols, GV_ROWS) * 200.0 + (split > 1 ? 1000.0 : 0.0);
        if(best == 0.0 or ns < best)
            best = ns, p.split = split, p.clusters = clusters;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(cfg, attr, p.clusters, p.split, 64 + static_cast<int>(ceil_div(p.M, GV_RPW)) * GV_ROWS, stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, tw, ta, p));
}

} // namespace

// the skinny-M kernel covers: one batch, at most 16 rows of A, weights [N, K] K-contiguous, no
// residual, no fused quantizelinear output, no per-row scale
bool qgemv_applicable(const mgx_qgemm_desc& d, bool has_residual, bool has_qout)
{
    return d.M <= GV_MB and d.batch == 1 and d.b_layout == MGX_B_NK and not has_residual and
           not has_qout and d.scale_mode != MGX_SCALE_PER_ROW and
           ceil_div(d.N, GV_ROWS) * ceil_div(d.K, GV_BK) < (int64_t{1} << 30);
}

int qgemv_launch(const mgx_qgemm_desc& d, const void* A, const void* B, void* D, const float* scale,
                 const float* bias, int64_t ldb, cudaStream_t stream)
{
    CUtensorMap tw, ta;
    int rc = encode_k_major(&tw, B, static_cast<uint64_t>(d.K), static_cast<uint64_t>(d.N),
                            static_cast<uint64_t>(ldb), GV_BOX);
    if(rc != MGX_OK)
        return rc;
    rc = encode_k_major(&ta, A, static_cast<uint64_t>(d.K), static_cast<uint64_t>(d.M),
                        static_cast<uint64_t>(d.lda), GV_MB);
    if(rc != MGX_OK)
        return rc;
    gv_params p{};
    p.D          = D;
    p.scale      = scale;
    p.bias       = bias;
    p.M          = static_cast<int>(d.M);
    p.N          = d.N;
    p.ldd        = d.ldd;
    p.scale_mode = d.scale_mode;
    p.act        = d.act;
    p.kblocks    = static_cast<int>(ceil_div(d.K, GV_BK));
    p.col_units  = static_cast<int>(ceil_div(d.N, 16));
    const bool is_int = d.ab_type == MGX_I8;
    if(d.out_type == MGX_I32)
        return launch_gv<true, int32_t>(tw, ta, p, stream);
    if(d.out_type == MGX_F16)
        return is_int ? launch_gv<true, __half>(tw, ta, p, stream) : launch_gv<false, __half>(tw, ta, p, stream);
    return is_int ? launch_gv<true, float>(tw, ta, p, stream) : launch_gv<false, float>(tw, ta, p, stream);
}

int qgemv_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
