// Weight-only int4 linear for prefill (M > 16 activation rows) on the tcgen05 tensor core:
//
//   D[m,n] = sum_k a[m,k] * (q[n,k] - zp[n,k/group]) * s[n,k/group]
//
// as an fp16 x fp16 -> fp32 GEMM whose A operand is dequantised on the fly: the packed weights
// of 128 output columns x 128 k arrive by TMA, sixteen warps (four threads per weight row) turn them
// into fp16 values (q - zp) * s and write them straight into TENSOR MEMORY, and the MMAs read
// their A operand from there; the B operand is the caller's fp16 activation matrix, fetched by
// TMA as it lies in memory.  The dequantised weights never exist in shared or global memory
// (the reference materialises them: src/onnx/parse_matmulnbits.cpp:85-158 IR on the ref target).
//
// CTA tile = 128 output columns x up to 192 activation rows, a multiple of 16 chosen by the launch: all of K,
// persistent over tiles, or, where tiles are few, a share of K and one tile.
// The tensor core cuts its running sum at every step, which pulls a long one towards zero.  So a sum
// runs over no more than half of K: the two halves of a tile have an accumulator each and are added in
// the epilogue, and with tiles of up to 128 rows a third one lets the next tile begin meanwhile.  Mean relative error against 64-bit
// sums, weights and activations of one sign, with one accumulator a tile and with two: K 4096 -2.3e-5 /
// -1.1e-5, 11008 -5.8e-5 / -2.9e-5, 28672 -1.6e-4 / -8.1e-5.
// CTA = 832 threads:
//   warp 0       TMA producer: per 128-k group 8 KB of packed weights and 2 x 16 KB of activations
//   warp 1       MMA issuer
//   warps 2..17  dequantise (nibbles -> fp16 pairs: a byte permute, a mask, one multiply-add and one multiply per
//                pair) -> tcgen05.st.  Two sets of eight take groups in turn, so that a group's chain from the landed
//                bytes to the MMA has the time of two groups' MMAs
//   warps 18..25 epilogue, half of a tile's activation rows each: tcgen05.ld, add, convert,
//                store (consecutive lanes = consecutive n)
// 512 rows, tiles of 128 (us), with one set of eight warps (19 instructions a word and a wait before them) and so:
// 12288 x 4096 56.3 / 47.9, 22016 x 4096 92.0 / 82.1, 4096 x 11008 48.3 / 42.9.  What bounds it: issue slots (3200
// instructions a group, a third of them the conversion) and the operands' stream from L2, which alone takes 34 us of
// the first.
// Only plain TMA loads; every wait is bounded.
#include "common.cuh"
#include "ptx.cuh"
#include <algorithm>
#include <cuda_fp16.h>
#include <mutex>

namespace mgx {

constexpr int PF_ROWS    = 128; // output columns (weight rows) per tile = UMMA M
constexpr int PF_MAX_TOKENS = 192; // activation rows per tile = UMMA N, at most
constexpr int PF_GROUP_K = 128;
constexpr int PF_MAX_STAGES = 8;
constexpr int PF_W_BYTES = PF_ROWS * PF_GROUP_K / 2;      // 8192
constexpr int PF_TSTAGES = 2;                             // A operand buffers in tensor memory (four: no faster)
constexpr int PF_MAX_ACCS = 3;                            // accumulators there
constexpr int PF_A_COL0  = 384;                           // behind three of 128 columns or two of 192
constexpr int PF_A_COLS  = PF_GROUP_K / 2;                // 64 columns per group
constexpr int PF_SMEM    = 226 * 1024;
constexpr int PF_DEQUANT = 16; // warps that dequantise
constexpr int PF_EPI0    = 2 + PF_DEQUANT; // first epilogue warp
constexpr int PF_THREADS = 32 * (PF_EPI0 + 8);
constexpr int PF_EPI     = 256; // threads of the epilogue
constexpr int PF_MAX_SPLIT = 8; // CTAs of a cluster

struct pf_params
{
    const __half* scales;
    const uint8_t* zp; // may be null
    __half* D;
    int64_t M, N, K, ldd;
    int group, groups_per_row, zp_const;
    int tiles_m, num_tiles;
    int split; // CTAs of a cluster that share a tile's K; then every CTA has one tile
    int tokens, stages, accs; // activation rows of a tile; stages of the ring; accumulators
};

// Bytes of half a group's activations (64 k: 128 bytes a row) and of a stage of the ring.
__host__ __device__ constexpr int pf_atom(int tokens) { return tokens * 128; }
__host__ __device__ constexpr int pf_stage(int tokens) { return PF_W_BYTES + 2 * pf_atom(tokens); }

// SPLIT: a cluster shares a tile's K
template <bool SPLIT>
__global__ void __launch_bounds__(PF_THREADS, 1)
    w4a16_prefill_kernel(const __grid_constant__ CUtensorMap tmap_w,
                         const __grid_constant__ CUtensorMap tmap_a,
                         const pf_params p)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem           = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
    const int TOKENS = p.tokens, STAGES = p.stages, ACCS = p.accs, ATOM = pf_atom(TOKENS), STAGE = pf_stage(TOKENS);
    uint8_t* bar_base       = smem + STAGES * STAGE;
    uint64_t* full_bar      = reinterpret_cast<uint64_t*>(bar_base);
    uint64_t* empty_bar     = full_bar + PF_MAX_STAGES;  // weights read (a warp each) + MMAs retired (1)
    uint64_t* unp_bar       = empty_bar + PF_MAX_STAGES; // A operand in tensor memory
    uint64_t* tfree_bar     = unp_bar + PF_TSTAGES;  // MMAs that read it retired
    uint64_t* accf_bar      = tfree_bar + PF_TSTAGES; // accumulator ready
    uint64_t* acce_bar      = accf_bar + PF_MAX_ACCS;     // accumulator drained
    uint64_t* peer_bar      = acce_bar + PF_MAX_ACCS;          // the cluster's partial results are in place
    uint32_t* tmem_slot     = reinterpret_cast<uint32_t*>(peer_bar + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    float* part             = reinterpret_cast<float*>(smem); // [activation row][column], after the main loop

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    grid_launch_dependents();
    if(threadIdx.x == 0)
    {
        for(int s = 0; s < STAGES; ++s)
        {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], PF_DEQUANT / 2 + 1);
        }
        for(int s = 0; s < PF_TSTAGES; ++s)
        {
            mbar_init(&unp_bar[s], PF_DEQUANT / 2);
            mbar_init(&tfree_bar[s], 1);
        }
        for(int b = 0; b < ACCS; ++b)
        {
            mbar_init(&accf_bar[b], 1);
            mbar_init(&acce_bar[b], PF_EPI / 32);
        }
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

    if constexpr(SPLIT)
        cluster_barrier(); // the other CTAs' barriers exist before anyone arrives on them
    const int G      = static_cast<int>(p.K / PF_GROUP_K);
    const int rank   = SPLIT ? static_cast<int>(blockIdx.x) % p.split : 0;
    const int first  = SPLIT ? static_cast<int>(blockIdx.x) / p.split : blockIdx.x;
    const int step   = SPLIT ? static_cast<int>(gridDim.x) / p.split : gridDim.x;
    const int g_lo   = SPLIT ? G * rank / p.split : 0, g_hi = SPLIT ? G * (rank + 1) / p.split : G;
    // two segments of K, each with an accumulator (a CTA's share of K that is one of several: one)
    const int g_mid  = SPLIT or G == 1 ? g_hi : (g_lo + g_hi) / 2;
    const int rshift = 31 - __clz(p.group / PF_GROUP_K); // groups are powers of two

    // everything the roles touch may be the previous kernel's: activations, packed weights, scales and zero
    // points as its results, D as its input.  (The bounded waits below must not count its time either.)
    grid_dependency_wait();

    if(warp == 0)
    {
        // ---------------------------------------------------- TMA producer
        uint32_t s = 0, ph = 1;
        bool ok    = true;
        for(int t = first; ok and t < p.num_tiles; t += step)
        {
            const int n0 = (t / p.tiles_m) * PF_ROWS;
            const int m0 = (t % p.tiles_m) * TOKENS;
            for(int g = g_lo; g < g_hi; ++g)
            {
                if(not mbar_wait_warp(&empty_bar[s], ph, abort_flag, 2))
                {
                    ok = false;
                    break;
                }
                if(elect_one())
                {
                    uint8_t* st = smem + s * STAGE;
                    mbar_expect_tx(&full_bar[s], STAGE);
                    tma_load_2d(st, &tmap_w, &full_bar[s], g * (PF_GROUP_K / 2), n0);
                    tma_load_2d(st + PF_W_BYTES, &tmap_a, &full_bar[s], g * PF_GROUP_K, m0);
                    tma_load_2d(st + PF_W_BYTES + ATOM, &tmap_a, &full_bar[s], g * PF_GROUP_K + 64, m0);
                }
                if(++s == static_cast<uint32_t>(STAGES))
                    s = 0, ph ^= 1u;
            }
        }
    }
    else if(warp == 1)
    {
        // ---------------------------------------------------- MMA issuer
        // D f32 += A f16 (weights, tensor memory) * B f16 (activation rows, K-major shared
        // memory); M = 128, N = the tile's rows, K = 16 per instruction.  The accumulators take turns over the
        // segments: with three the epilogue of a tile overlaps the main loop of the next.
        const uint32_t idesc = make_idesc(1u, 0u, 0u, PF_ROWS, static_cast<uint32_t>(TOKENS));
        const uint64_t bdesc0    = make_smem_desc_sw128(smem_u32(smem + PF_W_BYTES));
        uint32_t s = 0, ts = 0, tp = 0, buf = 0, bp = 1;
        bool ok    = true;
        for(int t = first; ok and t < p.num_tiles; t += step)
            for(int g = g_lo; ok and g < g_hi;)
            {
                const int g0 = g, g1 = g0 < g_mid ? g_mid : g_hi;
                ok = mbar_wait_warp(&acce_bar[buf], bp, abort_flag, 4);
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + buf * TOKENS;
                for(; ok and g < g1; ++g)
                {
                    // implies that the stage's TMA requests have landed
                    ok = mbar_wait_warp(&unp_bar[ts], tp, abort_flag, 5);
                    if(not ok)
                        break;
                    tc_fence_after_sync();
                    if(elect_one())
                    {
                        const uint64_t bdesc  = bdesc0 + static_cast<uint64_t>((s * STAGE) >> 4);
                        const uint32_t a_tmem = tmem_base + PF_A_COL0 + ts * PF_A_COLS;
#pragma unroll
                        for(int k = 0; k < 8; ++k) // (64 k per 128-byte atom)
                            mma_f16_tmem_a(d_tmem, a_tmem + k * 8,
                                           bdesc + static_cast<uint64_t>(((k >> 2) * ATOM + (k & 3) * 32) >> 4), idesc,
                                           (g != g0 or k != 0) ? 1u : 0u);
                        tc_commit(&tfree_bar[ts]);
                        tc_commit(&empty_bar[s]);
                        if(g == g1 - 1)
                            tc_commit(&accf_bar[buf]);
                    }
                    if(++s == static_cast<uint32_t>(STAGES))
                        s = 0;
                    if(++ts == PF_TSTAGES)
                        ts = 0, tp ^= 1u;
                }
                if(++buf == static_cast<uint32_t>(ACCS))
                    buf = 0, bp ^= 1u;
            }
    }
    else if(warp < PF_EPI0)
    {
        // ---------------------------------------------------- dequantise: nibbles -> fp16
        // Two sets of eight warps take groups in turn, each with a place of its own in tensor memory.  In a set two
        // threads per weight row, 64 k each: 32 packed bytes (64-byte swizzle: a quarter warp's 16-byte reads fall in
        // eight different bank groups) -> 32 words of two fp16 each, in k order, to this row's lane of tensor memory.
        const uint32_t set       = (warp - 2) >> 3;
        const int half           = ((warp - 2) >> 2) & 1;
        const int row            = (warp & 3) * 32 + lane;
        const uint32_t a_tmem    = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + PF_A_COL0 + set * PF_A_COLS + half * 32;
        const int sw             = (row >> 1) & 3;
        const uint8_t* const pk0 = smem + row * 64 + (((half * 2) ^ sw) << 4);
        const uint8_t* const pk1 = smem + row * 64 + (((half * 2 + 1) ^ sw) << 4);
        // A packed byte holds k (low nibble) and k + 1: as 0x6400 | q and 0x6400 | q << 4 they are the halves
        // 1024 + q and 1024 + 16 q.  times (1, 1/16) less (1024 + zp, 64 + zp) is q - zp, exact in fp16; one
        // rounding in the multiply with the scale
        const __half2 unit = __halves2half2(__float2half_rn(1.0f), __float2half_rn(0.0625f));
        auto less_zp       = [](int z) { return __halves2half2(__int2half_rn(-1024 - z), __int2half_rn(-64 - z)); };
        __half2 zz2        = less_zp(p.zp_const);
        uint32_t s = 0, ph = 0, turn = 0, tp = 1;
        bool ok = true;
        for(int t = first; ok and t < p.num_tiles; t += step)
        {
            const int n  = min((t / p.tiles_m) * PF_ROWS + row, static_cast<int>(p.N) - 1);
            const unsigned short* srow =
                reinterpret_cast<const unsigned short*>(p.scales) + static_cast<int64_t>(n) * p.groups_per_row;
            const uint8_t* zrow = p.zp == nullptr ? nullptr : p.zp + static_cast<int64_t>(n) * p.groups_per_row;
            // scale and zero point of this set's next group are fetched one ahead
            int ahead             = min(g_lo + static_cast<int>(turn ^ set), g_hi - 1) >> rshift;
            unsigned short s_next = __ldg(srow + ahead);
            uint8_t z_next        = zrow == nullptr ? 0 : __ldg(zrow + ahead);
#pragma unroll 1
            for(int g = g_lo; g < g_hi; ++g, turn ^= 1u)
            {
                if(turn == set)
                {
                    const unsigned short s_cur = s_next;
                    if(zrow != nullptr)
                        zz2 = less_zp(z_next);
                    ahead  = min(g + 2, g_hi - 1) >> rshift;
                    s_next = __ldg(srow + ahead);
                    if(zrow != nullptr)
                        z_next = __ldg(zrow + ahead);
                    // the tensor-memory stores below are warp-wide: leave only as a whole warp
                    ok = mbar_wait_warp(&full_bar[s], ph, abort_flag, 1);
                    if(not ok)
                        break;
                    const uint4 w0 = *reinterpret_cast<const uint4*>(pk0 + s * STAGE);
                    const uint4 w1 = *reinterpret_cast<const uint4*>(pk1 + s * STAGE);
                    __syncwarp();
                    if(lane == 0)
                        mbar_arrive(&empty_bar[s]); // the packed block is in registers
                    const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
                    const uint32_t ss    = static_cast<uint32_t>(s_cur) * 0x00010001u;
                    const __half2 ss2    = *reinterpret_cast<const __half2*>(&ss);
                    uint32_t u[32];
#pragma unroll
                    for(int i = 0; i < 8; ++i)
#pragma unroll
                        for(int j = 0; j < 4; ++j)
                        {
                            const uint32_t h = __byte_perm(ww[i], 0x64646464u, 0x4040u + j * 0x0101u) & 0xFFF0FF0Fu;
                            const __half2 x  = __hmul2(__hfma2(*reinterpret_cast<const __half2*>(&h), unit, zz2), ss2);
                            u[4 * i + j]     = *reinterpret_cast<const uint32_t*>(&x);
                        }
                    // (the place is waited for last: the MMAs that free it run during all of the above)
                    ok = mbar_wait_warp(&tfree_bar[set], tp, abort_flag, 8);
                    if(not ok)
                        break;
                    tp ^= 1u;
                    tc_fence_after_sync();
                    tmem_st_32x32b_x32(a_tmem, u);
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if(lane == 0)
                        mbar_arrive(&unp_bar[set]);
                }
                if(++s == static_cast<uint32_t>(STAGES))
                    s = 0, ph ^= 1u;
            }
        }
    }
    else
    {
        // ---------------------------------------------------- epilogue
        const int quarter = warp & 3;
        // this warp's activation rows of the tile, 16 at a time
        const int chunks = TOKENS / 16, lower = (chunks + 1) / 2;
        const int c0 = warp >= PF_EPI0 + 4 ? lower * 16 : 0, mine = warp >= PF_EPI0 + 4 ? chunks - lower : lower;
        const int segs    = g_mid < g_hi ? 2 : 1;
        uint32_t buf = 0, bp = 0;
        for(int t = first; t < p.num_tiles; t += step)
        {
            const int64_t n  = static_cast<int64_t>(t / p.tiles_m) * PF_ROWS + quarter * 32 + lane;
            const int64_t m0 = static_cast<int64_t>(t % p.tiles_m) * TOKENS;
            const uint32_t buf0 = buf;
            bool ok = true;
            for(int i = 0; ok and i < segs; ++i)
            {
                ok = mbar_wait_warp(&accf_bar[buf], bp, abort_flag, 3);
                if(++buf == static_cast<uint32_t>(ACCS))
                    buf = 0, bp ^= 1u;
            }
            // (in a cluster a wait that gave up goes on without waiting: the barriers below need every thread)
            if(not SPLIT and not ok)
                break;
            const uint32_t buf1 = buf0 + 1 == static_cast<uint32_t>(ACCS) ? 0 : buf0 + 1;
            tc_fence_after_sync();
            const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c0;
            __half* dst    = p.D + (m0 + c0) * p.ldd + n;
            const int rows = static_cast<int>(min(p.M - m0 - c0, static_cast<int64_t>(mine * 16))); // of this warp's that exist
#pragma unroll 1
            for(int c = 0; c < mine; ++c)
            {
                uint32_t acc[16];
                tmem_ld_32x32b_x16(tbase + buf0 * TOKENS + c * 16, acc);
                if(not SPLIT and segs == 2)
                {
                    uint32_t acc1[16];
                    tmem_ld_32x32b_x16(tbase + buf1 * TOKENS + c * 16, acc1);
                    tmem_ld_wait();
#pragma unroll
                    for(int j = 0; j < 16; ++j)
                        acc[j] = __float_as_uint(__uint_as_float(acc[j]) + __uint_as_float(acc1[j]));
                }
                else
                    tmem_ld_wait();
                if constexpr(SPLIT)
                {
                    // (every request has landed and every MMA has read: the ring is free)
#pragma unroll
                    for(int j = 0; j < 16; ++j)
                        part[(c0 + c * 16 + j) * PF_ROWS + quarter * 32 + lane] = __uint_as_float(acc[j]);
                }
                else if(n < p.N)
                {
#pragma unroll
                    for(int j = 0; j < 16; ++j, dst += p.ldd)
                        if(c * 16 + j < rows)
                            *dst = __float2half_rn(__uint_as_float(acc[j]));
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if(lane == 0)
            {
                mbar_arrive(&acce_bar[buf0]);
                if(segs == 2)
                    mbar_arrive(&acce_bar[buf1]);
            }
            if constexpr(SPLIT)
            {
                // CTA r adds up the r-th share of the tile's columns, four at a time
                asm volatile("bar.sync 1, %0;" ::"n"(PF_EPI) : "memory");
                const int et = static_cast<int>(threadIdx.x) - 32 * PF_EPI0;
                if(et < p.split)
                    cluster_arrive(peer_bar, et);
                if(ok and __all_sync(0xffffffffu, mbar_wait_cluster_bounded(peer_bar, 0u, abort_flag, 6)))
                {
                    const int share = PF_ROWS / p.split, per = share / 4;
                    const int col   = rank * share + et % per * 4;
                    const int64_t n4 = static_cast<int64_t>(t / p.tiles_m) * PF_ROWS + col;
                    for(int m = et / per; m < TOKENS and m0 + m < p.M; m += PF_EPI / per)
                    {
                        float v[PF_MAX_SPLIT][4], sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for(int r = 0; r < PF_MAX_SPLIT; ++r)
                            if(r < p.split)
                                cluster_load4(part + m * PF_ROWS + col, r, v[r]);
#pragma unroll
                        for(int r = 0; r < PF_MAX_SPLIT; ++r)
                            if(r < p.split)
#pragma unroll
                                for(int e = 0; e < 4; ++e)
                                    sum[e] += v[r][e];
#pragma unroll
                        for(int e = 0; e < 4; ++e)
                            if(n4 + e < p.N)
                                p.D[(m0 + m) * p.ldd + n4 + e] = __float2half_rn(sum[e]);
                    }
                }
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
        tmem_dealloc(tmem_base, 512);
    }
    if constexpr(SPLIT)
        cluster_barrier(); // no CTA leaves while another may read its partial result
}

// ------------------------------------------------------------------ host
namespace {

int encode_rows(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t inner,
                uint64_t rows, uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_rows,
                CUtensorMapSwizzle swz)
{
    cuTensorMapEncodeTiled_t encode = get_tensor_map_encoder();
    if(encode == nullptr)
        return MGX_E_DRIVER;
    cuuint64_t dims[2]    = {inner, rows};
    cuuint64_t strides[1] = {pitch_bytes};
    cuuint32_t box[2]     = {box_inner, box_rows};
    cuuint32_t estr[2]    = {1u, 1u};
    CUresult r = encode(map, type, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MGX_OK : MGX_E_INVALID_ARG;
}

void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, cudaStream_t stream)
{
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(PF_THREADS);
    cfg.dynamicSmemBytes = PF_SMEM;
    cfg.stream           = stream;
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id               = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(split);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs    = attr;
    cfg.numAttrs = split > 1 ? 2 : 1;
}

// Clusters of `split` CTAs that fit the device at once (asked once per device): a cluster lies inside a
// GPC, so that fewer fit than the SMs alone would allow.
int max_clusters(int split)
{
    static std::mutex m;
    static int cached[64][PF_MAX_SPLIT + 1] = {};
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess or dev < 0 or dev >= 64)
        return device_sm_count() / (2 * split);
    std::lock_guard<std::mutex> lock(m);
    int& n = cached[dev][split];
    if(n == 0)
    {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[2];
        configure(cfg, attr, device_sm_count() / split, split, nullptr);
        attr[0]      = attr[1];
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, w4a16_prefill_kernel<true>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

// The rows of a tile and the split of its K with the smallest estimated time, in cycles: waves of tiles, each its
// groups at the slowest of the MMAs, the operands' stream from L2 (62 bytes per cycle) and the dequantising warps, then
// what the epilogue keeps to itself.  (512 rows, 12288 x 4096: 384 tiles of 128 rows are two and a half waves, 47.9 us,
// 288 of 176 rows two, 41.8; 4096 x 11008: 128 tiles of 128 rows 43.1, 96 of 176 48.9.  1000 rows, 12288 x 4096: 92.6 and
// 81.6.)
// K is shared by a cluster where tiles are few, each CTA at least four groups, and only where all the clusters run at
// once, as one left over costs a second wave (24 tokens, 4096 x 11008, 32 tiles: 44 us in one CTA each, 17 us; 16
// tiles of K 4096, eight CTAs each 17.6 us, four 10.7; 36 tiles of K 11008, four 36.3, two 29.3).
void pf_plan(const mgx_w4_desc& d, pf_params& p)
{
    const int64_t tiles_n = ceil_div(d.N, PF_ROWS), groups = d.K / PF_GROUP_K, sms = device_sm_count();
    double best  = 0.0;
    int64_t last = 0;
    const int clusters[3] = {max_clusters(2), max_clusters(4), max_clusters(8)};
    // Of the numbers of tiles with the same rows in a tile the smallest is the best: one candidate for every multiple of
    // 16 rows, whatever M is.
    for(int rows = PF_MAX_TOKENS; rows > 0 and ceil_div(d.M, rows) <= ceil_div(d.M, 64); rows -= 16)
    {
        const int64_t tiles_m = ceil_div(d.M, rows);
        if(tiles_m == last)
            continue;
        last                = tiles_m;
        const int tokens    = static_cast<int>(ceil_div(ceil_div(d.M, tiles_m), 16) * 16);
        const int64_t tiles = tiles_n * tiles_m;
        int split           = 1;
        for(int i = 0; i < 3 and groups >= 8 << i and tiles <= clusters[i]; ++i)
            split = 2 << i;
        const double group = std::max({4.0 * tokens, pf_stage(tokens) / 62.0, 560.0}) + 100.0;
        const double waves = split > 1 ? 1.0 : static_cast<double>(ceil_div(tiles, sms));
        const double alone = 12.0 * tokens; // the last tile's epilogue, and every one's with two accumulators
        const double cost  = waves * ceil_div(groups, split) * group + (tokens > 128 ? waves : 1.0) * alone + (split > 1 ? 2500.0 : 0.0);
        if(best != 0.0 and cost >= best)
            continue;
        best        = cost;
        p.tokens    = tokens;
        p.tiles_m   = static_cast<int>(tiles_m);
        p.num_tiles = static_cast<int>(tiles);
        p.split     = split;
    }
    p.accs   = p.tokens <= 128 ? 3 : 2;
    p.stages = static_cast<int>(std::min<int64_t>(PF_MAX_STAGES, (PF_SMEM - 1536) / pf_stage(p.tokens)));
}

} // namespace

bool w4a16_prefill_applicable(const mgx_w4_desc& d, const void* A, const void* Bp)
{
    const int64_t ratio = d.group / PF_GROUP_K;
    return d.M > 16 and d.K % PF_GROUP_K == 0 and d.group % PF_GROUP_K == 0 and
           (ratio & (ratio - 1)) == 0 and d.act == MGX_ACT_NONE and d.lda % 8 == 0 and
           ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(Bp)) & 15u) == 0 and
           ceil_div(d.N, PF_ROWS) * ceil_div(d.M, 64) < (int64_t{1} << 30) and
           d.N * (d.K / d.group) < (int64_t{1} << 40);
}

int w4a16_prefill_launch(const mgx_w4_desc& d, const void* A, const void* Bp, const void* scales,
                         const void* zp, void* D, cudaStream_t stream)
{
    CUtensorMap tw, ta;
    int rc = encode_rows(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, Bp, static_cast<uint64_t>(d.K / 2),
                         static_cast<uint64_t>(d.N), static_cast<uint64_t>(d.K / 2), PF_GROUP_K / 2,
                         PF_ROWS, CU_TENSOR_MAP_SWIZZLE_64B);
    if(rc != MGX_OK)
        return rc;
    pf_params p{};
    p.scales         = static_cast<const __half*>(scales);
    p.zp             = static_cast<const uint8_t*>(zp);
    p.D              = static_cast<__half*>(D);
    p.M              = d.M;
    p.N              = d.N;
    p.K              = d.K;
    p.ldd            = d.ldd;
    p.group          = d.group;
    p.groups_per_row = static_cast<int>(d.K / d.group);
    p.zp_const       = d.zp_const;
    rc = ensure_smem_optin(reinterpret_cast<const void*>(w4a16_prefill_kernel<true>), PF_SMEM);
    if(rc == MGX_OK)
        rc = ensure_smem_optin(reinterpret_cast<const void*>(w4a16_prefill_kernel<false>), PF_SMEM);
    if(rc != MGX_OK)
        return rc;
    pf_plan(d, p);
    rc = encode_rows(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT16, A, static_cast<uint64_t>(d.K), static_cast<uint64_t>(d.M),
                     static_cast<uint64_t>(d.lda) * 2, 64, static_cast<uint32_t>(p.tokens), CU_TENSOR_MAP_SWIZZLE_128B);
    if(rc != MGX_OK)
        return rc;
    auto* kernel = p.split > 1 ? w4a16_prefill_kernel<true> : w4a16_prefill_kernel<false>;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(cfg, attr, p.split > 1 ? p.num_tiles : std::min(p.num_tiles, device_sm_count()), p.split, stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, tw, ta, p));
}

int w4a16_prefill_status(unsigned int* out) { return read_and_clear_status(out); }

} // namespace mgx
