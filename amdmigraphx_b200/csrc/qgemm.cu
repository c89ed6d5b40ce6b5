// C ABI of quant_dot and fp16 dot: checks of the arguments, the [K,N] re-layout, the choice of kernel and tile.
#include "common.cuh"
#include "qgemm_host.cuh"
#include <algorithm>
#include <cstdlib>
#include <mutex>

namespace mgx {

// The tile with the smallest estimated time
//   waves x max(main loop, epilogue) + a quarter of the smaller of the two + what a pair of CTAs costs once,
// the epilogue of a tile being under the main loop of the next.  A k-block (128 bytes of K) costs a tile of one CTA
// 2.44 x (128 + BN): the operand rows it takes out of L2, which bound it; a pair 249 + 2.22 x BN; a tile's epilogue
// 509 + 38.2 x BN; a pair 2858 more per launch (two barriers over the cluster, 256 rows to fill).  The constants are
// fitted to 47 shapes (256 to 8192 rows, K 256 to 8192, int8, fp8 and fp16) timed with all seven tiles: the choice is
// at most 4 % off the fastest, 0.5 % on average.  Pairs against the best tile of one CTA, int8 / fp8: 8192^3 405 -> 328
// us, 1000 x 8192 x 8192 57.5 / 61.4 -> 49.5 / 54.4 (224: 148 pairs' tiles, two full waves), 6144 x 1024 x 4096 27.1 ->
// 22.3, 700 x 4000 x 2000 18.8 -> 14.5; but 1024^3 5.7 -> 7.9 and 3072 x 3072 x 768 16.6 -> 18.3, where K is short.
// Tiles of 128 x 64 that are so few that clusters of 2, 4 or 8 CTAs with a share of K each all run at once: a k-block costs
// the same, the launch of clusters and the exchange of their sums 2740 (1.2 us) + 25 per CTA + 230 (S - 2) more, fitted
// to 24 shapes.  Against the best without: 100 x 1000 x 4096 9.3 -> 6.6 us, 20 x 2048 x 8192 14.4 -> 9.2, 200 x 768 x 3072
// 7.2 -> 6.5, 512 x 1024 x 4096 9.3 -> 8.5; but 128 x 2048 x 2048 6.1 -> 6.6 by four, 256 x 1024 x 1024 4.4 -> 5.2 by two.
struct tile_choice
{
    bool pair;
    int bn;
    int split = 1; // CTAs that share a tile's K
};

static tile_choice pick_tile(const mgx_qgemm_desc& d)
{
    // tuning knob: MGX_CUDA_QGEMM_BN = 64 | 128 | 256 forces tiles of one CTA of that width, 1128 | 1192 | 1224 | 1256
    // tiles of a pair, 2002 | 2004 | 2008 a shared K
    static const int forced = [] {
        const char* e = std::getenv("MGX_CUDA_QGEMM_BN");
        return e != nullptr ? std::atoi(e) : 0;
    }();
    static constexpr tile_choice all[] = {{false, 256}, {false, 128}, {false, 64}, {true, 256}, {true, 224}, {true, 192}, {true, 128}};
    const int64_t sms = device_sm_count();
    const double kb   = static_cast<double>(ceil_div(d.K * (d.ab_type == MGX_F16 ? 2 : 1), 128));
    tile_choice best{false, 64};
    double best_cost = 0.0;
    for(const tile_choice c : all)
    {
        if(forced == c.bn + (c.pair ? 1000 : 0))
            return c;
        const int64_t tiles = ceil_div(d.M, c.pair ? 256 : 128) * ceil_div(d.N, c.bn) * d.batch;
        const double waves  = static_cast<double>(ceil_div(tiles, c.pair ? sms / 2 : sms));
        const double main   = kb * (c.pair ? 249.0 + 2.22 * c.bn : 2.44 * (128 + c.bn));
        const double epi    = 509.0 + 38.2 * c.bn;
        const double cost   = waves * std::max(main, epi) + 0.25 * std::min(main, epi) + (c.pair ? 2858.0 : 0.0);
        if(best_cost == 0.0 or cost < best_cost)
            best_cost = cost, best = c;
    }
    for(int split : {2, 4, 8})
    {
        if(split > kb)
            break;
        if(forced == 2000 + split)
            return {false, 64, split};
        const int64_t tiles = ceil_div(d.M, 128) * ceil_div(d.N, 64) * d.batch;
        const double cost   = static_cast<double>(ceil_div(static_cast<int64_t>(kb), split)) * 2.44 * 192 + 3478.0 +
                            25.0 * static_cast<double>(tiles * split) + 230.0 * (split - 2);
        if(forced == 0 and cost < best_cost and tiles * split <= sms and tiles <= qgemm_split_clusters(split))
            best_cost = cost, best = {false, 64, split};
    }
    return best;
}

} // namespace mgx

using namespace mgx;

extern "C" size_t mgx_cuda_qgemm_workspace(const mgx_qgemm_desc* d)
{
    if(d == nullptr)
        return 0;
    if(d->b_layout != MGX_B_KN)
    {
        // [N,K] operands need no scratch.  Launches of at most 16 rows announced some when their kernel kept
        // partial sums in global memory; the answer stays positive, nothing reads what is lent
        if(d->M > 0 and d->N > 0 and d->K > 0 and d->ab_type != MGX_F16 and qgemv_applicable(*d, false, false))
            return 256;
        return 0;
    }
    if(d->ab_type == MGX_F16)
        return static_cast<size_t>(d->batch) * d->N * ((d->K + 7) / 8 * 8) * 2;
    const int64_t kpad = (d->K + 15) / 16 * 16;
    return static_cast<size_t>(d->batch) * d->N * kpad;
}

extern "C" int mgx_cuda_qgemm(const mgx_qgemm_desc* d, const void* A, const void* B, void* D,
                              const float* scale, const float* bias, const void* residual,
                              void* workspace, size_t workspace_bytes, void* stream_)
{
    if(D == nullptr)
        return MGX_E_INVALID_ARG;
    return mgx_cuda_qgemm_ex(d, A, B, D, scale, bias, residual, nullptr, workspace, workspace_bytes,
                             stream_);
}

extern "C" int mgx_cuda_qgemm_ex(const mgx_qgemm_desc* d, const void* A, const void* B, void* D,
                                 const float* scale, const float* bias, const void* residual,
                                 const mgx_qgemm_qout* q, void* workspace, size_t workspace_bytes,
                                 void* stream_)
{
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if(d == nullptr or A == nullptr or B == nullptr)
        return MGX_E_INVALID_ARG;
    qout_args qo;
    if(q != nullptr and q->q != nullptr)
    {
        if(q->q_type != MGX_I8 and q->q_type != MGX_FP8_E4M3FN)
            return MGX_E_UNSUPPORTED;
        if(d->out_type == MGX_I32 or q->ldq < d->N or not(q->scale > 0.0f))
            return MGX_E_INVALID_ARG;
        qo.Dq       = q->q;
        qo.ldq      = q->ldq;
        qo.stride_q = q->stride_q;
        qo.scale    = q->scale;
        qo.zp       = q->zero_point;
        qo.fp8      = q->q_type == MGX_FP8_E4M3FN ? 1 : 0;
        qo.write_d  = D != nullptr ? 1 : 0;
        qo.lut      = (q->flags & MGX_QOUT_LUT) != 0 ? q->lut : nullptr;
    }
    else if(D == nullptr)
        return MGX_E_INVALID_ARG;
    if(D == nullptr)
        D = qo.Dq; // never written (write_d = 0); keeps the pointer checks below uniform
    if(d->M <= 0 or d->N <= 0 or d->K <= 0 or d->batch <= 0)
        return MGX_E_INVALID_ARG;
    if(d->ab_type != MGX_I8 and d->ab_type != MGX_FP8_E4M3FN and d->ab_type != MGX_F16)
        return MGX_E_UNSUPPORTED;
    const bool f16       = d->ab_type == MGX_F16;
    const int64_t ealign = f16 ? 8 : 16; // elements per 16 bytes
    if(f16 and qo.Dq != nullptr)
        return MGX_E_UNSUPPORTED;
    if(d->scale_mode < MGX_SCALE_NONE or d->scale_mode > MGX_SCALE_PER_ROW)
        return MGX_E_INVALID_ARG;
    if(d->scale_mode != MGX_SCALE_NONE and scale == nullptr)
        return MGX_E_INVALID_ARG;
    if(d->act < MGX_ACT_NONE or d->act > MGX_ACT_SILU)
        return MGX_E_INVALID_ARG;
    if(d->out_type == MGX_I32 and
       (d->ab_type != MGX_I8 or d->scale_mode != MGX_SCALE_NONE or bias != nullptr or
        residual != nullptr or d->act != MGX_ACT_NONE))
        return MGX_E_UNSUPPORTED;
    if(d->M > INT32_MAX or d->N > INT32_MAX or d->K > INT32_MAX)
        return MGX_E_TOO_LARGE;
    if(d->lda < d->K or d->ldd < d->N)
        return MGX_E_INVALID_ARG;
    if((reinterpret_cast<uintptr_t>(A) & 15u) or (d->lda % ealign) or
       (d->batch > 1 and (d->stride_a % ealign)))
        return MGX_E_ALIGNMENT;

    const void* Bk   = B;
    int64_t ldb      = d->ldb;
    int64_t stride_b = d->stride_b;
    if(d->b_layout == MGX_B_KN)
    {
        // quant_dot's [K,N] operand is re-laid out K-contiguous into the workspace
        if(d->ldb != d->N or (d->batch > 1 and d->stride_b != d->K * d->N))
            return MGX_E_UNSUPPORTED;
        const size_t need = mgx_cuda_qgemm_workspace(d);
        if(workspace == nullptr or workspace_bytes < need)
            return MGX_E_WORKSPACE;
        if(reinterpret_cast<uintptr_t>(workspace) & 15u)
            return MGX_E_ALIGNMENT;
        const int64_t kpad = (d->K + ealign - 1) / ealign * ealign;
        int rc = f16 ? transpose_16bit_ld(B, workspace, d->K, d->N, d->batch, kpad, stream)
                     : transpose_8bit_ld(B, workspace, d->K, d->N, d->batch, kpad, stream);
        if(rc != MGX_OK)
            return rc;
        Bk       = workspace;
        ldb      = kpad;
        stride_b = d->N * kpad;
    }
    else if(d->b_layout != MGX_B_NK)
        return MGX_E_INVALID_ARG;
    if(ldb < d->K)
        return MGX_E_INVALID_ARG;
    if((reinterpret_cast<uintptr_t>(Bk) & 15u) or (ldb % ealign) or
       (d->batch > 1 and (stride_b % ealign)))
        return MGX_E_ALIGNMENT;

    // at most 16 rows: stream the weights once
    if(not f16 and qgemv_applicable(*d, residual != nullptr, qo.Dq != nullptr))
        return qgemv_launch(*d, A, Bk, D, scale, bias, ldb, stream);
    const qgemm_operands o{A, Bk, D, scale, bias, residual, ldb, stride_b};
    const tile_choice tile = pick_tile(*d);
    const qgemm_kind kind  = tile.split > 1 ? QGEMM_SPLIT : (tile.pair ? QGEMM_PAIR : QGEMM_ONE);
#define MGX_QGEMM_LAUNCH(NAME, TYPE, KIND, BN)                          \
    if(d->ab_type == TYPE and kind == KIND and tile.bn == BN)           \
        return qgemm_launch_##NAME(*d, o, qo, tile.split, stream);
    MGX_QGEMM_FORMS(MGX_QGEMM_LAUNCH)
#undef MGX_QGEMM_LAUNCH
    return MGX_E_UNSUPPORTED;
}

int mgx::qgemm_status(unsigned int* out)
{
    *out = 0;
#define MGX_QGEMM_STATUS(NAME, TYPE, KIND, BN) qgemm_status_##NAME,
    for(auto f : {MGX_QGEMM_FORMS(MGX_QGEMM_STATUS)})
#undef MGX_QGEMM_STATUS
    {
        unsigned int v = 0;
        const int rc   = f(&v);
        if(rc != 0)
            return rc;
        if(*out == 0)
            *out = v;
    }
    return 0;
}

// ------------------------------------------------------------------ allocation-free variant
// Scratch for mgx_cuda_qgemm_static_scratch(): lives in the library's device image, one copy
// per GPU that loads the library, held until the process exits.
namespace {
constexpr size_t static_scratch_bytes = size_t{16} << 20; // 16 MiB
static __device__ __align__(256) uint8_t g_static_scratch[static_scratch_bytes];

// Device address of g_static_scratch on the current device.  In host code the array's name
// is only a handle for the runtime, not a device pointer, so the address is looked up once
// per device (with that device current) and cached.
int static_scratch_address(void** out)
{
    constexpr int max_devices = 64;
    static std::mutex m;
    static void* cached[max_devices] = {};
    int dev       = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if(e != cudaSuccess)
        return static_cast<int>(e);
    if(dev < 0 or dev >= max_devices)
        return MGX_E_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(m);
    if(cached[dev] == nullptr)
    {
        void* p = nullptr;
        e       = cudaGetSymbolAddress(&p, g_static_scratch);
        if(e != cudaSuccess)
            return static_cast<int>(e);
        cached[dev] = p;
    }
    *out = cached[dev];
    return MGX_OK;
}
} // namespace

extern "C" size_t mgx_cuda_qgemm_static_scratch_limit(void) { return static_scratch_bytes; }

extern "C" int mgx_cuda_qgemm_static_scratch(const mgx_qgemm_desc* d, const void* A, const void* B,
                                             void* D, const float* scale, const float* bias,
                                             const void* residual, void* stream)
{
    if(d == nullptr)
        return MGX_E_INVALID_ARG;
    if(d->M <= 0 or d->N <= 0 or d->K <= 0 or d->batch <= 0)
        return MGX_E_INVALID_ARG;
    // only the re-laid-out copy of a [K,N] operand is kept in the scratch
    const size_t need = d->b_layout == MGX_B_KN ? mgx_cuda_qgemm_workspace(d) : 0;
    if(need > static_scratch_bytes)
        return MGX_E_TOO_LARGE;
    void* scratch = nullptr;
    if(need > 0)
    {
        const int rc = static_scratch_address(&scratch);
        if(rc != MGX_OK)
            return rc;
    }
    return mgx_cuda_qgemm(d, A, B, D, scale, bias, residual, scratch, need, stream);
}
