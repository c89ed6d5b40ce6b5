// Weight-only int4 linear for decode (M <= 16 rows of activations), bound by the HBM stream of packed weights:
//
//   D[m,n] = sum_g  s[n,g] * sum_{k in g} (q[n,k] - zp[n,g]) * a[m,k]
//
// q - zp is exact in half, its products with the activations are exact in the tensor core, a group of 128 k is
// summed there in fp32 and folded with its scale into fp32 registers.  (The reference,
// src/onnx/parse_matmulnbits.cpp:85-158 on the ref target, rounds every dequantised weight to half instead.)
//
// A decode linear of a layer is a few microseconds of stream, so what counts is how little stands around it: a warp
// does everything for its weights, from the request to the sum, and waits for nobody in between.
//   * A lane requests its 16 bytes of packed weights (32 k of a row) into its own slots of shared memory, a ring
//     of ST_RING steps deep, and reads the same bytes back: no barrier, and the first of them are under way
//     before the kernel that this one follows is complete.
//   * mma.sync m16n8k16 with 16 weight rows as the A operand, unpacked in registers; the activations are the 8
//     columns (two MMAs for more than 8 rows).  The order of k inside a product is free: the pairs of a packed
//     word are (k, k + 4), and the activations are stored in that order once, when they arrive.
//     (tcgen05 needs the unpacked weights in tensor memory or shared memory, and four hand-overs between warps
//     to get them there and the sums back: at 16 rows they made a work item of 32 KB take 1.5 us on an SM that
//     receives it in 0.7.)
//   * Work: a cluster of CTAs takes consecutive row tiles of 16, each CTA a share of K, whose activations stay in
//     its shared memory; the (tile, group) steps of a CTA are dealt out evenly to its 16 warps.  Sums of a tile
//     meet in shared memory, the CTAs' through distributed shared memory, both in a fixed order.
// One norm and the linear, back to back (us), with the tcgen05 kernels in its place and with this one, 1 / 8 / 16 rows:
// 4096 x 4096 8.0 / 9.6 / 10.2 -> 5.8 / 7.4 / 9.0, 12288 x 4096 10.4 / 15.7 / 17.2 -> 10.4 / 11.7 / 16.4, 4096 x 11008
// 13.6 / 17.2 / 22.4 -> 12.4 / 14.4 / 18.9, 1280 x 8192 8.6 / 10.3 / 10.3 -> 6.7 / 7.9 / 9.1.  What bounds it: issue
// (140 instructions a KB and row tile, of them 35 unpacking logic operations at half rate), at 16 rows also what a
// launch does before and after its steps.  Relative error against 64-bit sums 2.0e-4 to 2.1e-4, the result's rounding
// to half (with the activations as 15-bit integers 2.1e-4 to 2.15e-4).
#include "common.cuh"
#include "ptx.cuh"
#include <algorithm>
#include <cuda_fp16.h>
#include <mutex>

namespace mgx {
namespace {

constexpr int ST_WARPS   = 16;
constexpr int ST_THREADS = 32 * ST_WARPS;
constexpr int ST_GROUP_K = 128;
constexpr int ST_MAX_SPLIT = 8;
constexpr size_t ST_SMEM   = 226 * 1024;

struct st_params
{
    const __half* A;
    const uint8_t* B;
    const __half* scales;
    const uint8_t* zp; // may be null
    __half* D;
    int64_t lda, ldd, N, row_bytes; // row_bytes: K / 2
    int M, groups;                  // groups of 128 k
    int rshift, groups_per_row;     // scale of group g: g >> rshift
    int scale_vec, zp_vec;          // scales and zero points of a step's groups read together: 4, 2 or 1
    int zp_const;
    int clusters, split, split_log; // CTAs of a cluster
    int tiles_each, tiles_left; // tiles of a cluster; so many clusters have one more
    int steps_each, steps_left; // steps of a tile that a CTA has; so many have one more
    int share, max_tiles;       // most groups of a CTA, most tiles of a cluster
};

// A form of the kernel.  MT: tiles of 8 activation rows.  A step: NT x 16 weight rows x GS groups.  RING: steps a warp
// has under way.
template <int MT_, int NT_, int GS_, int RING_>
struct st_form
{
    static constexpr int MT = MT_, NT = NT_, GS = GS_, RING = RING_;
    static constexpr int STEP = NT * GS * 1024;  // bytes of a step
    static constexpr int ROWS = 16 * NT;
    static constexpr int SUMS = ROWS * 8 * MT;   // partial sums of a tile
    // shared memory: activations of a share of K, rings, partial sums of the warps (those of the CTA lie where the
    // rings were)
    static constexpr int rings(int max_tiles)
    {
        const int r = ST_WARPS * RING * STEP, s = max_tiles * SUMS * 4;
        return r > s ? r : s;
    }
    static size_t smem(int M, int share, int max_tiles)
    {
        return static_cast<size_t>(M) * (share * ST_GROUP_K * 2 + 64) + 128 + rings(max_tiles) +
               static_cast<size_t>(max_tiles + ST_WARPS) * SUMS * 4;
    }
};

__device__ __forceinline__ void st_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void st_mma_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// Eight nibbles less their zero point as halves, pairs (k, k + 4): 1024 + q is 0x6400 | q, 1024 + 16 q is
// 0x6400 | q << 4; both differences are exact.  z0 = -(1024 + z), z1 = -(64 + z), in both halves.
// `magic` is 0x64006400 in a register that the compiler does not know as a constant: with two constants it makes two
// instructions of (w & mask) | magic, and logic operations, at half rate, are what a step is made of.
__device__ __forceinline__ void st_unpack(uint32_t w, uint32_t magic, __half2 z0, __half2 z1, uint32_t (&x)[4])
{
    const __half2 sixteenth = __float2half2_rn(0.0625f);
    const uint32_t v        = w >> 8;
    auto select             = [&](uint32_t a, uint32_t mask) {
        uint32_t r;
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(magic));
        return *reinterpret_cast<const __half2*>(&r);
    };
    auto bits_of = [](__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); };
    x[0] = bits_of(__hadd2(select(w, 0x000F000Fu), z0));
    x[1] = bits_of(__hfma2(select(w, 0x00F000F0u), sixteenth, z1));
    x[2] = bits_of(__hadd2(select(v, 0x000F000Fu), z0));
    x[3] = bits_of(__hfma2(select(v, 0x00F000F0u), sixteenth, z1));
}

template <class FORM>
__global__ void __launch_bounds__(ST_THREADS, 1) w4a16_stream_kernel(const st_params p)
{
    constexpr int MT = FORM::MT, NT = FORM::NT, GS = FORM::GS, RING = FORM::RING, STEP = FORM::STEP, ROWS = FORM::ROWS,
                  SUMS = FORM::SUMS;
    static_assert((RING & (RING - 1)) == 0, "the ring's offset wraps by a mask");
    extern __shared__ __align__(128) uint8_t st_shared[];
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int g = lane >> 2, t = lane & 3;
    grid_launch_dependents();

    const int rank    = static_cast<int>(blockIdx.x) & (p.split - 1);
    const int cluster = static_cast<int>(blockIdx.x) >> p.split_log;
    const int steps   = p.steps_each + (rank < p.steps_left ? 1 : 0); // of a row tile: this CTA's share of K
    const int g_lo    = (rank * p.steps_each + min(rank, p.steps_left)) * GS;
    const int mine    = min(p.groups - g_lo, steps * GS); // groups of this CTA
    const int ntiles  = p.tiles_each + (cluster < p.tiles_left ? 1 : 0);
    const int t_lo    = cluster * p.tiles_each + min(cluster, p.tiles_left);
    const int total   = ntiles * steps; // of this CTA, tile-major
    const int per     = (total + ST_WARPS - 1) / ST_WARPS;
    const int first   = min(total, warp * per), last = min(total, first + per);
    const int short_step = mine - (steps - 1) * GS; // groups of a tile's last step

    const uint32_t pitch = static_cast<uint32_t>(p.share) * (ST_GROUP_K * 2) + 64; // of an activation row
    uint8_t* acts  = st_shared;
    uint8_t* rings = acts + ((p.M * pitch + 127) & ~127u);
    float* part    = reinterpret_cast<float*>(rings); // when the rings are done with: [tile][column][row]
    float* red     = reinterpret_cast<float*>(rings + FORM::rings(p.max_tiles));
    uint8_t* ring  = rings + warp * (RING * STEP) + lane * 16; // of this lane

    // ---- the stream: rows g and g + 8 of every 16 of a step, which this lane requests, reads back and multiplies
    const int tile0 = first / steps, left0 = steps - (first - tile0 * steps); // steps left of its tile
    const int n_max = static_cast<int>(p.N) - 1;
    auto row_of     = [&](int tile, int r) { return min((t_lo + tile) * ROWS + r, n_max); };
    int q_tile = tile0, q_left = left0, q_step = first; // next to request
    uint32_t q_off = 0;
    const uint8_t* q_row[2 * NT]; // its bytes
    auto weight_rows = [&] {
        const uint8_t* b = p.B + (g_lo + GS * (steps - q_left)) * 64 + t * 16;
#pragma unroll
        for(int i = 0; i < 2 * NT; ++i)
            q_row[i] = b + row_of(q_tile, g + 8 * i) * p.row_bytes;
    };
    auto request = [&] {
        if(q_step < last)
        {
            const uint32_t dst = smem_u32(ring) + q_off;
            const int count    = q_left > 1 ? GS : short_step;
#pragma unroll
            for(int j = 0; j < GS; ++j)
                if(j < count)
                {
#pragma unroll
                    for(int i = 0; i < 2 * NT; ++i)
                        asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst + (j * 2 * NT + i) * 512),
                                     "l"(q_row[i] + j * 64)
                                     : "memory");
                }
#pragma unroll
            for(int i = 0; i < 2 * NT; ++i)
                q_row[i] += 64 * GS;
            if(--q_left == 0)
            {
                q_left = steps;
                ++q_tile;
                weight_rows();
            }
        }
        ++q_step;
        q_off = (q_off + STEP) & (RING * STEP - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // whatever wrote the weights is complete (ptx.cuh)
    weight_rows();
#pragma unroll 1
    for(int i = 0; i < RING; ++i)
        request();

    grid_dependency_wait();

    // ---- scales (and zero points) of a step: read one step ahead
    const bool has_zp = p.zp != nullptr;
    int tile = tile0, left = left0;
    int index[2 * NT]; // of the rows' first scales
    auto meta_rows = [&] {
#pragma unroll
        for(int i = 0; i < 2 * NT; ++i)
            index[i] = row_of(tile, g + 8 * i) * p.groups_per_row;
    };
    uint32_t sc[NT * GS]; // halves: rows' scales of the next step, [row][group], two to a word
    uint32_t zps[(NT * GS + 1) / 2];
    auto load_meta = [&] {
        const int grp = g_lo + GS * (steps - left);
        const int end = mine - 1 - (grp - g_lo); // the last group of this CTA, from grp on
        // (grp is a multiple of GS.  A tile's last step may read what belongs to groups beyond it, of this row or the
        // next: not used.)
        if(p.rshift > 0)
        {
            // two neighbours share a scale and a zero point
#pragma unroll
            for(int i = 0; i < 2 * NT; ++i)
#pragma unroll
                for(int j = 0; j < GS; j += 2)
                    sc[(i * GS + j) / 2] =
                        __half_as_ushort(p.scales[index[i] + ((grp + min(j, end)) >> p.rshift)]) * 0x00010001u;
        }
        else
        {
#pragma unroll
            for(int i = 0; i < 2 * NT; ++i)
            {
                const __half* at = p.scales + index[i] + grp;
                if(GS == 4 and p.scale_vec == 4)
                {
                    const uint2 v           = *reinterpret_cast<const uint2*>(at);
                    sc[i * GS / 2]          = v.x;
                    sc[(i * GS + GS - 1) / 2] = v.y;
                }
                else
                {
#pragma unroll
                    for(int j = 0; j < GS; j += 2)
                        sc[(i * GS + j) / 2] = p.scale_vec >= 2
                                                   ? *reinterpret_cast<const uint32_t*>(at + min(j, end & ~1))
                                                   : static_cast<uint32_t>(__half_as_ushort(at[min(j, end)])) |
                                                         static_cast<uint32_t>(__half_as_ushort(at[min(j + 1, end)])) << 16;
                }
            }
        }
        if(has_zp)
        {
            // 16 bits for two groups of a row.  (A byte at a time, and two conversions a row and group: with zero points
            // 12288 x 4096 at 1 and 16 rows 12.0 and 18.5 us, 4096 x 4096 7.0 and 10.0; so 11.5 and 17.9, 6.7 and 9.7.)
            uint32_t pair[NT * GS];
#pragma unroll
            for(int i = 0; i < 2 * NT; ++i)
            {
                const uint8_t* at = p.zp + index[i] + (p.rshift > 0 ? 0 : grp);
                if(GS == 4 and p.rshift == 0 and p.zp_vec == 4)
                {
                    const uint32_t v               = *reinterpret_cast<const uint32_t*>(at);
                    pair[i * GS / 2]               = v & 0xFFFFu;
                    pair[(i * GS + GS - 1) / 2] = v >> 16;
                }
                else
                {
#pragma unroll
                    for(int j = 0; j < GS; j += 2)
                        pair[(i * GS + j) / 2] =
                            p.rshift > 0     ? at[(grp + min(j, end)) >> p.rshift] * 0x0101u
                            : p.zp_vec >= 2 ? *reinterpret_cast<const uint16_t*>(at + min(j, end & ~1))
                                             : at[min(j, end)] | static_cast<uint32_t>(at[min(j + 1, end)]) << 8;
                }
            }
#pragma unroll
            for(int i = 0; i < NT * GS; i += 2)
                zps[i / 2] = pair[i] | (i + 1 < NT * GS ? pair[i + 1] << 16 : 0u);
        }
    };
    meta_rows();
    if(first < last)
        load_meta();

    // ---- activations of the share, a lane's 64 bytes of a group as four chunks of 16 in the order of the packed
    // words: chunk w of lane t at (4 w + t) * 16, so that the lanes of a row read 64 consecutive bytes
    {
        const int chunks = mine * 16; // of a row
        const int dm = ST_THREADS / chunks, dc = ST_THREADS - dm * chunks;
        int m = static_cast<int>(threadIdx.x) / chunks, c = static_cast<int>(threadIdx.x) - m * chunks;
        const __half* src    = p.A + m * p.lda + (g_lo * ST_GROUP_K + c * 8);
        const int64_t stride = dm * p.lda + dc * 8, wrap = p.lda - chunks * 8;
        uint32_t row         = m * pitch; // of the destination
        constexpr int BATCH  = 4;         // in flight together
#pragma unroll 1
        while(m < p.M)
        {
            uint4 v[BATCH];
            uint32_t to[BATCH];
#pragma unroll
            for(int b = 0; b < BATCH; ++b)
            {
                to[b] = 0xFFFFFFFFu;
                if(m < p.M)
                {
                    v[b]  = *reinterpret_cast<const uint4*>(src);
                    to[b] = row + ((c & ~15) | ((c & 3) << 2) | ((c >> 2) & 3)) * 16;
                }
                c += dc, m += dm, src += stride, row += dm * pitch;
                if(c >= chunks)
                    c -= chunks, ++m, src += wrap, row += pitch;
            }
#pragma unroll
            for(int b = 0; b < BATCH; ++b)
                if(to[b] != 0xFFFFFFFFu)
                    *reinterpret_cast<uint4*>(acts + to[b]) =
                        make_uint4(__byte_perm(v[b].x, v[b].z, 0x5410), __byte_perm(v[b].x, v[b].z, 0x7632),
                                   __byte_perm(v[b].y, v[b].w, 0x5410), __byte_perm(v[b].y, v[b].w, 0x7632));
        }
    }
    __syncthreads();

    // ---- steps
    uint32_t magic;
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(magic));
    __half2 z0[2 * NT], z1[2 * NT]; // of the rows
#pragma unroll
    for(int i = 0; i < 2 * NT; ++i)
        z0[i] = __half2half2(__int2half_rn(-1024 - p.zp_const)), z1[i] = __half2half2(__int2half_rn(-64 - p.zp_const));
    // rows beyond M read one that exists; their columns are not stored
    const uint8_t* act_row[MT];
    auto act_rows = [&] {
#pragma unroll
        for(int i = 0; i < MT; ++i)
            act_row[i] = acts + min(g + 8 * i, p.M - 1) * pitch + t * 16 + (steps - left) * (GS * 256);
    };
    act_rows();
    float out[NT][MT][4];
#pragma unroll
    for(int x = 0; x < NT * MT * 4; ++x)
        out[x / (4 * MT)][x / 4 % MT][x % 4] = 0.0f;
    uint32_t off = 0;
#pragma unroll 1
    for(int n = last - first; n > 0; --n)
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
        const uint8_t* from = ring + off;
        off                 = (off + STEP) & (RING * STEP - 1);
        uint32_t s[NT * GS], z[(NT * GS + 1) / 2];
#pragma unroll
        for(int i = 0; i < NT * GS; ++i)
            s[i] = sc[i];
#pragma unroll
        for(int i = 0; i < (NT * GS + 1) / 2; ++i)
            z[i] = zps[i];
        const bool end  = left == 1;
        const int count = end ? short_step : GS;
        const int at    = tile;
        const uint8_t* acts_now[MT];
#pragma unroll
        for(int i = 0; i < MT; ++i)
            acts_now[i] = act_row[i], act_row[i] += GS * 256;
        if(--left == 0)
        {
            left = steps;
            ++tile;
            meta_rows();
            act_rows();
        }
        if(n > 1)
            load_meta();
#pragma unroll
        for(int j = 0; j < GS; ++j)
        {
            if(j > 0 and j >= count)
                break;
            float acc[NT][MT][4];
            uint4 wr[2 * NT];
            if(has_zp)
            {
#pragma unroll
                for(int i = 0; i < 2 * NT; ++i)
                {
                    // 0xE400 | z is -(1024 + z); 960 more is -(64 + z), exactly
                    const int e      = i * GS + j;
                    const uint32_t b = __byte_perm(z[e / 4], 0xE4E4E4E4u, 0x4040u | (e & 3) * 0x0101u);
                    z0[i]            = *reinterpret_cast<const __half2*>(&b);
                    z1[i]            = __hadd2(z0[i], __float2half2_rn(960.0f));
                }
            }
#pragma unroll
            for(int i = 0; i < 2 * NT; ++i)
                wr[i] = *reinterpret_cast<const uint4*>(from + (j * 2 * NT + i) * 512);
#pragma unroll
            for(int w = 0; w < 4; ++w)
            {
                uint4 b[MT];
#pragma unroll
                for(int i = 0; i < MT; ++i)
                    b[i] = *reinterpret_cast<const uint4*>(acts_now[i] + j * 256 + w * 64);
#pragma unroll
                for(int x = 0; x < NT; ++x)
                {
                    auto word = [&](const uint4& v) { return w == 0 ? v.x : (w == 1 ? v.y : (w == 2 ? v.z : v.w)); };
                    uint32_t a[4], c[4];
                    st_unpack(word(wr[2 * x]), magic, z0[2 * x], z1[2 * x], a);
                    st_unpack(word(wr[2 * x + 1]), magic, z0[2 * x + 1], z1[2 * x + 1], c);
#pragma unroll
                    for(int i = 0; i < MT; ++i)
                    {
                        if(w == 0)
                            st_mma_first(acc[x][i], a[0], c[0], a[1], c[1], b[i].x, b[i].y);
                        else
                            st_mma(acc[x][i], a[0], c[0], a[1], c[1], b[i].x, b[i].y);
                        st_mma(acc[x][i], a[2], c[2], a[3], c[3], b[i].z, b[i].w);
                    }
                }
            }
#pragma unroll
            for(int x = 0; x < NT; ++x)
            {
                auto scale = [&](int e) {
                    const __half2 h = *reinterpret_cast<const __half2*>(&s[e / 2]);
                    return (e & 1) != 0 ? __high2float(h) : __low2float(h);
                };
                const float f0 = scale(2 * x * GS + j), f1 = scale((2 * x + 1) * GS + j);
#pragma unroll
                for(int i = 0; i < MT; ++i)
                {
                    out[x][i][0] = fmaf(f0, acc[x][i][0], out[x][i][0]);
                    out[x][i][1] = fmaf(f0, acc[x][i][1], out[x][i][1]);
                    out[x][i][2] = fmaf(f1, acc[x][i][2], out[x][i][2]);
                    out[x][i][3] = fmaf(f1, acc[x][i][3], out[x][i][3]);
                }
            }
        }
        request(); // into the slot just read
        if(end or n == 1)
        {
            // this warp's part of the tile: slot tile + warp is its own (tiles and warps both ascend)
            float* r = red + (at + warp) * SUMS + g;
#pragma unroll
            for(int x = 0; x < NT; ++x)
#pragma unroll
                for(int i = 0; i < MT; ++i)
                {
                    r[(8 * i + 2 * t) * ROWS + 16 * x]         = out[x][i][0];
                    r[(8 * i + 2 * t + 1) * ROWS + 16 * x]     = out[x][i][1];
                    r[(8 * i + 2 * t) * ROWS + 16 * x + 8]     = out[x][i][2];
                    r[(8 * i + 2 * t + 1) * ROWS + 16 * x + 8] = out[x][i][3];
                    out[x][i][0] = out[x][i][1] = out[x][i][2] = out[x][i][3] = 0.0f;
                }
        }
    }
    __syncthreads();

    // ---- sums of the warps, then of the cluster's CTAs: a warp takes 32 of a tile's sums at a time
    constexpr int MS = 32 / ROWS; // activation rows at a time
    const int m_sets = (p.M + MS - 1) / MS, units = ntiles * m_sets;
    const int r      = lane % ROWS;
    // x / d for x d < 2^32 by the multiplication with 2^32 / d rounded up
    auto reciprocal = [](int d) { return d > 1 ? 0xFFFFFFFFu / static_cast<uint32_t>(d) + 1u : 0u; };
    auto quotient   = [](int x, uint32_t rcp) { return rcp != 0u ? static_cast<int>(__umulhi(static_cast<uint32_t>(x), rcp)) : x; };
    const uint32_t by_sets = reciprocal(m_sets), by_per = reciprocal(per);
    auto store             = [&](int x, int m, float v) {
        const int64_t n = static_cast<int64_t>(t_lo + x) * ROWS + r;
        if(n < p.N and m < p.M)
            p.D[m * p.ldd + n] = __float2half_rn(v);
    };
#pragma unroll 1
    for(int u = warp; u < units; u += ST_WARPS)
    {
        const int x = quotient(u, by_sets), m = MS * (u - x * m_sets) + lane / ROWS;
        const int w0 = quotient(x * steps, by_per), w1 = quotient(x * steps + steps - 1, by_per); // who had a part of the tile
        const float* from = red + (x + w0) * SUMS + m * ROWS + r;
        float v           = 0.0f;
#pragma unroll 4
        for(int w = w0; w <= w1; ++w, from += SUMS)
            v += *from;
        if(p.split == 1)
            store(x, m, v);
        else
            part[x * SUMS + m * ROWS + r] = v;
    }
    if(p.split == 1)
        return;
    cluster_barrier();
#pragma unroll 1
    for(int u = warp + rank * ST_WARPS; u < units; u += p.split * ST_WARPS)
    {
        const int x = quotient(u, by_sets), m = MS * (u - x * m_sets) + lane / ROWS;
        const float* from = part + x * SUMS + m * ROWS + r;
        float v[ST_MAX_SPLIT], sum = 0.0f;
#pragma unroll
        for(int q = 0; q < ST_MAX_SPLIT; ++q)
            v[q] = q < p.split ? __uint_as_float(cluster_load(from, q)) : 0.0f;
#pragma unroll
        for(int q = 0; q < ST_MAX_SPLIT; ++q)
            sum += v[q];
        store(x, m, sum);
    }
    cluster_barrier(); // no CTA leaves while another may read its sums
}

void configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int clusters, int split, size_t smem, cudaStream_t stream)
{
    cfg                  = cudaLaunchConfig_t{};
    cfg.gridDim          = dim3(static_cast<unsigned>(clusters * split));
    cfg.blockDim         = dim3(ST_THREADS);
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
    static int cached[64][ST_MAX_SPLIT + 1] = {};
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
        configure(cfg, attr, device_sm_count() / split, split, ST_SMEM, nullptr);
        attr[0]      = attr[1];
        cfg.numAttrs = 1;
        if(cudaOccupancyMaxActiveClusters(&n, w4a16_stream_kernel<FORM>, &cfg) != cudaSuccess or n < 1)
        {
            (void)cudaGetLastError();
            n = device_sm_count() / (2 * split);
        }
    }
    return n;
}

// The work of a launch split in the way that is estimated to be fastest (ns; 0: no room in shared memory).
template <class FORM>
double plan(st_params& p)
{
    if(ensure_smem_optin(reinterpret_cast<const void*>(w4a16_stream_kernel<FORM>), ST_SMEM) != MGX_OK)
        return 0.0;
    const int all   = static_cast<int>(ceil_div(p.groups, FORM::GS));
    const int tiles = static_cast<int>(ceil_div(p.N, FORM::ROWS));
    double best     = 0.0;
    for(int log = 0; (1 << log) <= ST_MAX_SPLIT and (1 << log) <= all; ++log)
    {
        const int split = 1 << log;
        const int clusters  = std::min(max_clusters<FORM>(split), tiles);
        const int steps     = static_cast<int>(ceil_div(all, split));
        const int max_tiles = static_cast<int>(ceil_div(tiles, clusters));
        if(FORM::smem(p.M, steps * FORM::GS, max_tiles) > ST_SMEM)
            continue;
        // steps of a warp at what 16 warps take for a KB each, at least at the pace of the HBM stream; the
        // activations; the sums
        const double per = static_cast<double>(ceil_div(int64_t{max_tiles} * steps, ST_WARPS));
        const double ns  = per * FORM::STEP / 1024 * std::max(FORM::MT == 1 ? 550.0 : 700.0, 16 * 1024.0 * clusters * split / 6500.0) +
                          p.M * steps * FORM::GS * 256 / 40.0 + max_tiles * p.M * 4.0 + (split > 1 ? 1500.0 : 0.0);
        if(best == 0.0 or ns < best)
        {
            best         = ns;
            p.split      = split;
            p.split_log  = log;
            p.clusters   = clusters;
            p.tiles_each = tiles / clusters;
            p.tiles_left = tiles % clusters;
            p.steps_each = all / split;
            p.steps_left = all % split;
            p.share      = steps * FORM::GS;
            p.max_tiles  = max_tiles;
        }
    }
    return best;
}

template <class FORM>
int launch(const st_params& p, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    configure(cfg, attr, p.clusters, p.split, FORM::smem(p.M, p.share, p.max_tiles), stream);
    return static_cast<int>(cudaLaunchKernelEx(&cfg, w4a16_stream_kernel<FORM>, p));
}

// The faster of two forms; where neither fits, the one with the smallest rings.
template <class F0, class F1, class SMALL>
int launch_best(const st_params& p, cudaStream_t stream)
{
    st_params p0 = p, p1 = p;
    const double t0 = plan<F0>(p0), t1 = plan<F1>(p1);
    if(t0 != 0.0 and (t1 == 0.0 or t0 <= t1))
        return launch<F0>(p0, stream);
    if(t1 != 0.0)
        return launch<F1>(p1, stream);
    return plan<SMALL>(p0) != 0.0 ? launch<SMALL>(p0, stream) : MGX_E_UNSUPPORTED;
}

} // namespace

static int64_t kb32(const mgx_w4_desc& d) { return ceil_div(d.N, 128) * ceil_div(d.K, 512); }

// Where it is the faster of the two decode kernels, by 32 KB of packed weights per SM.  Above 8 rows, and with zero points
// up to 4: up to 7 (linears back to back, us, here and w4a16_tc.cu: 16 rows, 8192 x 8192 (6.9) 17.1 and 18.3, 6144 x 11008
// (7.1) 20.4 and 19.1; 4 rows with zero points, the same two 13.6 and 13.7, 14.0 and 13.2, 6144 x 14336 (9.1) 18.6 and
// 14.9).  Up to 4 rows without: up to 10 (6144 x 11008 12.3 and 12.4, 6144 x 14336 15.7 and 15.2, a norm and 22016 x 4096
// (9.3) at 4 rows 15.2 and 15.7; in a decoder layer the second kernel's launch costs 2 us more, 64.2 and 66.1).
// 5 to 8 rows: everywhere (57344 x 8192 (48) 59 and 63), but for large matrices of so long a K that only an eighth of the
// activations fits beside the large rings, whose clusters leave SMs without one (8 rows, 8192 x 20480 (17) 24.5 and 27.8,
// 4096 x 28672 (12) 20.3 and 23.5, 6144 x 28672 (18) 30.7 and 29.2, 8192 x 28672 (24) 38.9 and 35.5; 5 rows 31.2 and 35.2).
bool w4a16_stream_preferred(const mgx_w4_desc& d, bool has_zp)
{
    const int64_t sms = device_sm_count();
    if(d.M > 4 and d.M <= 8)
        return d.M * d.K <= 168 * 1000 or kb32(d) <= 16 * sms;
    return kb32(d) <= (d.M <= 4 and not has_zp ? 10 : 7) * sms;
}

// Activations of an eighth of K beside the smallest rings and the sums of a few tiles.
bool w4a16_stream_fits(const mgx_w4_desc& d)
{
    return kb32(d) <= 7 * static_cast<int64_t>(device_sm_count()) and d.K <= (d.M <= 4 ? 65536 : 28672);
}

int w4a16_stream_launch(const mgx_w4_desc& d, const void* A, const void* Bp, const void* scales, const void* zp, void* D,
                        cudaStream_t stream)
{
    st_params p{};
    p.A              = static_cast<const __half*>(A);
    p.B              = static_cast<const uint8_t*>(Bp);
    p.scales         = static_cast<const __half*>(scales);
    p.zp             = static_cast<const uint8_t*>(zp);
    p.D              = static_cast<__half*>(D);
    p.lda            = d.lda;
    p.ldd            = d.ldd;
    p.N              = d.N;
    p.row_bytes      = d.K / 2;
    p.M              = static_cast<int>(d.M);
    p.groups         = static_cast<int>(d.K / ST_GROUP_K);
    p.groups_per_row = static_cast<int>(d.K / d.group);
    for(p.rshift = 0; (ST_GROUP_K << p.rshift) < d.group; ++p.rshift)
        ;
    p.zp_const = d.zp_const;
    // scales (2 bytes) and zero points (1 byte) of four or two groups are one aligned access
    const auto together = [&](const void* at, int bytes) {
        for(int v : {4, 2})
            if(p.groups_per_row % v == 0 and reinterpret_cast<uintptr_t>(at) % (bytes * v) == 0)
                return v;
        return 1;
    };
    p.scale_vec = together(scales, 2);
    p.zp_vec    = together(zp, 1);
    return d.M <= 8 ? launch_best<st_form<1, 1, 4, 2>, st_form<1, 1, 2, 4>, st_form<1, 1, 2, 2>>(p, stream)
                    : launch_best<st_form<2, 2, 2, 2>, st_form<2, 1, 2, 4>, st_form<2, 1, 2, 2>>(p, stream);
}

} // namespace mgx
