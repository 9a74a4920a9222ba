// Dequantize-fused linear for 9 to 16 batch rows and much weight on sm_100a, weights streamed through shared memory:
//     y[M,N] = epi(pro(x)[M,K] . dequant(W)[N,K]^T),  fp16 x, uint4 W
//
// Replaces the same launches of the reference as its neighbours do (Convert -> Subtract -> Multiply,
// src/nnfusion/core/kernels/cuda_gpu/kernels/elementwise.hpp:33-157, and the Dot,
// src/nnfusion/core/kernels/cuda_gpu/kernels/dot.cpp:27-372).
//
// Why a form of its own: with 16 rows the small-M kernel (dq_gemv_direct.cu) spills, keeps half of the activation fragments in
// shared memory per warp, meets over its 16 warps once per batch of tiles and cuts a K beyond 4096 over CTAs.  Two launches
// instead.  The first (stream_prep_kernel) brings the activations, a few hundred KB, into the order in which the second one's
// lanes want them, normalised and rounded to fp16, with the sums that take the unpacking's offsets and the zero-points out of
// the products (summed as the products are, in the tensor core).  The second:
//   * work is counted in units of 128 weight rows x 128 elements of K; the units, tile by tile, are dealt out to the CTAs in
//     equal contiguous shares, so that a narrow matrix with a long K and a wide one load the SMs alike;
//   * the lanes of one warp keep a ring of units filled by TMA: 8 KB of packed weights, which leave before the launch ahead has
//     ended, and the unit's 4 KB of prepared activations by a bulk copy;
//   * eight warps consume it.  A warp owns 16 rows of the tile for all of the share's K: its sums stay in its registers, scaled
//     in fp32 after every unit, and no warp ever meets another.  Weights become exact fp16 integers by the exponent trick (five
//     instructions per eight weights) and multiply by mma.sync.m16n8k16;
//   * a tile that several CTAs share goes through the workspace, warp by warp: each stores its sums and takes a ticket, the last
//     one adds them in the order of their K ranges (bitwise repeatable; nobody waits for another CTA);
//   * two weight sets (SiLU(gate) * up): a tile is 64 gate rows and the same 64 rows of the up projection, and a warp's 16 rows
//     are 8 of each, so that a lane holds both sums of an output.
// A CTA takes half an SM (113 KB, 288 threads), two are resident.
// What bounds it: with much weight some 180 instructions a warp and unit at half of the issue rate (so are its neighbours); with
// little a fixed cost, the two launches' hand-over and the shared tiles' tickets and sums.  Over 209 shapes at 16 rows both launches
// take 10.3 us + 0.34 us a unit and SM + 1.06 us per 10,000 elements of K (with the norm 12.8, 0.34 and 2.2), within 13 %: small
// weights stay with the small-M kernel.
// Every mbarrier wait is bounded.  On a time-out the CTA raises the status flag; its warps store nothing and take no ticket at the
// ends of tiles that they reach from then on, and it waits (bounded, too) for its copies.  What it has stored by then stays, and
// tickets of shared tiles may be half counted: the workspace has to be zero-filled before its next use.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>

#include "nnf_internal.h"
#include "sm100_ptx.cuh"
#include "stream_shares.h"

namespace
{
using namespace nnf::ptx;

constexpr int kRows = 128;      // weight rows of a tile
constexpr int kUnitK = 128;     // elements of K per unit
constexpr int kBatch = 16;      // batch rows of a block of activations
constexpr int MB = kBatch / 8;
constexpr int kConsumers = 8;   // warps, 16 weight rows of a tile each
constexpr int kThreads = (kConsumers + 1) * 32;
constexpr int kWBytes = kRows * kUnitK / 2;              // packed weights of a unit
constexpr int kBlockBytes = kBatch * (2 * kUnitK + 8);   // prepared activations of a unit
constexpr int kStages = 9;                               // ring of units
constexpr int kSums = MB * 4 * 32;                       // a warp's sums of a tile
constexpr int kSmem = kStages * (kWBytes + kBlockBytes) + 2 * kStages * 8 + 16;
constexpr int kPrepThreads = 128, kPrepUnits = kPrepThreads / 4; // 32 elements a thread
static_assert(kSmem <= 113 * 1024, "two CTAs an SM");
static_assert(kStages <= 32, "a lane per stage");

struct StreamParams
{
    const void* scale[2];
    const uint8_t* zp[2];
    const void* bias;        // fp32 [N], or (has_addend) [M,N] of y's type, or null
    void* y;
    int* status;
    uint32_t* counters;      // [tiles][warps] arrivals at shared tiles; zero before and after
    float* slots;            // [slots][warps][kSums] partial sums of shared tiles
    const uint8_t* xblocks;  // [units of K][kBlockBytes] prepared activations
    int M, N;
    nnf::StreamShares shares;
    int dual;
    int G, zp_row_bytes;
    int group_units;         // units per quantisation group
    uint32_t group_magic;    // ceil(2^32 / group_units)
    int y_f32, scale_f32, has_addend;
};

// 16-byte aligned addresses, a size that is a multiple of 16
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__global__ void __launch_bounds__(kThreads, 2)
    dq_stream_kernel(const StreamParams p, const __grid_constant__ CUtensorMap tmap_w0, const __grid_constant__ CUtensorMap tmap_w1)
{
    extern __shared__ __align__(1024) uint8_t smem[]; // [stages][weights], [stages][activations], barriers, abort flag
    // The next launch on the stream may start as soon as there is room (it waits for this grid's results itself).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t smem_s = smem_u32(smem);
    const uint32_t x_ring = smem_s + kStages * kWBytes;
    const uint32_t bar0 = x_ring + kStages * kBlockBytes;
    auto full = [&](int s) { return bar0 + 8u * s; };              // weights and activations of a unit have landed
    auto empty = [&](int s) { return bar0 + 8u * (kStages + s); }; // ... and have been read by every warp
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(smem + kStages * (kWBytes + kBlockBytes) + 2 * kStages * 8);
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int KU = p.shares.KU;
    const int u_begin = p.shares.begin((int)blockIdx.x);
    const int n_units = p.shares.units((int)blockIdx.x);
    const int tile_begin = u_begin / KU, ku_begin = u_begin - tile_begin * KU;

    // (the producer's lanes each ask for a unit: the four instructions and the wait of a unit take one thread several hundred clocks)
    auto ask_weights = [&](int st, int unit) {
        const int at = ku_begin + unit, tile = tile_begin + at / KU, col = at % KU * (kUnitK / 2);
        const uint32_t dst = smem_s + (uint32_t)(st * kWBytes);
        mbar_arrive_expect_tx(full(st), kWBytes);
        if (p.dual)
        {
            tma_load_2d(dst, &tmap_w0, full(st), col, tile * 64);
            tma_load_2d(dst + kWBytes / 2, &tmap_w1, full(st), col, tile * 64);
        }
        else
            tma_load_2d(dst, &tmap_w0, full(st), col, tile * kRows);
    };
    const int first_round = min(n_units, kStages);
    if (warp == kConsumers)
    {
        if (lane < kStages)
        {
            mbar_init(full(lane), 2); // the weights' announcement and the activations'
            mbar_init(empty(lane), kConsumers);
        }
        if (lane == 0)
            *abort_flag = (smem_s & 1023u) != 0u; // (the swizzle counts on an aligned window)
        fence_barrier_init();
        __syncwarp();
        if (lane < first_round) // weights are constants: they leave before anything else
            ask_weights(lane, lane);
    }
    __syncthreads();

    if (warp == kConsumers)
    {
        // ------------------------------------------------------------ producer
        asm volatile("griddepcontrol.wait;" ::: "memory"); // the activations are what the launch ahead writes
        auto ask_x = [&](int st, int unit) {
            mbar_arrive_expect_tx(full(st), kBlockBytes);
            bulk_load(x_ring + (uint32_t)(st * kBlockBytes), p.xblocks + (size_t)((ku_begin + unit) % KU) * kBlockBytes, kBlockBytes, full(st));
        };
        if (lane < first_round)
            ask_x(lane, lane);
        constexpr int batch = 4; // units at a time (fewer than stages: a lane per stage)
        int i = first_round;
        for (; i < n_units; i += batch)
        {
            const int unit = i + lane, st = unit % kStages;
            const bool active = lane < batch && unit < n_units;
            bool ok = false;
            for (uint32_t tries = 0; tries < kRoleSpin; tries++)
            {
                ok = !active || mbar_try_wait(empty(st), ((unit / kStages) & 1u) ^ 1u);
                if (__all_sync(0xffffffffu, ok) || ((tries & 255u) == 255u && __any_sync(0xffffffffu, *abort_flag != 0)))
                    break;
            }
            if (!__all_sync(0xffffffffu, ok))
            {
                *abort_flag = 1;
                break;
            }
            if (active)
            {
                ask_weights(st, unit);
                ask_x(st, unit);
            }
        }
        // The last copies of every stage land before the CTA ends, whether or not a consumer has waited for them.
        const int last = min(n_units, i) - 1 - lane; // a lane per stage
        if (lane < kStages && last >= 0)
        {
            bool landed = false;
            for (uint32_t tries = 0; tries < kRoleSpin && !landed; tries++)
                landed = mbar_try_wait(full(last % kStages), (last / kStages) & 1u);
            if (!landed)
                *abort_flag = 1;
        }
    }
    else
    {
        // ------------------------------------------------------------ consumers
        const int g = lane >> 2, t = lane & 3;
        // rows of the tile (in shared memory) of accumulator rows g and g + 8
        const int r0 = p.dual ? 8 * warp + g : 16 * warp + g, r1 = p.dual ? r0 + 64 : r0 + 8;
        // raw bytes of a row: 16-byte piece j of row r lies at piece j ^ (r >> 1 & 3).  Lane t holds elements 32 t .. 32 t + 31 of
        // the unit.
        const uint32_t w_at[2] = {smem_s + (uint32_t)(r0 * 64 + ((t ^ ((r0 >> 1) & 3)) << 4)), smem_s + (uint32_t)(r1 * 64 + ((t ^ ((r1 >> 1) & 3)) << 4))};
        const uint32_t x_at = x_ring + (uint32_t)(g * 64 + t * 16);
        const uint32_t nc_at = x_ring + (uint32_t)(kBatch * 256 + t * 16);
        const uint32_t k6400 = held_constant(0x64006400u), k5400 = held_constant(0x54005400u);

        // Scales and zero-points: lane t of a row's four asks for those of unit 4 i + t, four units ahead; a unit's come round by
        // shuffles.  (A warp's rows lie in as many lines: asked for unit by unit they would take the load unit's turns from shared
        // memory's users.)
        int s_tile = tile_begin, s_ku = ku_begin; // unit of this lane's next request
        auto advance = [&](int by) {
            for (s_ku += by; s_ku >= KU; s_ku -= KU)
                s_tile++;
        };
        uint32_t s_raw[2] = {0u, 0u}, z_raw[2] = {0u, 0u}, s_cur[2], z_cur[2];
        int z_shift = 0;
        auto ask_params = [&] {
            const int gr = p.group_units == 1 ? s_ku : (int)__umulhi((uint32_t)s_ku, p.group_magic);
            z_shift = 4 * (gr & 1);
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                const int set = p.dual ? h : 0;
                const size_t n = (size_t)min(p.dual ? s_tile * 64 + r0 : s_tile * kRows + (h == 0 ? r0 : r1), p.N - 1); // (rows past N are never stored)
                s_raw[h] = p.scale_f32 ? __ldg(static_cast<const uint32_t*>(p.scale[set]) + n * p.G + gr)
                                       : (uint32_t)__ldg(static_cast<const unsigned short*>(p.scale[set]) + n * p.G + gr);
                z_raw[h] = (uint32_t)__ldg(p.zp[set] + n * p.zp_row_bytes + (gr >> 1));
            }
        };
        advance(t);
        if (t < n_units)
            ask_params();

        float tot[MB][4];
#pragma unroll
        for (int mb = 0; mb < MB; mb++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                tot[mb][c] = 0.f;
        // y, the addend and the workspace may be the launch ahead's
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int tile = tile_begin, ku = ku_begin, seg_ku0 = ku_begin, st = 0;
        uint32_t phase = 0;
        for (int i = 0; i < n_units; i++)
        {
            if ((i & 3) == 0)
            {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    s_cur[h] = s_raw[h], z_cur[h] = (z_raw[h] >> z_shift) & 0xFu;
                advance(4);
                if (i + 4 + t < n_units)
                    ask_params();
            }
            float sc[2], nz[2];
#pragma unroll
            for (int h = 0; h < 2; h++)
            {
                const uint32_t s = __shfl_sync(0xffffffffu, s_cur[h], (lane & ~3) | (i & 3));
                sc[h] = p.scale_f32 ? __uint_as_float(s) : __half2float(__ushort_as_half((unsigned short)s));
                nz[h] = (float)__shfl_sync(0xffffffffu, z_cur[h], (lane & ~3) | (i & 3));
            }
            if (!wait_warp<0>(full(st), phase, abort_flag))
                break;
            const uint32_t w_off = (uint32_t)(st * kWBytes), x_off = (uint32_t)(st * kBlockBytes);
            const uint4 w[2] = {lds128(w_at[0] + w_off), lds128(w_at[1] + w_off)};
            float acc[MB][4];
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
                uint32_t a[2][4]; // [row half][pair]
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    const uint32_t q = j == 0 ? w[h].x : (j == 1 ? w[h].y : (j == 2 ? w[h].z : w[h].w)), q8 = q >> 8;
                    a[h][0] = and_or<0x000F000Fu>(q, k6400);  // 1024 + (n0, n4)
                    a[h][1] = and_or<0x00F000F0u>(q, k5400);  //   64 + (n1, n5)
                    a[h][2] = and_or<0x000F000Fu>(q8, k6400); // 1024 + (n2, n6)
                    a[h][3] = and_or<0x00F000F0u>(q8, k5400); //   64 + (n3, n7)
                }
#pragma unroll
                for (int mb = 0; mb < MB; mb++)
                {
                    const uint4 x = lds128(x_at + x_off + (uint32_t)((j * kBatch + 8 * mb) * 64));
                    if (j == 0)
                        mma16816_first(acc[mb], a[0][0], a[1][0], a[0][1], a[1][1], x.x, x.y);
                    else
                        mma16816(acc[mb], a[0][0], a[1][0], a[0][1], a[1][1], x.x, x.y);
                    mma16816(acc[mb], a[0][2], a[1][2], a[0][3], a[1][3], x.z, x.w);
                }
            }
#pragma unroll
            for (int mb = 0; mb < MB; mb++)
            {
                const uint4 nc = lds128(nc_at + x_off + (uint32_t)(mb * 64));
#pragma unroll
                for (int c = 0; c < 4; c++)
                {
                    const float nc1 = __uint_as_float(c & 1 ? nc.z : nc.x), nc2 = __uint_as_float(c & 1 ? nc.w : nc.y);
                    tot[mb][c] = fmaf(sc[c >> 1], acc[mb][c] + fmaf(nz[c >> 1], nc2, nc1), tot[mb][c]);
                }
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(empty(st));
            if (++st == kStages)
                st = 0, phase ^= 1u;
            if (ku != KU - 1 && i != n_units - 1)
            {
                ku++;
                continue;
            }
            // ---- the end of this CTA's part of the tile
            if (__any_sync(0xffffffffu, *abort_flag != 0)) // (a role gave up: no stores, no tickets from here on)
                break;
            bool mine = true; // does this warp finish its rows?
            if (seg_ku0 != 0 || ku != KU - 1)
            {
                auto slot = [&](int cta) { return p.slots + (size_t)(p.shares.slot(cta, tile) * kConsumers + warp) * kSums + lane; };
                const int c_first = p.shares.owner(tile * KU), c_last = p.shares.owner(tile * KU + KU - 1);
                float* const my = slot((int)blockIdx.x);
#pragma unroll
                for (int mb = 0; mb < MB; mb++)
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        __stcg(my + (mb * 4 + c) * 32, tot[mb][c]);
                __threadfence();
                __syncwarp();
                uint32_t before = 0;
                if (lane == 0)
                {
                    before = atomicAdd(p.counters + tile * kConsumers + warp, 1u);
                    if (before == (uint32_t)(c_last - c_first))
                        p.counters[tile * kConsumers + warp] = 0u; // leave the counter zeroed for the next call
                }
                before = __shfl_sync(0xffffffffu, before, 0);
                mine = before == (uint32_t)(c_last - c_first);
                if (mine)
                {
                    __threadfence();
#pragma unroll
                    for (int mb = 0; mb < MB; mb++)
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            tot[mb][c] = 0.f;
#pragma unroll 1
                    for (int c0 = c_first; c0 <= c_last; c0 += 4) // four parts' sums in flight
                    {
                        const float* part[4];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            part[e] = slot(min(c0 + e, c_last));
#pragma unroll
                        for (int mb = 0; mb < MB; mb++)
                        {
                            float v[4][4];
#pragma unroll
                            for (int e = 0; e < 4; e++)
#pragma unroll
                                for (int c = 0; c < 4; c++)
                                    v[e][c] = __ldcg(part[e] + (mb * 4 + c) * 32);
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if (c0 + e <= c_last)
#pragma unroll
                                    for (int c = 0; c < 4; c++)
                                        tot[mb][c] += v[e][c];
                        }
                    }
                }
            }
            if (mine)
            {
                const int n0 = p.dual ? tile * 64 + r0 : tile * kRows + r0;
                const int y_shift = p.y_f32 ? 2 : 1;
                auto store = [&](int m, int n, float v) {
                    if (m >= p.M || n >= p.N)
                        return;
                    const size_t at = ((size_t)m * p.N + n) << y_shift;
                    if (p.has_addend)
                    {
                        const char* add = static_cast<const char*>(p.bias) + at;
                        v += p.y_f32 ? *reinterpret_cast<const float*>(add) : __half2float(*reinterpret_cast<const __half*>(add));
                    }
                    else if (p.bias != nullptr)
                        v += static_cast<const float*>(p.bias)[n];
                    char* y = static_cast<char*>(p.y) + at;
                    if (p.y_f32)
                        *reinterpret_cast<float*>(y) = v;
                    else
                        *reinterpret_cast<__half*>(y) = __float2half_rn(v);
                };
#pragma unroll
                for (int mb = 0; mb < MB; mb++)
#pragma unroll
                    for (int c = 0; c < 2; c++)
                    {
                        const int m = 8 * mb + 2 * t + c;
                        if (p.dual)
                        {
                            const float v = tot[mb][c];
                            store(m, n0, v * (1.0f / (1.0f + expf(-v))) * tot[mb][2 + c]);
                        }
                        else
                        {
                            store(m, n0, tot[mb][c]);
                            store(m, n0 + 8, tot[mb][2 + c]);
                        }
                    }
            }
#pragma unroll
            for (int mb = 0; mb < MB; mb++)
#pragma unroll
                for (int c = 0; c < 4; c++)
                    tot[mb][c] = 0.f;
            ku = 0, seg_ku0 = 0, tile++;
        }
    }
    __syncthreads();
    if (tid == 0 && *abort_flag)
        atomicExch(p.status, 1);
}

// 16 bytes that the launch ahead may have written; loads that follow one another stay together
__device__ __forceinline__ uint4 load16(const void* p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// The activations, normalised and rounded, as the blocks that dq_stream_kernel copies (rows past M are zeros).  A block is a unit
// of K: [j][batch row][t] 16 bytes with elements 32 t + 8 j .. + 7 of the unit, in the order 0 4 1 5 2 6 3 7 that the unpacking
// of the weights leaves, then per batch row -sum(offset_k x_k) and -sum(x_k), pairs of rows side by side.  These two are summed by
// the tensor core, in the order and from the fragments of the products, with the offsets alone as the left operand: what the
// accumulator rounds away of 1024 x then goes out with it (weights of q = zp = 0 give exactly 0; summed exactly instead, the error
// of a result against 64 bits grew by an eighth, and by a third for activations of mean 1).A warp takes eight units of a batch row,
// a column of the accumulator each, a CTA 32 units; with the norm every CTA of a row sums up all of its squares, eight loads in
// flight a thread (bound by a few round trips to L2 and the launch; a row whole to one CTA, a load at a time, took 25 us at
// K = 28672).  128 threads, which fit beside two CTAs of the linear.
__global__ void __launch_bounds__(kPrepThreads) stream_prep_kernel(const __half* x, const float* gain, uint8_t* blocks, int M, int K, float eps)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float part[kPrepThreads / 32];
    const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int KU = K / kUnitK;
    const int ub = blockIdx.y * kPrepUnits + 8 * (tid >> 5), u = ub + g; // this warp's first unit and the lane's
    const __half* const row = x + (size_t)m * K;
    uint4 raw[4]; // elements 32 t .. 32 t + 31 of the unit
#pragma unroll
    for (int j = 0; j < 4; j++)
        raw[j] = m < M && u < KU ? load16(row + u * kUnitK + 32 * t + 8 * j) : make_uint4(0u, 0u, 0u, 0u);
    auto floats = [&](const uint4& a, float (&v)[8]) {
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
            v[2 * j] = f.x, v[2 * j + 1] = f.y;
        }
    };
    float r = 1.f;
    if (gain != nullptr)
    {
        float ss = 0.f;
        constexpr int in_flight = 8;
        const int K8 = m < M ? K / 8 : 0;
        for (int i = tid; i < K8; i += in_flight * kPrepThreads)
        {
            uint4 a[in_flight];
#pragma unroll
            for (int e = 0; e < in_flight; e++)
                a[e] = load16(row + (size_t)min(i + e * kPrepThreads, K8 - 1) * 8);
#pragma unroll
            for (int e = 0; e < in_flight; e++)
            {
                float v[8], add = 0.f;
                floats(a[e], v);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    add = fmaf(v[j], v[j], add);
                ss += i + e * kPrepThreads < K8 ? add : 0.f;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0)
            part[tid >> 5] = ss;
        __syncthreads();
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kPrepThreads / 32; w++) // fixed order: repeatable, and the same in every CTA of the row
            sum += part[w];
        r = 1.0f / sqrtf(sum / (float)K + eps);
    }
    float d[4]; // sums with the offsets / plain ones of units ub + 2t and ub + 2t + 1
#pragma unroll
    for (int j = 0; j < 4; j++)
    {
        uint32_t h[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
        if (gain != nullptr && u < KU)
        {
            float v[8];
            floats(raw[j], v);
            const float* const gj = gain + u * kUnitK + 32 * t + 8 * j;
            const float4 a = reinterpret_cast<const float4*>(gj)[0], b = reinterpret_cast<const float4*>(gj)[1];
            const float gn[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const __half2 n = __floats2half2_rn(v[2 * q] * r * gn[2 * q], v[2 * q + 1] * r * gn[2 * q + 1]);
                h[q] = *reinterpret_cast<const uint32_t*>(&n);
            }
        }
        const uint4 f = make_uint4(__byte_perm(h[0], h[2], 0x5410), __byte_perm(h[0], h[2], 0x7632), __byte_perm(h[1], h[3], 0x5410),
                                   __byte_perm(h[1], h[3], 0x7632));
        if (u < KU)
            *reinterpret_cast<uint4*>(blocks + (size_t)u * kBlockBytes + (j * kBatch + m) * 64 + t * 16) = f;
        // rows 0-7 of the left operand: what the unpacking leaves, 1024 on even elements and 64 on odd ones; rows 8-15: ones
        if (j == 0)
            mma16816_first(d, 0x64006400u, 0x3C003C00u, 0x54005400u, 0x3C003C00u, f.x, f.y);
        else
            mma16816(d, 0x64006400u, 0x3C003C00u, 0x54005400u, 0x3C003C00u, f.x, f.y);
        mma16816(d, 0x64006400u, 0x3C003C00u, 0x54005400u, 0x3C003C00u, f.z, f.w);
    }
    if (g == 0)
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (ub + 2 * t + c < KU)
                *reinterpret_cast<float2*>(blocks + (size_t)(ub + 2 * t + c) * kBlockBytes + kBatch * 256 + m * 8) = make_float2(-d[c], -d[2 + c]);
}
} // namespace

namespace nnf
{
// The workspace: the split form's arrival counters, which this form leaves as they are (zero), the slots and the prepared activations
// over that form's partial sums, and this form's counters behind all of what the split form uses.  So both find their counters
// zeroed, in whatever order the calls of a descriptor take one form or the other (the sum over ranks takes the split form).
struct StreamLayout
{
    StreamShares shares;
    size_t slots_at, blocks_at, counters_at, total;
};

static StreamLayout stream_layout(const nnf_b200_ctx* ctx, const nnf_b200_linear_desc& d, const GemvPlan& split)
{
    auto up = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
    StreamLayout L{};
    const int sms = ctx ? ctx->sm_count : 148;
    const bool dual = d.epilogue == NNF_B200_EPILOGUE_SILU_MUL;
    L.shares.set((d.N + (dual ? 63 : 127)) / (dual ? 64 : 128), d.K / kUnitK, 2 * sms);
    L.slots_at = up((size_t)split.row_tiles * sizeof(unsigned));
    L.blocks_at = L.slots_at + (size_t)L.shares.slots() * kConsumers * kSums * sizeof(float);
    L.counters_at = up(std::max(L.blocks_at + (size_t)L.shares.KU * kBlockBytes, split.workspace_bytes));
    L.total = L.counters_at + (L.shares.any_shared() ? (size_t)L.shares.tiles * kConsumers * sizeof(uint32_t) : 0);
    return L;
}

// Whether this form serves a call with enough workspace.  `plan` is the small-M kernel's for the same descriptor: where that would
// cut K into a cluster that the device holds (halves of K, in practice), its sums meet in shared memory and it touches no workspace,
// so that calls of one node on two streams may overlap.  Those stay there, also where this would be faster, as does a K of up to
// 4096, which is not cut (gate/up pair 11008 x 4096 at 16 rows 25.5 / 23.7 us, small-M kernel / this).
// Otherwise by what the small-M kernel makes of the shape: `n` 16-row tiles and weight sets to walk for a warp, and warps of the CTA.
// It is at its best with nearly all of its 16 warps at work and few tiles to walk, where this form pays for many CTAs to a tile.
// Measured at 9, 12 and 16 rows, with and without the norm, 209 shapes of 16 to 194 units per SM of 148 (us at 16 rows without the
// norm, small-M kernel / this; n, warps):
//   4096 x 11008 (7, 11) 19.9 / 18.4, 8192 x 28672 (25, 16) 71.5 / 45.5, 28672 x 8192 pair (50, 16) 120 / 79.5,
//   3936 x 12288 (7, 12) 20.0 / 18.8, 1680 x 11520 pair (6, 12) 17.5 / 16.9;
//   left there: 3344 x 12288 (6, 12) 16.3 / 18.6, 4608 x 9728 (6, 13) 17.2 / 18.5, 672 x 28672 pair (4, 16) 16.6 / 19.2,
//   3104 x 17920 (7, 14) 20.2 / 20.6, 2064 x 28672 with norm (7, 16) 26.9 / 29.0.
// Of the 640 measured calls that this rule admits the slowest takes 0.98 times the small-M kernel's time, on average 0.71; of the
// 183 that it leaves there the fastest would take 0.84.  Fewer than 16 units per SM were not measured.  Up to 8 rows the small-M
// kernel keeps all activations in registers and is faster nearly everywhere.
bool stream_serves(const nnf_b200_ctx* ctx, const nnf_b200_linear_desc& d, const GemvPlan& plan)
{
    const int group = d.group_size > 0 ? d.group_size : d.K;
    if (d.M < 9 || d.M > kBatch || d.w_bits != 4 || d.x_dtype != NNF_B200_F16 || d.split_k != 0 || (d.flags & NNF_B200_FLAG_EXACT_ZP) ||
        d.kernel == NNF_B200_KERNEL_GEMM || d.K % kUnitK != 0 || group % kUnitK != 0 || d.K % group != 0)
        return false;
    const int sms = ctx ? ctx->sm_count : 148;
    const long long KU = d.K / kUnitK, tiles = d.epilogue == NNF_B200_EPILOGUE_SILU_MUL ? (d.N + 63ll) / 64 : (d.N + 127ll) / 128;
    if (tiles * KU >= (1ll << 27) || KU >= (1 << 16)) // (counted in 32 bits)
        return false;
    if (plan.splits <= 1)
        return false;
    if (plan.cluster)
    {
        // Clusters of 2 to 8 one-per-SM CTAs that 148 SMs hold at once (the occupancy calculator's answers, see gemv_direct_plan);
        // CTAs of fewer warps may have twice or four times as many.
        constexpr int held[9] = {0, 0, 74, 45, 33, 26, 22, 15, 15};
        if (plan.ctas_per_split <= held[plan.splits] * std::max(1, std::min(4, 16 / plan.warps)))
            return false;
    }
    const int sets = plan.dual ? 2 : 1, n = sets * ((plan.row_tiles + plan.ctas_per_split - 1) / plan.ctas_per_split);
    return d.K > 4096 && tiles * KU >= 16ll * sms && (plan.warps <= 11 || n >= (d.K <= 15360 ? 8 - sets : 8));
}

size_t stream_workspace_bytes(const nnf_b200_ctx* ctx, const nnf_b200_linear_desc& d, const GemvPlan& plan)
{
    return stream_layout(ctx, d, plan).total;
}

int stream_launch(nnf_b200_ctx* ctx, cudaStream_t stream, const nnf_b200_linear_desc& d, const GemvPlan& plan, const void* x,
                  const nnf_b200_qweight* w, const nnf_b200_qweight* w2, const void* gain, const void* bias, void* y, void* workspace)
{
    static bool configured[kMaxDevices] = {}; // the attributes belong to the device that is current
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= kMaxDevices))
        e = cudaErrorInvalidDevice;
    if (e == cudaSuccess && !configured[dev])
    {
        e = cudaFuncSetAttribute(dq_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(dq_stream_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e == cudaSuccess) // (so that an SM need not drain before it can hold the linear's CTAs)
            e = cudaFuncSetAttribute(stream_prep_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        configured[dev] = e == cudaSuccess;
    }
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("dq_stream set-up: ") + cudaGetErrorString(e));
    const StreamLayout L = stream_layout(ctx, d, plan);
    uint8_t* const ws = static_cast<uint8_t*>(workspace);
    uint8_t* const blocks = ws + L.blocks_at;

    StreamParams p{};
    p.dual = d.epilogue == NNF_B200_EPILOGUE_SILU_MUL;
    const nnf_b200_qweight* sets[2] = {w, p.dual ? w2 : w};
    alignas(64) CUtensorMap tw[2];
    for (int i = 0; i < 2; i++)
    {
        p.scale[i] = sets[i]->scale, p.zp[i] = static_cast<const uint8_t*>(sets[i]->zp);
        if (!weight_tensor_map(ctx, sets[i]->wq, d.N, d.K / 2, kUnitK / 2, p.dual ? 64 : kRows, &tw[i]))
            return set_error(ctx, NNF_B200_ECUDA, "cuTensorMapEncodeTiled failed for the weight tensor");
    }
    p.bias = bias;
    p.has_addend = d.epilogue == NNF_B200_EPILOGUE_ADD;
    p.y = y;
    p.status = ctx->dev_status;
    p.counters = reinterpret_cast<uint32_t*>(ws + L.counters_at);
    p.slots = reinterpret_cast<float*>(ws + L.slots_at);
    p.xblocks = blocks;
    p.M = d.M, p.N = d.N;
    p.shares = L.shares;
    const int group = d.group_size > 0 ? d.group_size : d.K;
    p.G = d.K / group;
    p.zp_row_bytes = (p.G + 1) / 2;
    p.group_units = group / kUnitK;
    p.group_magic = p.group_units > 1 ? (uint32_t)((0x100000000ull + p.group_units - 1) / p.group_units) : 0u;
    p.y_f32 = d.y_dtype == NNF_B200_F32, p.scale_f32 = d.scale_dtype == NNF_B200_F32;

    (void)cudaGetLastError(); // do not inherit a stale error left behind by an unrelated earlier call
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    overlap_attribute(attr, &cfg.numAttrs);
    cfg.attrs = attr;
    cfg.stream = stream;
    cfg.gridDim = dim3(kBatch, (L.shares.KU + kPrepUnits - 1) / kPrepUnits);
    cfg.blockDim = dim3(kPrepThreads);
    e = cudaLaunchKernelEx(&cfg, stream_prep_kernel, static_cast<const __half*>(x), static_cast<const float*>(gain), blocks, (int)d.M, (int)d.K, d.rms_eps);
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("stream_prep launch: ") + cudaGetErrorString(e));
    ctx->launches++;
    cfg.gridDim = dim3(L.shares.ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    e = cudaLaunchKernelEx(&cfg, dq_stream_kernel, p, tw[0], tw[1]);
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("dq_stream launch: ") + cudaGetErrorString(e));
    ctx->launches++;
    return NNF_B200_OK;
}
} // namespace nnf
