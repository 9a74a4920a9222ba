// Large-M (prefill) dequantize-fused linear for sm_100a on the 5th-generation tensor cores.
//
//   y[M,N] = epi( x[M,K] . dequant(W)[N,K]^T )        x fp16, W uint4 / uint8 with group scales and zero-points
//
// Fused replacement of the reference's Convert -> Subtract -> Multiply element-wise kernels that materialise the
// dequantised weights (src/nnfusion/core/kernels/cuda_gpu/kernels/elementwise.hpp:33-157,
// elementwise_fused.cpp:42-189) followed by cublasHgemm / cublasSgemm behind cuda::Dot
// (src/nnfusion/core/kernels/cuda_gpu/kernels/dot.cpp:103-125,264-363).
//
// A tile of the output is computed transposed,  D[256 weight rows, BX batch rows] = Wdq[256, K] . X[BX, K]^T,  by a PAIR
// of CTAs (tcgen05 cta_group::2): each holds 128 of the weight rows and half of the batch rows.  The dequantised weights
// are the A operand and go to the tensor core through TENSOR MEMORY; x is the B operand in shared memory.  A pair, because
// with one CTA per tile the operand that both need from shared memory was what bounded the kernel: a 128 x 256 tile reads
// 64 bytes of x per clock from shared memory while TMA writes another 64, all there is; the pair halves both.
// BX is any multiple of 16 up to 256, so that a ragged batch is cut into equal tiles (333 rows: two of 176, not 512).
// Roles inside a CTA:
//   * warps "W", "X" : one thread each streams raw packed-weight chunks (128 rows x 128 bytes) and this CTA's half of the
//                   x tiles (BX/2 rows x 64 fp16), both 128-byte swizzled, into shared-memory rings;
//   * warps "DQ"  : thread r owns weight row r of the CTA's half = TMEM lane r.  Per 64-element k-block it turns its 32
//                   (uint4) or 64 (uint8) raw bytes into fp16 (q - zp) * scale with the exponent trick (PRMT + LOP3 +
//                   HSUB2 + HMUL2 per pair, exact integer before the scale) and writes the 32 packed registers into the
//                   A stage in TMEM with tcgen05.st.  Groups of four warps share the k-blocks;
//   * warp "MMA"  : one thread of the even CTA issues tcgen05.mma.kind::f16 (256 x BX x 16, fp32 accumulators in both
//                   CTAs' TMEM) and releases stages in both CTAs with tcgen05.commit;
//   * warps "EPI" : eight (four) warps read D with tcgen05.ld, apply bias / addend / SiLU(gate) * up, convert and store y while
//                   the other roles are at the next tile (two accumulators take turns when BX <= 128).
// How a launch's tiles meet the pairs, chosen by the host from an estimate:
//   * whole tiles, dealt out to the pairs;
//   * few tiles: the pairs that share a tile's K are the CTAs of one cluster (2, 3 or 4 pairs) and exchange their partial
//     sums through distributed shared memory, each finishing its share of the batch rows;
//   * otherwise tiles x raw chunks of K in equal shares, so that a tile at a seam is computed by two or more pairs: each
//     writes its fp32 partial sums to a slot of the workspace, and the one that arrives last adds the slots.
// Partial sums are always added in the order of their K ranges: bitwise repeatable.
// SiLU(x . Wg^T) * (x . Wu^T): a tile is the gate's chunks followed by the up projection's; the gate products of a tile
// wait in y (in y's type) for the same threads that wrote them.
// Every mbarrier wait is bounded; on a time-out the CTA raises a status flag, skips its remaining work, and still frees
// its tensor memory.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>

#include "nnf_internal.h"
#include "sm100_ptx.cuh"

namespace
{
using namespace nnf::ptx;

constexpr int kBN = 128;                      // weight rows per CTA (TMEM lanes); a pair's tile has 256
constexpr int kBK = 64;                       // k-block: one 128-byte swizzle row of fp16
constexpr int kWStageBytes = kBN * 128;       // one raw chunk
constexpr int kTmemCols = 512;                // all of it: it starts at column 0
constexpr int kASlotCols = 32;                // a converted k-block in tensor memory: 64 fp16 per lane
constexpr int kMaxPairs = 128;                // pairs of a launch, at most
constexpr int kEpiBarrier = 1;                // named barrier of the epilogue warps

// BX: the most batch rows of a tile, 64, 128 or 256.
// SMALL: tiles of up to 128 batch rows, whose multiplication takes no longer than the conversion of the weights: four
// groups of conversion warps instead of two (about 220 clocks per k-block instead of 380; a k-block of 128 batch rows takes
// the tensor core 256) and a raw ring of 128 KB (160 KB up to 64 batch rows; HBM's latency at full rate is about 100 KB per SM), paid for with half of
// the epilogue warps and a smaller x ring.
// Up to 64 batch rows the two accumulators leave room for 12 converted k-blocks instead of 8, three stages instead of two: a
// stage's conversion, its multiplies and the handing over between them follow one another, and what bounds these tiles is how
// many stages are at it side by side.  With the quantisation parameters hoisted out of the conversion's loop: 48 x 11008 x 4096
// 18.9 -> 17.6 us, the gate/up pair of that shape 35.6 -> 33.2, 48 x 4096 x 11008 19.3 -> 18.8 (graph replay, weights beyond L2).
// (uint4 only: with uint8 weights, whose conversion is shorter, the smaller x ring costs 1 to 3 % at 4096 x 4096.)
// Where the line lies: 65 rows would need accumulators of 80 columns, and 11 k-blocks are two whole stages again.
template <int BX>
struct Cfg
{
    static constexpr bool SMALL = BX <= 128;
    static constexpr int MAX_BX = BX;
    static constexpr int ACC_COLS = SMALL ? BX : 128;    // TMEM columns from one accumulator to the next
    static constexpr int DQ_GROUPS = SMALL ? 4 : 2, DQ_WARPS = 4 * DQ_GROUPS;
    static constexpr int EPI_WARPS = SMALL ? 4 : 8;
    static constexpr int X_WARP = DQ_WARPS + EPI_WARPS, MMA_WARP = X_WARP + 1, W_WARP = X_WARP + 2;
    static constexpr int THREADS = (X_WARP + 4) * 32;    // whole warpgroups: registers are moved between them
    static constexpr int X_BYTES = (BX <= 64 ? 64 : SMALL ? 96 : 128) * 1024; // ring of x tiles: as many stages as fit
    static constexpr int MAX_X_STAGES = 16;
    static constexpr int W_STAGES = BX <= 64 ? 10 : SMALL ? 8 : 6;       // ring of raw chunks
    // A stage is what the tensor core is handed at a time: waits, commits and bookkeeping cost its warp about 500 clocks a
    // stage, whatever the stage holds (with two k-blocks of up to 128 batch rows they set the pace: 445 clocks a k-block).
    static constexpr int STAGE_KB = SMALL ? 4 : 2;       // k-blocks per stage
    static constexpr int A_SLOTS = (kTmemCols - 2 * ACC_COLS) / kASlotCols; // converted k-blocks
    static constexpr int STAGES = A_SLOTS / STAGE_KB;    // ring of stages of converted weights
    // Large tiles: a group converts whole stages, in turn.  Small ones: every group converts one k-block of every stage.
    static constexpr int VISIT_KB = 2, VISIT_STAGES = 2;
    static constexpr int A_COL0 = 2 * ACC_COLS;                   // first TMEM column of the A stages; the accumulators are below
    static constexpr int PACKED = MAX_BX / (EPI_WARPS / 4) / 2; // registers for an epilogue thread's fp16 results
    // full / empty per stage of weights, of x and per raw chunk, full / empty per accumulator, exchange ready / complete
    static constexpr int BARRIERS = 2 * STAGES + 2 * MAX_X_STAGES + 2 * W_STAGES + 6;
    static constexpr size_t SMEM_BYTES =
        1024 + (size_t)X_BYTES + (size_t)W_STAGES * kWStageBytes + BARRIERS * 8 + 64 + 2 * kMaxPairs * sizeof(int);
    // Registers a thread: launched with LAUNCH_REGS each, then the roles take what they need.
    static constexpr int LAUNCH_REGS = SMALL ? 80 : 96;
    static constexpr int DQ_REGS = 72, EPI_REGS = SMALL ? 136 : 144, ISSUE_REGS = SMALL ? 56 : 48;
    static_assert(DQ_GROUPS * DQ_REGS + EPI_WARPS / 4 * EPI_REGS + ISSUE_REGS <= THREADS / 128 * LAUNCH_REGS, "registers the CTA has");
    static_assert(LAUNCH_REGS * THREADS <= 65536, "registers the SM has");
    static_assert(A_COL0 + A_SLOTS * kASlotCols <= kTmemCols, "tensor memory budget");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

struct GemmParams
{
    const void* scale[2];
    const uint8_t* zp[2];
    const float* bias;
    void* y;
    int* status;
    uint32_t* counters; // [2 * tiles] arrivals at the halves of a tile that several pairs share; zero before and after
    float* slots;       // [CTAs][2 * sets][128 * BX] partial sums of shared tiles
    int M, N, K;
    int group, G, zp_row_bytes;
    int y_f32, scale_f32, has_bias;
    int has_addend;  // bias points at an [M,N] tensor of y's type instead of fp32 [N]
    int bx;          // batch rows per tile, a multiple of 16
    int x_stages;    // stages of the x ring
    int m_tiles;     // batch tiles; tile t covers batch tile t % m_tiles of weight-row tile t / m_tiles
    int tiles;       // output tiles in all
    int sets;        // weight sets: 2 for SiLU(gate) * up
    int whole_tiles; // every tile is computed by one pair (no partial sums)
    int ksplit;      // pairs of a cluster that share a tile's K (1: none; then the cluster is the pair)
    int slice;       // ... and the batch rows of the tile that each of them finishes
    int kbpg_shift;  // log2(group / 64) if that is a power of two, else -1
    int cpt;         // raw chunks (the unit of work) per tile and weight set
};

// UMMA shared-memory descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k_sw128(uint32_t smem_addr)
{
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

// A pair's share of the launch: units [u, u_end) of tiles * sets * cpt raw chunks, walked as segments that each lie
// inside one tile and one weight set.  Every role of both CTAs walks the same list.
struct Segment
{
    int tile;     // output tile
    int set;      // weight set
    int c0, c1;   // raw chunks [c0, c1) of the tile
    bool whole;   // the pair computes the tile (both weight sets of it) alone
    bool last;    // the pair's last segment of the tile
};

struct WorkList
{
    int u, u_begin, u_end; // tiles * sets * cpt fits 31 bits (checked on the host)
    __device__ WorkList(const GemmParams& p)
    {
        if (p.ksplit > 1)
        {
            u = u_begin = 0, u_end = p.sets; // this pair's chunks of either weight set
            return;
        }
        const int per_tile = p.sets * p.cpt;
        // whole tiles only: the shares are cut at tile boundaries
        const long long U = p.whole_tiles ? (long long)p.tiles : (long long)p.tiles * per_tile;
        const int scale = p.whole_tiles ? per_tile : 1;
        const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
        u = u_begin = (int)((long long)pair * U / pairs) * scale;
        u_end = (int)((long long)(pair + 1) * U / pairs) * scale;
    }
    __device__ bool next(const GemmParams& p, Segment& s)
    {
        if (u >= u_end)
            return false;
        if (p.ksplit > 1)
        {
            const int pair = blockIdx.x >> 1, part = pair % p.ksplit;
            s.tile = pair / p.ksplit, s.set = u;
            s.c0 = part * p.cpt / p.ksplit, s.c1 = (part + 1) * p.cpt / p.ksplit;
            s.whole = false, s.last = ++u == u_end;
            return true;
        }
        const int per_tile = p.sets * p.cpt;
        s.tile = u / per_tile;
        const int base = s.tile * per_tile, in = u - base;
        s.set = in >= p.cpt ? 1 : 0;
        s.c0 = in - s.set * p.cpt;
        s.c1 = min(p.cpt, s.c0 + (u_end - u));
        s.whole = u_begin <= base && base + per_tile <= u_end;
        u += s.c1 - s.c0;
        s.last = u == u_end || u == base + per_tile;
        return true;
    }
};

// The pair whose share holds unit u: the largest c with floor(c * U / G) <= u.
__device__ __forceinline__ int pair_of_unit(long long u, long long U, int G)
{
    return (int)(((u + 1) * G + U - 1) / U) - 1;
}

// Where a CTA of pair c keeps its partial sum of weight set `set` of tile t: a share has at most two tiles that it does
// not compute alone, its first and its last.
__device__ __forceinline__ int slot_of(const GemmParams& p, int c, int rank, int t, int set, long long U, int G)
{
    const int first_tile = (int)(((long long)c * U / G) / (p.sets * p.cpt));
    return ((2 * c + rank) * 2 + (t == first_tile ? 0 : 1)) * p.sets + set;
}

// A value the compiler must keep as it is: without this it works out 128 addresses ahead of their stores.
__device__ __forceinline__ uint32_t held(uint32_t v)
{
    uint32_t r;
    asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// SiLU(g) = g / (1 + e^-g), ~1e-6 relative; 0 far left
__device__ __forceinline__ float silu(float g)
{
    return g > -80.f ? __fdividef(g, 1.0f + __expf(-g)) : 0.f;
}

// A gate product that waited in y as fp16.  (One that left the fp16 range on its way comes back as the largest fp16
// number, so that SiLU stays finite: SiLU(-inf) would be -inf / inf.)
__device__ __forceinline__ float gate_of_half(uint32_t bits)
{
    return fminf(fmaxf(__half2float(__ushort_as_half((unsigned short)bits)), -65504.f), 65504.f);
}

__device__ __forceinline__ float4 load_part(const float4* p)
{
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Adds up the parts of a tile's half that several pairs computed, in the order of their K ranges, and writes y.  A lane
// keeps four neighbouring weight rows (16-byte loads), a warp takes every WARPS-th batch row; ROWS rows of two parts are
// asked for at a time.  load(set, part, row): a lane's four sums; parts0 / parts1: how many parts either weight set has.
template <int SETS, int ROWS, int WARPS, typename Load>
__device__ __forceinline__ void add_parts(const GemmParams& p, Load load, int parts0, int parts1, int n4, int m0, int rows,
                                          int ew)
{
    if (n4 >= p.N)
        return;
    const bool vec = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15u) == 0 &&
                     (!p.has_addend || (reinterpret_cast<uintptr_t>(p.bias) & 15u) == 0);
    float bias[4];
#pragma unroll
    for (int e = 0; e < 4; e++)
        bias[e] = p.has_bias && n4 + e < p.N ? p.bias[n4 + e] : 0.f;
    for (int row = ew; row < rows; row += ROWS * WARPS)
    {
        float v[SETS][ROWS][4];
#pragma unroll
        for (int set = 0; set < SETS; set++)
        {
#pragma unroll
            for (int j = 0; j < ROWS; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    v[set][j][e] = 0.f;
            // (unconditional loads, past the last part or row of the last one: a choice per load costs a branch per load.  No
            // more of them at a time than registers hold beside the sums: the compiler would take turns)
            const int parts = set == 0 ? parts0 : parts1;
            for (int i = 0; i < parts; i += 2)
            {
                float4 a[2][ROWS];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int j = 0; j < ROWS; j++)
                        a[c][j] = load(set, min(i + c, parts - 1), min(row + j * WARPS, rows - 1));
                const bool two = i + 1 < parts;
#pragma unroll
                for (int j = 0; j < ROWS; j++)
                {
                    v[set][j][0] += a[0][j].x, v[set][j][1] += a[0][j].y, v[set][j][2] += a[0][j].z, v[set][j][3] += a[0][j].w;
                    if (two)
                        v[set][j][0] += a[1][j].x, v[set][j][1] += a[1][j].y, v[set][j][2] += a[1][j].z, v[set][j][3] += a[1][j].w;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < ROWS; j++)
        {
            if (row + j * WARPS >= rows)
                break;
            const size_t at = (size_t)(m0 + row + j * WARPS) * p.N + n4;
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; e++)
            {
                if constexpr (SETS == 2) // (the gate products pass through y's type here too)
                    o[e] = v[1][j][e] * silu(p.y_f32 ? v[0][j][e] : gate_of_half(__half_as_ushort(__float2half_rn(v[0][j][e]))));
                else
                    o[e] = v[0][j][e] + bias[e];
            }
            if (vec)
            {
                if (p.y_f32)
                {
                    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p.has_addend)
                        c = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.bias) + at);
                    *reinterpret_cast<float4*>(static_cast<float*>(p.y) + at) = make_float4(o[0] + c.x, o[1] + c.y, o[2] + c.z, o[3] + c.w);
                }
                else
                {
                    if (p.has_addend)
                    {
                        const uint2 c = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(p.bias) + at);
                        const float2 c0 = __half22float2(*reinterpret_cast<const __half2*>(&c.x));
                        const float2 c1 = __half22float2(*reinterpret_cast<const __half2*>(&c.y));
                        o[0] += c0.x, o[1] += c0.y, o[2] += c1.x, o[3] += c1.y;
                    }
                    const __half2 h0 = __floats2half2_rn(o[0], o[1]), h1 = __floats2half2_rn(o[2], o[3]);
                    uint2 pk;
                    pk.x = *reinterpret_cast<const uint32_t*>(&h0), pk.y = *reinterpret_cast<const uint32_t*>(&h1);
                    *reinterpret_cast<uint2*>(static_cast<__half*>(p.y) + at) = pk;
                }
            }
            else
            {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (n4 + e < p.N)
                    {
                        if (p.has_addend)
                            o[e] += p.y_f32 ? reinterpret_cast<const float*>(p.bias)[at + e]
                                            : __half2float(reinterpret_cast<const __half*>(p.bias)[at + e]);
                        if (p.y_f32)
                            static_cast<float*>(p.y)[at + e] = o[e];
                        else
                            static_cast<__half*>(p.y)[at + e] = __float2half_rn(o[e]);
                    }
            }
        }
    }
}

// ONE_GROUP: two neighbouring k-blocks (of a raw chunk) always lie in one quantisation group.
template <int WBITS, bool ONE_GROUP, int BX>
__global__ void __launch_bounds__(Cfg<BX>::THREADS, 1)
    dq_gemm_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                   const __grid_constant__ CUtensorMap tmap_w1)
{
    using C = Cfg<BX>;
    constexpr int KBC = (WBITS == 4) ? 4 : 2;           // k-blocks per raw chunk
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* xs = base;                                        // [x stages][2][BX / 2 rows][128 B]
    uint8_t* wsm = xs + (size_t)C::X_BYTES;                    // [raw stages][128][128 B]
    uint64_t* bars = reinterpret_cast<uint64_t*>(wsm + (size_t)C::W_STAGES * kWStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::BARRIERS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile uint32_t* ticket_slot = reinterpret_cast<volatile uint32_t*>(tmem_slot + 2);
    int* slot_list = reinterpret_cast<int*>(tmem_slot + 4);    // [2][kMaxPairs]

    const uint32_t bar0 = smem_u32(bars);
    // full_a(q), in the even CTA: the conversion warps of both CTAs have stored the stage's weights (4 warps each per k-block or stage);
    // full_x(q), in the even CTA: both CTAs' x tiles of the stage have landed (TMA transaction bytes);
    // empty_a(q), empty_x(q), in both: the MMAs that read the stage have completed.
    auto full_a = [&](int q) { return bar0 + 8u * q; };
    auto empty_a = [&](int q) { return bar0 + 8u * (C::STAGES + q); };
    auto full_w = [&](int s) { return bar0 + 8u * (2 * C::STAGES + s); };
    auto empty_w = [&](int s) { return bar0 + 8u * (2 * C::STAGES + C::W_STAGES + s); };
    auto acc_full = [&](int b) { return bar0 + 8u * (2 * C::STAGES + 2 * C::W_STAGES + b); };      // in both CTAs
    auto acc_empty = [&](int b) { return bar0 + 8u * (2 * C::STAGES + 2 * C::W_STAGES + 2 + b); }; // in the even CTA
    auto full_x = [&](int q) { return bar0 + 8u * (2 * C::STAGES + 2 * C::W_STAGES + 4 + q); };
    auto empty_x = [&](int q) { return bar0 + 8u * (2 * C::STAGES + 2 * C::W_STAGES + 4 + C::MAX_X_STAGES + q); };

    const uint32_t peers_ready = bar0 + 8u * (C::BARRIERS - 2); // every pair of the cluster has multiplied: the rings are free
    const uint32_t parts_here = bar0 + 8u * (C::BARRIERS - 1);  // every pair's sums of this CTA's batch rows have arrived

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0); // (known to be the same for the whole warp)
    const uint32_t rank = blockIdx.x & 1u;                                    // CTA of the pair
    const uint32_t even = 2u * ((blockIdx.x >> 1) % (uint32_t)p.ksplit);      // the pair's even CTA in the cluster
    const int KB = p.K / kBK;
    const int acc_bufs = p.bx <= 128 ? 2 : 1;
    WorkList work(p);
    Segment sg{};

    // ---------------------------------------------------------------- set-up (once per CTA)
    if (warp == C::X_WARP)
    {
        if (lane == 0)
            prefetch_tensormap(&tmap_x);
        if (lane < C::STAGES)
        {
            mbar_init(full_a(lane), 2 * 4 * (C::STAGE_KB / C::VISIT_KB));
            mbar_init(empty_a(lane), 1);
        }
        if (lane < C::MAX_X_STAGES)
        {
            mbar_init(full_x(lane), 1);
            mbar_init(empty_x(lane), 1);
        }
        if (lane < 2)
        {
            mbar_init(acc_full(lane), 1);
            mbar_init(acc_empty(lane), 2 * C::EPI_WARPS);
        }
        if (lane == 0)
        {
            mbar_init(peers_ready, (uint32_t)p.ksplit);
            mbar_init(parts_here, (uint32_t)(p.ksplit * C::EPI_WARPS));
            *abort_flag = 0;
        }
        fence_barrier_init();
    }
    // Raw weight chunks: the ring belongs to this CTA alone, so that its first round leaves before anything else is set up
    // (set-up takes 3000 clocks, as long as HBM takes to answer).
    uint32_t w_asked = 0; // chunks asked for so far
    auto ask_chunk = [&](const Segment& s, int c) {
        const int st = (int)(w_asked % C::W_STAGES);
        mbar_arrive_expect_tx(full_w(st), kWStageBytes);
        tma_load_2d(smem_u32(wsm + (size_t)st * kWStageBytes), s.set ? &tmap_w1 : &tmap_w0, full_w(st), c * 128,
                    (s.tile / p.m_tiles) * (2 * kBN) + (int)rank * kBN);
        w_asked++;
    };
    int w_next = 0; // the chunk of segment sg to ask for next (warp W)
    bool w_more = false;
    auto next_chunk = [&] {
        if (++w_next == sg.c1)
        {
            w_more = work.next(p, sg);
            w_next = sg.c0;
        }
    };
    if (warp == C::W_WARP && lane == 0)
    {
        for (int s = 0; s < C::W_STAGES; s++)
        {
            mbar_init(full_w(s), 1);
            mbar_init(empty_w(s), 4 * KBC); // (a warp arrives once per k-block)
        }
        fence_barrier_init();
        w_more = work.next(p, sg);
        w_next = sg.c0;
        while (w_more && w_asked < C::W_STAGES)
        {
            ask_chunk(sg, w_next);
            next_chunk();
        }
    }
    if (warp == C::MMA_WARP)
    {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols); // whole warp of both CTAs; the address lands in shared memory
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_arrive(); // the other CTA's barriers are initialised, its tensor memory is allocated
    cluster_wait();
    tcgen05_fence_after();
    constexpr uint32_t tmem_base = 0; // (a constant, so that the multiplies' addresses are known to be the same for all lanes)
    if (tid == 0 && *tmem_slot != tmem_base)
        *abort_flag = 1;
    // Launched as the programmatic dependent of the kernel before it on the stream, this CTA may have started while
    // that kernel's last CTAs were still running.  Weights, scales and zero-points are constants: the raw chunks and the
    // conversion into tensor memory start at once.  The activations, the result, the addend and the workspace may be the
    // earlier kernel's: the thread that loads x waits before its first tile and the epilogue warps before their first
    // segment.  The launch behind this one may be scheduled from here on.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp >= C::X_WARP)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::ISSUE_REGS));
    if (warp == C::W_WARP)
    {
        // ------------------------------------------------------------ TMA producer: raw weight chunks
        // A thread of its own, as for x: either runs as far ahead as its own ring allows.
        if (lane == 0)
            while (w_more)
            {
                if (!wait_or_abort<40>(empty_w(w_asked % C::W_STAGES), ((w_asked / C::W_STAGES) & 1u) ^ 1u, abort_flag))
                    break;
                ask_chunk(sg, w_next);
                next_chunk();
            }
    }
    else if (warp == C::X_WARP)
    {
        // ------------------------------------------------------------ TMA producer: x tiles
        if (lane == 0)
        {
            bool ok = true;
            const int half = p.bx >> 1;
            const uint32_t x_bytes = (uint32_t)half * 128u; // one k-block of this CTA's batch rows
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int q = 0;            // stage ...
            uint32_t phase = 1;   // ... and the parity of its release
            uint32_t x_dst = smem_u32(xs), bar = map_to_rank(full_x(0), even);
            while (ok && work.next(p, sg))
            {
                const int m0 = (sg.tile % p.m_tiles) * p.bx + (int)rank * half;
                const int kb_end = min(KB, sg.c1 * KBC);
                for (int kb = sg.c0 * KBC; kb < kb_end; kb += C::STAGE_KB)
                {
                    ok = wait_or_abort<20>(empty_x(q), phase, abort_flag);
                    if (!ok)
                        break;
                    const int nkb = min(C::STAGE_KB, kb_end - kb);
                    if (rank == 0) // (counted at the even CTA, for both)
                        mbar_arrive_expect_tx(full_x(q), 2u * (uint32_t)nkb * x_bytes);
                    for (int h = 0; h < nkb; h++)
                        tma_load_2d_pair(x_dst + (uint32_t)h * x_bytes, &tmap_x, bar, (kb + h) * kBK, m0);
                    if (++q == p.x_stages)
                        q = 0, phase ^= 1u, x_dst = smem_u32(xs), bar = map_to_rank(full_x(0), even);
                    else
                        x_dst += (uint32_t)C::STAGE_KB * x_bytes, bar += 8u;
                }
            }
        }
    }
    else if (warp == C::MMA_WARP)
    {
        // ------------------------------------------------------------ MMA issuer (even CTA)
        // (the whole warp walks the loop, one elected lane issues)
        if (rank == 0)
        {
            // instruction descriptor: fp32 accumulate, fp16 A and B, both K-major, N = BX, M = 256.  (N: kind::f16 with
            // cta_group::2 and M = 256 takes 16 to 256 in steps of 16.  The PTX ISA's table of tcgen05.mma shapes goes by kind,
            // CTA group and M, not by whether A lies in shared or in tensor memory; every width is held against the oracle in
            // the tests.)
            const uint32_t idesc = (1u << 4) | ((uint32_t)(p.bx >> 3) << 17) | ((uint32_t)((2 * kBN) >> 4) << 24);
            bool ok = true;
            uint32_t si = 0;
            // Ring positions kept as (slot, phase) with the slot's addresses carried along: every instruction not needed
            // between two MMAs is tensor time.
            int q = 0, qx = 0;
            uint32_t phase = 0, phase_x = 0;
            const uint64_t x_block = (uint64_t)(p.bx * 64 >> 4); // one k-block of this CTA's x rows
            const uint64_t xdesc0 = smem_desc_k_sw128(smem_u32(xs));
            const uint32_t a_tmem0 = tmem_base + (uint32_t)C::A_COL0;
            const uint32_t issue = elect_one() ? 1u : 0u;
            const uint16_t pair_mask = (uint16_t)(3u << even);
            uint64_t xdesc = xdesc0;
            uint32_t a_tmem = a_tmem0;
            while (ok && work.next(p, sg))
            {
                const uint32_t b = acc_bufs == 2 ? (si & 1u) : 0u, use = acc_bufs == 2 ? si >> 1 : si;
                // the accumulator still holds an earlier segment until the epilogue warps of both CTAs have read it
                ok = wait_warp<0>(acc_empty(b), (use & 1u) ^ 1u, abort_flag);
                if (!ok)
                    break;
                tcgen05_fence_after();
                const uint32_t d_tmem = tmem_base + b * (uint32_t)C::ACC_COLS;
                uint32_t accumulate = 0u; // the segment's first MMA overwrites D
                const int kb_end = min(KB, sg.c1 * KBC);
                for (int kb = sg.c0 * KBC; kb < kb_end; kb += C::STAGE_KB)
                {
                    ok = wait_warp<0>(full_x(qx), phase_x, abort_flag) && wait_warp<0>(full_a(q), phase, abort_flag);
                    if (!ok)
                        break;
                    tcgen05_fence_after();
                    // (the descriptor's address field counts 16-byte units: k-block and k step are plain additions)
                    auto multiply = [&](int h, uint32_t acc) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; kk++)
                            tcgen05_mma_ts(d_tmem, a_tmem + (uint32_t)(h * kASlotCols + kk * 8), xdesc + (uint64_t)h * x_block + (uint64_t)(kk * 2),
                                           idesc, kk == 0 ? acc : 1u, issue);
                    };
                    multiply(0, accumulate);
                    accumulate = 1u;
                    if (kb + C::STAGE_KB <= kb_end)
                    {
#pragma unroll
                        for (int h = 1; h < C::STAGE_KB; h++)
                            multiply(h, 1u);
                    }
                    else
                    {
#pragma unroll 1
                        for (int h = 1; h < kb_end - kb; h++)
                            multiply(h, 1u);
                    }
                    tcgen05_commit_pair(empty_a(q), pair_mask, issue); // arrives when the MMAs above have consumed the stage
                    tcgen05_commit_pair(empty_x(qx), pair_mask, issue);
                    if (++q == C::STAGES)
                        q = 0, phase ^= 1u, a_tmem = a_tmem0;
                    else
                        a_tmem += C::STAGE_KB * kASlotCols;
                    if (++qx == p.x_stages)
                        qx = 0, phase_x ^= 1u, xdesc = xdesc0;
                    else
                        xdesc += C::STAGE_KB * x_block;
                }
                if (ok)
                    tcgen05_commit_pair(acc_full(b), pair_mask, issue);
                si++;
            }
            // K shared by the cluster's pairs: their plain stores follow where this pair's rings were.  The same kind of
            // arrival that hands a stage back to its producer announces that, here to every CTA of the cluster.  (A release
            // at cluster scope by the epilogue warps cost 0.3 us of 19.4 at 48 x 4096 x 11008.)
            if (ok && p.ksplit > 1)
                tcgen05_commit_pair(peers_ready, (uint16_t)((1u << (2 * p.ksplit)) - 1u), issue);
        }
    }
    else if (warp < C::DQ_WARPS)
    {
        // ------------------------------------------------------------ dequantise into tensor memory
        if constexpr (C::DQ_REGS < C::LAUNCH_REGS)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::DQ_REGS));
        // group g converts k-blocks [2 * part, 2 * part + 2) of every second stage
        const int turn = (warp >> 2) / (C::STAGE_KB / C::VISIT_KB), part = (warp >> 2) % (C::STAGE_KB / C::VISIT_KB);
        const int r = (warp & 3) * 32 + lane;                          // weight row of the CTA's half = TMEM lane
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const int kb_per_group = p.group / kBK;
        const uint32_t row_s = smem_u32(wsm) + (uint32_t)(r * 128);
        const uint32_t col0 = tmem_base + lane_addr + (uint32_t)C::A_COL0;
        const uint32_t full0 = map_to_rank(full_a(0), even); // the even CTA's barriers
        constexpr int VKB = C::VISIT_KB, VST = C::VISIT_STAGES, SKB = C::STAGE_KB;
        // A parity tells a barrier's phase from the one before, no more: a group's next stage must not be two rounds of the
        // A ring ahead, and its raw chunk not two rounds of the raw ring ahead of what has landed (everything up to the
        // stage VISIT_STAGES + STAGES back has been multiplied).
        static_assert(VST <= C::STAGES && (VST + C::STAGES) * SKB <= C::W_STAGES * KBC, "rounds of the rings");
        bool ok = true;
        uint32_t wc_base = 0, st_base = 0; // chunks and stages of this CTA before the segment in hand
        while (ok && work.next(p, sg))
        {
            // This thread's row of scales and of zero-points (rows past N read the last row's, never stored).
            const size_t n = (size_t)min((sg.tile / p.m_tiles) * (2 * kBN) + (int)rank * kBN + r, p.N - 1);
            const char* const sc = static_cast<const char*>(p.scale[sg.set]) + n * p.G * (p.scale_f32 ? 4 : 2);
            const uint8_t* const zp = p.zp[sg.set] + n * p.zp_row_bytes;
            const int kb0 = sg.c0 * KBC, kb_end = min(KB, sg.c1 * KBC), n_st = (kb_end - kb0 + SKB - 1) / SKB;
            // The raw words of the group's next visit are asked for one visit ahead, and nothing touches them before that
            // visit (a move or a conversion right after the load would make the thread sit out the load's latency).
            constexpr int NP = ONE_GROUP ? 1 : VKB; // (scale, zero-point) pairs per visit
            uint32_t s_now[NP], z_now[NP], s_next[NP], z_next[NP];
            int g_now[NP], g_next[NP];
            // the group's first k-block of stage i of the segment
            auto kb_of = [&](int i) { return kb0 + i * SKB + part * VKB; };
            auto ask = [&](int i) {
#pragma unroll
                for (int j = 0; j < NP; j++)
                {
                    const int kb = min(kb_of(i) + j, KB - 1);
                    const int g = p.kbpg_shift >= 0 ? kb >> p.kbpg_shift : kb / kb_per_group;
                    g_next[j] = g;
                    s_next[j] = p.scale_f32 ? __ldg(reinterpret_cast<const uint32_t*>(sc) + g)
                                            : (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(sc) + g);
                    z_next[j] = (uint32_t)__ldg(zp + (WBITS == 4 ? g >> 1 : g));
                }
            };
            const int i_first = (int)(((uint32_t)turn - st_base) & (VST - 1));
            if (i_first < n_st)
                ask(i_first);
            for (int i = i_first; i < n_st; i += VST)
            {
#pragma unroll
                for (int j = 0; j < NP; j++)
                    s_now[j] = s_next[j], z_now[j] = z_next[j], g_now[j] = g_next[j];
                const int kb = kb_of(i), nkb = min(VKB, kb_end - kb); // (nkb <= 0: a short stage has nothing for this group)
                const int chunk = (kb - kb0) / KBC, in_chunk = (kb - kb0) % KBC;
                const uint32_t wc = wc_base + (uint32_t)chunk, sti = st_base + (uint32_t)i;
                const int sw = wc % C::W_STAGES, q = sti % C::STAGES;
                if (nkb > 0)
                {
                    ok = wait_warp<20>(full_w(sw), (wc / C::W_STAGES) & 1u, abort_flag);
                    if (!ok)
                        break;
                }
                if (i + VST < n_st)
                    ask(i + VST);
                // this row's raw bytes: 16-byte piece i of row r is stored at piece i ^ (r & 7)
                const uint32_t row = row_s + (uint32_t)(sw * kWStageBytes);
                const uint32_t col = col0 + (uint32_t)((q * SKB + part * VKB) * kASlotCols);
                ok = wait_warp<20>(empty_a(q), ((sti / C::STAGES) & 1u) ^ 1u, abort_flag);
                if (!ok)
                    break;
                tcgen05_fence_after();
                // Half a k-block: raw bytes -> 32 fp16 (q - zp) * scale in k order (register i holds k = 2i in its low half and
                // k = 2i + 1 in its high half).  (A loop: unrolled over the visit, a fifth of the issue slots went to instruction
                // fetch.  uint4 takes a k-block per trip: half of one, and the quantisation parameters made anew in each, were a
                // sixth of the conversion's instructions.  uint8 takes half of one: a whole one's
                // bytes are eight registers too many, 172 instead of 128 bytes of spills a thread; 128 x 2048 x 8192 18.0 us for 17.7.)
                constexpr int HALVES = WBITS == 4 ? 2 : 1; // of a k-block per trip
                __half2 scale2, zc; // scale; uint4: (1024 + zp, 64 + zp), uint8: 1024 + zp in both halves
                auto set_params = [&](int j) {
                    const uint32_t sraw = s_now[j], zraw = z_now[j];
                    const __half2 from_f32 = __float2half2_rn(__uint_as_float(sraw));
                    const uint32_t s2 = p.scale_f32 ? *reinterpret_cast<const uint32_t*>(&from_f32) : __byte_perm(sraw, 0u, 0x1010);
                    scale2 = *reinterpret_cast<const __half2*>(&s2);
                    const uint32_t zq = WBITS == 4 ? (zraw >> (4 * (g_now[j] & 1))) & 0xFu : zraw;
                    const uint32_t z2 = WBITS == 4 ? (0x6400u | zq) | ((0x5400u | (zq << 4)) << 16) : (0x6400u | zq) * 0x00010001u;
                    zc = *reinterpret_cast<const __half2*>(&z2);
                };
                set_params(0);
#pragma unroll 1
                for (int trip = 0; trip < nkb * (2 / HALVES); trip++)
                {
                    uint4 raw[2];
#pragma unroll
                    for (int v = 0; v < 2; v++)
                        raw[v] = lds128(row + (uint32_t)((((in_chunk * (2 / HALVES) + trip) * 2 + v) ^ (r & 7)) * 16));
                    if (!ONE_GROUP && trip == 2 / HALVES)
                        set_params(NP - 1);
#pragma unroll
                    for (int half = 0; half < HALVES; half++)
                    {
                        uint32_t a[16];
                        if (WBITS == 4)
                        {
                            const uint32_t w4[4] = {raw[half].x, raw[half].y, raw[half].z, raw[half].w};
#pragma unroll
                            for (int wi = 0; wi < 4; wi++)
#pragma unroll
                                for (int b = 0; b < 4; b++)
                                {
                                    // byte b of the word holds elements 2b (bits 0-3) and 2b+1 (bits 4-7)
                                    uint32_t t = __byte_perm(w4[wi], 0u, 0x1111u * b);
                                    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(t) : "r"(t), "n"(0x00F0000Fu), "n"(0x54006400u));
                                    const __half2 h = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&t), zc), scale2);
                                    a[wi * 4 + b] = *reinterpret_cast<const uint32_t*>(&h);
                                }
                        }
                        else
                        {
#pragma unroll
                            for (int v = 0; v < 2; v++)
                            {
                                const uint32_t w4[4] = {raw[v].x, raw[v].y, raw[v].z, raw[v].w};
#pragma unroll
                                for (int wi = 0; wi < 4; wi++)
#pragma unroll
                                    for (int b = 0; b < 2; b++)
                                    {
                                        const uint32_t t = __byte_perm(w4[wi], 0x64646464u, b ? 0x4342 : 0x4140); // 1024 + (b0, b1)
                                        const __half2 h = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&t), zc), scale2);
                                        a[(v * 4 + wi) * 2 + b] = *reinterpret_cast<const uint32_t*>(&h);
                                    }
                            }
                        }
                        tmem_st_32x16(col + (uint32_t)((trip * HALVES + half) * 16), a);
                    }
                }
                tcgen05_wait_st();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0)
                {
                    mbar_arrive_cluster(full0 + 8u * q);
                    // The raw stage goes back to the copy engine only now: the arrival must not be issued before the
                    // shared-memory loads have delivered, and nothing but an instruction that needs their data makes an
                    // instruction wait for them: the tensor-memory stores above consumed every loaded word.  (One arrival
                    // per k-block, also for those that a short last chunk does not have.)
                    if (chunk < sg.c1 - sg.c0)
                        mbar_arrive_n_relaxed(empty_w(sw), SKB == 2 && kb + VKB >= KB ? (uint32_t)(KBC - in_chunk) : (uint32_t)VKB);
                }
            }
            wc_base += (uint32_t)(sg.c1 - sg.c0);
            st_base += (uint32_t)n_st;
        }
    }
    else if (warp < C::X_WARP)
    {
        // ------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::EPI_REGS));
        // D holds y transposed (lane = weight row n, column = batch row m): for one m the 32 lanes of a warp hold 32
        // consecutive n.  Warps 4h .. 4h + 3 take half h of the columns, 16 at a time.
        // With more than 128 batch rows a tile there is one accumulator, and the tensor core waits until it has been read:
        // fp16 results are therefore finished and packed first (up to 64 registers; the gates or the addend that are folded in
        // have been waiting in the same registers), D is handed back, and the stores follow beside the next tile.  (Storing piece
        // by piece held D for 14000 clocks of a tile's 33000; drained like this it is 1700.)
        const int ew = warp - C::DQ_WARPS, half = ew >> 2;
        const int r = (ew & 3) * 32 + lane;
        const uint32_t lane_addr = (uint32_t)((ew & 3) * 32) << 16;
        const int col_mid = C::EPI_WARPS == 4 ? p.bx : (((p.bx >> 4) + 1) >> 1) << 4;
        const int col_begin = half == 0 ? 0 : col_mid, col_end = half == 0 ? col_mid : p.bx;
        const int slot_floats = p.bx * kBN;
        bool ok = true;
        uint32_t si = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory"); // y, the addend and the workspace are touched from here on
        if (p.ksplit > 1)
            ok = false; // (below)
        while (ok && work.next(p, sg))
        {
            const uint32_t b = acc_bufs == 2 ? (si & 1u) : 0u, use = acc_bufs == 2 ? si >> 1 : si;
            si++;
            const int n_base = (sg.tile / p.m_tiles) * (2 * kBN) + (int)rank * kBN, m0 = (sg.tile % p.m_tiles) * p.bx;
            const int n = n_base + r;
            const bool row_ok = n < p.N;
            const int m_end = min(p.bx, p.M - m0); // columns that exist
            const float bias = p.has_bias && row_ok ? p.bias[n] : 0.f;
            const bool gated = sg.set == 1 && sg.whole;
            const uint32_t d_addr = tmem_base + lane_addr + b * (uint32_t)C::ACC_COLS;
            const long long U = (long long)p.tiles * p.sets * p.cpt;
            const int G = (int)(gridDim.x >> 1);
            auto release = [&] { // this warp's last read of D: a later segment may overwrite it
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0)
                    mbar_arrive_cluster(map_to_rank(acc_empty(b), even));
            };
            const int cols = row_ok ? min(m_end, col_end) - col_begin : 0; // this thread's columns that exist
            const size_t at0 = (size_t)(m0 + col_begin) * p.N + n;
            const bool packed = sg.whole && !p.y_f32;
            uint32_t pk[C::PACKED]; // two columns each
            if (packed && (gated || p.has_addend))
            {
                const unsigned short* g = (p.has_addend ? reinterpret_cast<const unsigned short*>(p.bias) : static_cast<const unsigned short*>(p.y)) + at0;
                const uint32_t step = held(2u * (uint32_t)p.N);
#pragma unroll
                for (int i = 0; i < C::PACKED / 8; i++) // sixteen loads in flight
                {
                    uint32_t lo[8], hi[8];
#pragma unroll
                    for (int j = 0; j < 8; j++)
                    {
                        lo[j] = 16 * i + 2 * j < cols ? (uint32_t)*g : 0u;
                        g = reinterpret_cast<const unsigned short*>(reinterpret_cast<const char*>(g) + step);
                        hi[j] = 16 * i + 2 * j + 1 < cols ? (uint32_t)*g : 0u;
                        g = reinterpret_cast<const unsigned short*>(reinterpret_cast<const char*>(g) + step);
                    }
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        pk[8 * i + j] = lo[j] | (hi[j] << 16);
                }
            }
            ok = wait_warp<100>(acc_full(b), use & 1u, abort_flag);
            if (!ok)
                break;
            tcgen05_fence_after();
            if (col_begin == col_end)
                release();
            else if (packed)
            {
                // (what is folded in is decided once per piece: a choice per value costs a branch per value, and the two or
                // three warps of a scheduler do not hide it)
#pragma unroll
                for (int i = 0; i < C::PACKED / 8; i++)
                    if (col_begin + 16 * i < col_end)
                    {
                        uint32_t d[16];
                        tmem_ld_32x16(d_addr + (uint32_t)(col_begin + 16 * i), d);
                        tcgen05_wait_ld();
                        if (col_begin + 16 * i + 16 == col_end)
                            release();
                        if (gated)
                        {
#pragma unroll
                            for (int j = 0; j < 8; j++)
                            {
                                d[2 * j] = __float_as_uint(__uint_as_float(d[2 * j]) * silu(gate_of_half(pk[8 * i + j] & 0xFFFFu)));
                                d[2 * j + 1] = __float_as_uint(__uint_as_float(d[2 * j + 1]) * silu(gate_of_half(pk[8 * i + j] >> 16)));
                            }
                        }
                        else if (p.has_addend)
                        {
#pragma unroll
                            for (int j = 0; j < 8; j++)
                            {
                                const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&pk[8 * i + j]));
                                d[2 * j] = __float_as_uint(__uint_as_float(d[2 * j]) + c.x);
                                d[2 * j + 1] = __float_as_uint(__uint_as_float(d[2 * j + 1]) + c.y);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 8; j++)
                        {
                            const __half2 h = __floats2half2_rn(__uint_as_float(d[2 * j]) + bias, __uint_as_float(d[2 * j + 1]) + bias);
                            pk[8 * i + j] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                    }
                unsigned short* y = static_cast<unsigned short*>(p.y) + at0;
                const uint32_t step = held(2u * (uint32_t)p.N);
#pragma unroll
                for (int j = 0; j < C::PACKED; j++)
                {
                    if (2 * j < cols)
                        *y = (unsigned short)pk[j];
                    y = reinterpret_cast<unsigned short*>(reinterpret_cast<char*>(y) + step);
                    if (2 * j + 1 < cols)
                        *y = (unsigned short)(pk[j] >> 16);
                    y = reinterpret_cast<unsigned short*>(reinterpret_cast<char*>(y) + step);
                }
            }
            else
            {
                float* mine = p.slots + (size_t)(sg.whole ? 0 : slot_of(p, (int)(blockIdx.x >> 1), (int)rank, sg.tile, sg.set, U, G)) * slot_floats +
                              (size_t)col_begin * kBN + r;
                // fp32 results, in pieces of 16 batch rows
                const uint32_t step = held(4u * (uint32_t)p.N);
                char* y = reinterpret_cast<char*>(static_cast<float*>(p.y) + at0);
                // what is combined with the products: the gates, or the addend
                const char* other = reinterpret_cast<const char*>((p.has_addend ? p.bias : static_cast<const float*>(p.y)) + at0);
                for (int col = col_begin; col < col_end; col += 16)
                {
                    const int left = cols - (col - col_begin);
                    float e[16];
                    if (sg.whole && (gated || p.has_addend))
                    {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                        {
                            e[j] = j < left ? *reinterpret_cast<const float*>(other) : 0.f;
                            other += step;
                        }
                    }
                    uint32_t d[16];
                    tmem_ld_32x16(d_addr + (uint32_t)col, d);
                    tcgen05_wait_ld();
                    if (col + 16 == col_end)
                        release();
                    if (!sg.whole)
                    {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            mine[j * kBN] = __uint_as_float(d[j]);
                        mine += 16 * kBN;
                        continue;
                    }
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        v[j] = __uint_as_float(d[j]) + bias;
                    if (gated)
                    {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            v[j] *= silu(e[j]);
                    }
                    else if (p.has_addend)
                    {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            v[j] += e[j];
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++)
                    {
                        if (j < left)
                            *reinterpret_cast<float*>(y) = v[j];
                        y += step;
                    }
                }
            }
            if (!sg.whole && sg.last)
            {
                // All of this pair's sums of the tile are in its slots: take a ticket; the last pair to arrive adds the
                // slots in the order of their K ranges and writes y.
                const int per_tile = p.sets * p.cpt;
                const int c_first = pair_of_unit((long long)sg.tile * per_tile, U, G);
                const int c_last = pair_of_unit((long long)(sg.tile + 1) * per_tile - 1, U, G);
                // the pairs with a part of the first and of the last weight set (the same one when there is one)
                const int set_first[2] = {c_first, p.sets == 1 ? c_first : pair_of_unit((long long)sg.tile * per_tile + p.cpt, U, G)};
                const int set_last[2] = {p.sets == 1 ? c_last : pair_of_unit((long long)sg.tile * per_tile + p.cpt - 1, U, G), c_last};
                __threadfence();
                asm volatile("bar.sync %0, %1;" ::"n"(kEpiBarrier), "n"(C::EPI_WARPS * 32) : "memory");
                if (ew == 0 && lane == 0)
                {
                    const uint32_t before = atomicAdd(p.counters + 2 * sg.tile + rank, 1u);
                    if (before == (uint32_t)(c_last - c_first))
                        p.counters[2 * sg.tile + rank] = 0u; // leave the counter zeroed for the next call
                    *ticket_slot = before;
                }
                // every weight set's slots in the order of their K ranges, once, while the ticket is on its way: the 64-bit
                // divisions behind a slot's place are far dearer than the additions
                for (int set = 0; set < p.sets; set++)
                    for (int i = (ew - 1) * 32 + lane; i >= 0 && i <= set_last[set] - set_first[set]; i += (C::EPI_WARPS - 1) * 32)
                        slot_list[set * kMaxPairs + i] = slot_of(p, set_first[set] + i, (int)rank, sg.tile, set, U, G);
                asm volatile("bar.sync %0, %1;" ::"n"(kEpiBarrier), "n"(C::EPI_WARPS * 32) : "memory");
                if (*ticket_slot == (uint32_t)(c_last - c_first))
                {
                    __threadfence();
                    auto load = [&](int set, int part, int row) {
                        return load_part(reinterpret_cast<const float4*>(p.slots + (size_t)slot_list[set * kMaxPairs + part] * slot_floats) +
                                         row * (kBN / 4) + lane);
                    };
                    const int n0 = set_last[0] - set_first[0] + 1, n1 = set_last[1] - set_first[1] + 1;
                    if (p.sets == 2)
                        add_parts<2, 4, C::EPI_WARPS>(p, load, n0, n1, n_base + 4 * lane, m0, m_end, ew);
                    else
                        add_parts<1, 4, C::EPI_WARPS>(p, load, n0, 0, n_base + 4 * lane, m0, m_end, ew);
                }
                // (nobody touches ticket_slot or slot_list again before everybody has passed the next tile's first barrier,
                // except this tile's slow readers: meet once more)
                asm volatile("bar.sync %0, %1;" ::"n"(kEpiBarrier), "n"(C::EPI_WARPS * 32) : "memory");
            }
        }
        if (p.ksplit > 1)
        {
            // The cluster's pairs have each multiplied their part of K (with two weight sets: both, one per accumulator).
            // Every CTA sends its sums of each peer's batch rows to that peer's shared memory - where the rings were, free
            // once the peer has multiplied - and finishes its own batch rows.
            bool fine = true;
            for (int set = 0; set < p.sets; set++)
                fine = fine && wait_warp<100>(acc_full(set), 0u, abort_flag);
            tcgen05_fence_after();
            const int pair = blockIdx.x >> 1, part = pair % p.ksplit, tile = pair / p.ksplit;
            fine = fine && wait_warp<0, true>(peers_ready, 0u, abort_flag);
            const uint32_t buf = smem_u32(xs); // [set][part][batch row of the slice][128] floats
            if (fine)
            {
                for (int set = 0; set < p.sets; set++)
                    for (int col = col_begin; col < col_end; col += 16)
                    {
                        const int dst = col / p.slice; // (slices are multiples of 16 batch rows)
                        uint32_t d[16];
                        tmem_ld_32x16(tmem_base + lane_addr + (uint32_t)(set * C::ACC_COLS + col), d);
                        const uint32_t to = map_to_rank(buf + (uint32_t)(((set * p.ksplit + part) * p.slice + col - dst * p.slice) * kBN + r) * 4u,
                                                        2u * (uint32_t)dst + rank);
                        tcgen05_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to + (uint32_t)(j * kBN * 4)), "r"(d[j]) : "memory");
                    }
                __syncwarp();
                if (lane < p.ksplit)
                    mbar_arrive_cluster_release(map_to_rank(parts_here, 2u * (uint32_t)lane + rank));
                bool here = false;
                for (uint32_t i = 0; i < kRoleSpin && !here && !*abort_flag; i++)
                    here = mbar_try_wait_cluster(parts_here, 0u);
                fine = __all_sync(0xffffffffu, here);
            }
            if (fine)
            {
                const int n_base = (tile / p.m_tiles) * (2 * kBN) + (int)rank * kBN, m0 = (tile % p.m_tiles) * p.bx + part * p.slice;
                const int rows = min(min(p.slice, p.bx - part * p.slice), p.M - m0);
                auto load = [&](int set, int pt, int row) {
                    const uint4 v = lds128(buf + (uint32_t)(((set * p.ksplit + pt) * p.slice + row) * kBN + 4 * lane) * 4u);
                    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
                };
                if (rows > 0)
                {
                    if (p.sets == 2)
                        add_parts<2, 4, C::EPI_WARPS>(p, load, p.ksplit, p.ksplit, n_base + 4 * lane, m0, rows, ew);
                    else
                        add_parts<1, 4, C::EPI_WARPS>(p, load, p.ksplit, 0, n_base + 4 * lane, m0, rows, ew);
                }
            }
            else
                *abort_flag = 1;
        }
    }

    // ---------------------------------------------------------------- tear-down
    tcgen05_fence_before();
    __syncthreads();
    cluster_arrive(); // nobody of the pair reaches into the other's shared or tensor memory any more
    cluster_wait();
    if (warp == C::MMA_WARP)
    {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (tid == 0 && *abort_flag)
        atomicExch(p.status, 1);
}

// Pre-pass for activations the tensor-core kernel does not take as they are: fp32 rows are rounded to fp16, and with
// the RMSNorm prologue every row is scaled by rsqrt(mean(x^2) + eps) * gain on the way (fp32 arithmetic, one
// rounding).  One CTA per row, 16-byte accesses, the whole row (up to 8192 elements; the rest is read again) asked for at
// once and kept in registers.  Bound by HBM; with scalar loads in two rounds 2000 rows of 6016 fp16 took 50 us, now 13.
// Replaces the reference's Multiply -> Sum -> Divide -> Add -> Rsqrt -> Multiply chain in front of the Dot
// (reduce: src/nnfusion/core/kernels/cuda_gpu/kernels/reduce.hpp:18-600) and its Convert.
template <bool XF32>
__global__ void __launch_bounds__(256) prep_activations_kernel(const void* x, const float* gain, __half* out, int K,
                                                               float eps)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float part[8];
    constexpr int kStep = 256 * 8, kKept = 4; // elements per step of the CTA, steps kept in registers
    const size_t row = (size_t)blockIdx.x * K;
    const int k0 = threadIdx.x * 8;
    auto load = [&](int k, float (&v)[8]) {
        if (XF32)
        {
            const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(x) + row + k);
            const float4 a = src[0], b = src[1];
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        }
        else
        {
            const uint4 a = *reinterpret_cast<const uint4*>(static_cast<const __half*>(x) + row + k);
            const __half2* h = reinterpret_cast<const __half2*>(&a);
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
                const float2 f = __half22float2(h[j]);
                v[2 * j] = f.x, v[2 * j + 1] = f.y;
            }
        }
    };
    float kept[kKept][8];
#pragma unroll
    for (int s = 0; s < kKept; s++)
        if (k0 + s * kStep < K) // (K is a multiple of 64)
            load(k0 + s * kStep, kept[s]);
    float r = 1.f;
    if (gain != nullptr)
    {
        float ss = 0.f;
#pragma unroll
        for (int s = 0; s < kKept; s++)
            if (k0 + s * kStep < K)
#pragma unroll
                for (int j = 0; j < 8; j++)
                    ss = fmaf(kept[s][j], kept[s][j], ss);
        for (int k = k0 + kKept * kStep; k < K; k += kStep)
        {
            float v[8];
            load(k, v);
#pragma unroll
            for (int j = 0; j < 8; j++)
                ss = fmaf(v[j], v[j], ss);
        }
        for (int o = 16; o > 0; o >>= 1)
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if ((threadIdx.x & 31) == 0)
            part[threadIdx.x >> 5] = ss;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) // fixed order: repeatable
            tot += part[w];
        r = 1.0f / sqrtf(tot / (float)K + eps);
    }
    auto store = [&](int k, const float (&v)[8]) {
        float g[8];
        if (gain != nullptr)
        {
            const float4 a = reinterpret_cast<const float4*>(gain + k)[0], b = reinterpret_cast<const float4*>(gain + k)[1];
            g[0] = a.x, g[1] = a.y, g[2] = a.z, g[3] = a.w, g[4] = b.x, g[5] = b.y, g[6] = b.z, g[7] = b.w;
        }
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const float lo = gain != nullptr ? v[2 * j] * r * g[2 * j] : v[2 * j], hi = gain != nullptr ? v[2 * j + 1] * r * g[2 * j + 1] : v[2 * j + 1];
            const __half2 q = __floats2half2_rn(lo, hi);
            h[j] = *reinterpret_cast<const uint32_t*>(&q);
        }
        *reinterpret_cast<uint4*>(out + row + k) = make_uint4(h[0], h[1], h[2], h[3]);
    };
#pragma unroll
    for (int s = 0; s < kKept; s++)
        if (k0 + s * kStep < K)
            store(k0 + s * kStep, kept[s]);
    for (int k = k0 + kKept * kStep; k < K; k += kStep)
    {
        float v[8];
        load(k, v);
        store(k, v);
    }
}

// Launched as a programmatic dependent like the linear behind it, which starts on its weights meanwhile; with the shared
// memory carve-out that the linear wants, so that an SM need not drain before it can hold one of its CTAs.
template <bool XF32>
cudaError_t launch_prep(const void* x, const float* gain, __half* out, int M, int K, float eps, cudaStream_t stream)
{
    static bool configured[nnf::kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= nnf::kMaxDevices)
        return cudaErrorInvalidDevice;
    if (!configured[dev])
    {
        e = cudaFuncSetAttribute(prep_activations_kernel<XF32>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess)
            return e;
        configured[dev] = true;
    }
    (void)cudaGetLastError();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    nnf::overlap_attribute(attr, &cfg.numAttrs);
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, prep_activations_kernel<XF32>, x, gain, out, K, eps);
}

template <int WBITS, bool ONE_GROUP, int BX>
cudaError_t launch(const GemmParams& p, const CUtensorMap& tx, const CUtensorMap& tw0, const CUtensorMap& tw1, int pairs,
                   cudaStream_t stream)
{
    using C = Cfg<BX>;
    static bool configured[nnf::kMaxDevices] = {}; // the attribute belongs to the device that is current
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= nnf::kMaxDevices)
        return cudaErrorInvalidDevice;
    if (!configured[dev])
    {
        e = cudaFuncSetAttribute(dq_gemm_kernel<WBITS, ONE_GROUP, BX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_BYTES);
        if (e != cudaSuccess)
            return e;
        configured[dev] = true;
    }
    (void)cudaGetLastError();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    nnf::overlap_attribute(attr, &cfg.numAttrs);
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = 2u * (unsigned)p.ksplit;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    cfg.numAttrs++;
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, dq_gemm_kernel<WBITS, ONE_GROUP, BX>, p, tx, tw0, tw1);
}

template <int BX>
cudaError_t dispatch(int wbits, bool one_group, const GemmParams& p, const CUtensorMap& tx, const CUtensorMap& tw0,
                     const CUtensorMap& tw1, int pairs, cudaStream_t stream)
{
    if (wbits == 4)
        return one_group ? launch<4, true, BX>(p, tx, tw0, tw1, pairs, stream) : launch<4, false, BX>(p, tx, tw0, tw1, pairs, stream);
    if constexpr (BX > 64)
        return one_group ? launch<8, true, BX>(p, tx, tw0, tw1, pairs, stream) : launch<8, false, BX>(p, tx, tw0, tw1, pairs, stream);
    return cudaErrorInvalidValue;
}
} // namespace

namespace nnf
{
// fp32 activations and the RMSNorm prologue go through a pre-pass that writes fp16 [M,K] into the workspace.
static bool needs_prepass(const nnf_b200_linear_desc& d)
{
    return d.x_dtype == NNF_B200_F32 || d.prologue == NNF_B200_PROLOGUE_RMSNORM;
}

// How a launch is laid out (see the top of this file).  The workspace holds, for tiles shared through it, the arrival
// counters of the tiles' halves and partial-sum slots of every CTA; and, when needed, the fp16 copy of x.
struct GemmLayout
{
    int bx, m_tiles, n_tiles, tiles, sets, cpt, pairs, whole_tiles, ksplit;
    size_t counter_bytes, slot_bytes, prepass_bytes;
    size_t total() const { return counter_bytes + slot_bytes + prepass_bytes; }
};

// Tiles shared through the workspace: counters for both halves of every tile, and slots of 128 x BX for two tiles per CTA
// and weight set.
static size_t shared_counter_bytes(int tiles)
{
    return ((size_t)2 * tiles * sizeof(uint32_t) + 255) / 256 * 256;
}
static size_t shared_slot_bytes(int pairs, int sets, int bx)
{
    return (size_t)2 * pairs * 2 * sets * 128 * bx * sizeof(float);
}

// room: bytes that counters and slots may take.
static GemmLayout gemm_layout(const nnf_b200_ctx* ctx, const nnf_b200_linear_desc& d, size_t room = SIZE_MAX)
{
    GemmLayout L{};
    const int sms = ctx ? ctx->sm_count : 148;
    const int max_pairs = std::min(std::max(1, sms / 2), kMaxPairs);
    // clusters of 1, 2, 3 and 4 pairs that 148 SMs hold at once (the occupancy calculator's answers; a launch of more of
    // them would only take longer)
    const int held[5] = {0, max_pairs, max_pairs * 33 / 74, max_pairs * 22 / 74, max_pairs * 15 / 74};
    L.n_tiles = (d.N + 255) / 256;
    L.sets = d.epilogue == NNF_B200_EPILOGUE_SILU_MUL ? 2 : 1;
    const int kb_per_chunk = d.w_bits == 4 ? 4 : 2;
    L.cpt = (d.K / 64 + kb_per_chunk - 1) / kb_per_chunk;
    // Batch tiles of equal width and how K is shared, by an estimate that ranks the choices: its constants were fitted to 20
    // shapes of 32 to 4096 batch rows times every choice, without what all choices share (the launch, the first loads, the
    // last stores), so that the microseconds themselves come out 20 to 40 % low (4096 x 11008 x 4096: 227 for 320 measured;
    // 48 x 4096 x 11008: 13.9 for 18.4; fitted when tiles of up to 64 rows had two stages of converted weights, and not again since
    // they have three).  What a k-block takes: up to 128 batch rows the conversion of the weights (and handing it over), 0.19 to 0.24; above, where two groups of warps convert, 0.31 to 0.345.  Whole tiles cost whole waves.
    // Partial sums through the workspace (store, ticket, read back) cost 9 to 26 us, inside a cluster 1 to 4 us.
    const double kb = (double)d.K / 64.0 * L.sets;
    auto pairs_of = [&](int tiles, bool whole) {
        return (int)std::min<long long>(whole ? tiles : (long long)tiles * L.sets * L.cpt, max_pairs);
    };
    double best = 0;
    const int m_min = (d.M + 255) / 256;
    for (int mt = m_min; mt <= m_min * 2 + 2 && mt <= (d.M + 15) / 16; mt++)
    {
        const int bx = ((d.M + mt - 1) / mt + 15) / 16 * 16; // 16 to 256: m_min tiles are no wider
        const int m_tiles = (d.M + bx - 1) / bx, tiles = m_tiles * L.n_tiles;
        const double t_kb = bx <= 128 ? 0.19 + 0.0004 * bx : 0.25 + 0.00037 * bx, out = (double)bx * L.sets;
        const double tile = kb * t_kb + 0.5 + 3.0 * (L.sets - 1);
        auto take = [&](double t, int whole, int ksplit) {
            if (best == 0 || t < best)
                best = t, L.bx = bx, L.m_tiles = m_tiles, L.whole_tiles = whole, L.ksplit = ksplit;
        };
        take(std::ceil((double)tiles / max_pairs) * tile + 0.004 * out, 1, 1);
        if (shared_counter_bytes(tiles) + shared_slot_bytes(pairs_of(tiles, false), L.sets, bx) <= room)
            take(std::max((double)tiles / max_pairs, 1.0 / L.cpt) * tile + 6.0 + (tiles < max_pairs ? 0.08 : 0.05) * out, 0, 1);
        for (int s = 2; s <= 4 && s <= L.cpt; s++)
            if (tiles <= held[s] && (L.sets == 1 || bx <= 128))
                take((double)((L.cpt + s - 1) / s) * kb_per_chunk * L.sets * t_kb + 1.0 + 0.008 * out, 0, s);
    }
    L.tiles = L.m_tiles * L.n_tiles;
    L.pairs = L.ksplit > 1 ? L.tiles * L.ksplit : pairs_of(L.tiles, L.whole_tiles);
    if (!L.whole_tiles && L.ksplit == 1)
    {
        L.counter_bytes = shared_counter_bytes(L.tiles);
        L.slot_bytes = shared_slot_bytes(L.pairs, L.sets, L.bx);
    }
    L.prepass_bytes = needs_prepass(d) ? ((size_t)d.M * d.K * sizeof(__half) + 255) / 256 * 256 : 0;
    return L;
}

size_t gemm_workspace_bytes(const nnf_b200_ctx* ctx, const nnf_b200_linear_desc& d)
{
    return gemm_layout(ctx, d).total();
}

int gemm_supported(const nnf_b200_ctx*, const nnf_b200_linear_desc& d, std::string* why)
{
    const int group = d.group_size > 0 ? d.group_size : d.K;
    if (d.K % 64 != 0 || group % 64 != 0 || d.K % group != 0)
    {
        *why = "K and group_size must be multiples of 64 and K a multiple of group_size";
        return NNF_B200_ENOTSUP;
    }
    if ((d.w_bits == 4 ? d.K / 2 : d.K) % 16 != 0)
    {
        *why = "weight rows must be a multiple of 16 bytes";
        return NNF_B200_ENOTSUP;
    }
    // the kernel counts its units of work (tiles x weight sets x raw chunks of K) in 32-bit integers
    const long long tiles = (long long)((d.M + 255) / 256 + 4) * ((d.N + 127) / 128);
    const long long chunks = 2 * ((d.K / 64 + (d.w_bits == 4 ? 3 : 1)) / (d.w_bits == 4 ? 4 : 2));
    if (tiles * chunks >= (1ll << 31) || tiles >= (1ll << 29))
    {
        *why = "M * N * K is beyond what one launch counts";
        return NNF_B200_ENOTSUP;
    }
    return NNF_B200_OK;
}

int gemm_launch(nnf_b200_ctx* ctx, cudaStream_t stream, const nnf_b200_linear_desc& d, const void* x,
                const nnf_b200_qweight* w, const nnf_b200_qweight* w2, const void* gain, const void* bias, void* y,
                void* workspace, size_t workspace_bytes)
{
    GemmLayout L = gemm_layout(ctx, d);
    if (L.total() > 0 && (!workspace || workspace_bytes < L.prepass_bytes))
        return set_error(ctx, NNF_B200_EWORKSPACE,
                         "workspace of " + std::to_string(L.total()) +
                             " bytes required (tile counters, partial sums of shared tiles, fp16 copy of the activations)");
    // A smaller one (a program that was generated when this shape asked for less) takes the best layout that it holds.
    if (workspace_bytes < L.total())
        L = gemm_layout(ctx, d, workspace_bytes - L.prepass_bytes);
    if (reinterpret_cast<uintptr_t>(workspace) & 15u)
        return set_error(ctx, NNF_B200_EALIGN, "the workspace must be 16-byte aligned");
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    if (needs_prepass(d))
    {
        __half* xh = reinterpret_cast<__half*>(ws + L.counter_bytes + L.slot_bytes);
        const float* g = d.prologue == NNF_B200_PROLOGUE_RMSNORM ? static_cast<const float*>(gain) : nullptr;
        const cudaError_t pe = d.x_dtype == NNF_B200_F32 ? launch_prep<true>(x, g, xh, d.M, d.K, d.rms_eps, stream)
                                                         : launch_prep<false>(x, g, xh, d.M, d.K, d.rms_eps, stream);
        if (pe != cudaSuccess)
            return set_error(ctx, NNF_B200_ECUDA, std::string("prep_activations launch: ") + cudaGetErrorString(pe));
        ctx->launches++;
        x = xh;
    }
    const bool silu_mul = d.epilogue == NNF_B200_EPILOGUE_SILU_MUL;
    const int row_bytes = d.w_bits == 4 ? d.K / 2 : d.K;
    const int cfg = L.bx <= 64 && d.w_bits == 4 ? 64 : L.bx <= 128 ? 128 : 256;
    GemmParams p{};
    p.y = y;
    p.status = ctx->dev_status;
    p.M = d.M, p.N = d.N, p.K = d.K;
    p.group = d.group_size > 0 ? d.group_size : d.K;
    p.G = d.K / p.group;
    p.zp_row_bytes = d.w_bits == 4 ? (p.G + 1) / 2 : p.G;
    p.y_f32 = d.y_dtype == NNF_B200_F32;
    p.scale_f32 = d.scale_dtype == NNF_B200_F32;
    p.bx = L.bx;
    const int x_ring = cfg == 64 ? Cfg<64>::X_BYTES : cfg == 128 ? Cfg<128>::X_BYTES : Cfg<256>::X_BYTES;
    p.x_stages = std::min(Cfg<64>::MAX_X_STAGES, x_ring / (L.bx * 64 * (cfg <= 128 ? Cfg<128>::STAGE_KB : Cfg<256>::STAGE_KB)));
    p.m_tiles = L.m_tiles;
    p.tiles = L.tiles;
    p.sets = L.sets;
    p.cpt = L.cpt;
    p.whole_tiles = L.whole_tiles;
    p.ksplit = L.ksplit;
    p.slice = ((L.bx >> 4) + L.ksplit - 1) / L.ksplit * 16;
    p.counters = reinterpret_cast<uint32_t*>(ws);
    p.slots = reinterpret_cast<float*>(ws + L.counter_bytes);
    p.has_addend = d.epilogue == NNF_B200_EPILOGUE_ADD;
    p.has_bias = bias != nullptr && !p.has_addend && !silu_mul;
    p.bias = static_cast<const float*>(bias);
    const nnf_b200_qweight* sets[2] = {w, silu_mul ? w2 : w};
    for (int i = 0; i < 2; i++)
    {
        p.scale[i] = sets[i]->scale;
        p.zp[i] = static_cast<const uint8_t*>(sets[i]->zp);
    }
    p.kbpg_shift = -1;
    for (int sh = 0; sh < 31; sh++)
        if ((p.group / 64) == (1 << sh))
            p.kbpg_shift = sh;
    const bool one_group = p.group % 128 == 0 || p.group == d.K;

    // x: fp16 [M][K], boxes of BX/2 rows x 64 elements (the tensor map is not cached: x moves between calls)
    alignas(64) CUtensorMap tx;
    if (!encode_tensor_map_2d(ctx->encode_tiled, &tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)d.K,
                              (uint64_t)d.M, (uint64_t)d.K * 2, 64, (uint32_t)L.bx / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return set_error(ctx, NNF_B200_ECUDA, "cuTensorMapEncodeTiled failed for the activations");
    alignas(64) CUtensorMap tw[2];
    for (int i = 0; i < 2; i++)
    {
        if (!weight_tensor_map(ctx, sets[i]->wq, d.N, row_bytes, 128, 128, &tw[i]))
            return set_error(ctx, NNF_B200_ECUDA, "cuTensorMapEncodeTiled failed for the weight tensor");
    }
    const cudaError_t e = cfg == 64    ? dispatch<64>(d.w_bits, one_group, p, tx, tw[0], tw[1], L.pairs, stream)
                          : cfg == 128 ? dispatch<128>(d.w_bits, one_group, p, tx, tw[0], tw[1], L.pairs, stream)
                                       : dispatch<256>(d.w_bits, one_group, p, tx, tw[0], tw[1], L.pairs, stream);
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("dq_gemm launch: ") + cudaGetErrorString(e));
    ctx->launches++;
    return NNF_B200_OK;
}
} // namespace nnf
