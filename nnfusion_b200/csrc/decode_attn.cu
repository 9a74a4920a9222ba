// Single-token (decode) attention over a key/value cache for sm_100a, with the rotary embedding of q and of the new
// key and the append of the new key/value row fused in:
//     out[h] = softmax(rot(q[h]) . K[kv(h)]^T * scale) . V[kv(h)],   K/V rows 0 .. position (the new row included).
//
// In the reference this is a chain of separate kernels: Slice / Negative / Concat / Multiply / Add for the rotary
// embedding (element-wise emitters, src/nnfusion/core/kernels/cuda_gpu/kernels/elementwise.hpp:33-157), a strided-batched
// cuBLAS GEMM for q.K^T (src/nnfusion/core/kernels/cuda_gpu/kernels/batch_matmul.cpp:49-144, adj_y), Softmax
// (src/nnfusion/core/kernels/cuda_gpu/kernels/softmax.cpp:78-122) and a second batched GEMM for P.V; the BERT-style
// fused Attention op (src/nnfusion/core/kernels/cuda_gpu/kernels/attention.cpp:13-152) stops at 1024 positions.
//
// The kernel is HBM-bound as long as a cache row is read once for ALL query heads that share it and its two products
// cost next to nothing.  Both run on mma.sync.m16n8k16 with the cache rows as the 16-row operand and up to 8 query heads
// as the 8-column operand (a group of more than 8 takes several blocks of 8):
//   S^T[16 rows, 8 q] = K[16 rows, 128] . Q^T        O^T[128, 8 q] += V^T[128, 16 rows] . P^T[16 rows, 8 q]
// The contraction index of either product may be numbered freely as long as both operands agree, so a warp takes K and V
// straight from global memory into fragments with 16-byte loads, without shared memory: a lane of K's operand owns 8
// neighbouring dimensions of a row, a lane of V's owns 8 neighbouring dimensions of four rows (pairs of rows meet in one
// register by PRMT).  q and the weights P go in as fp16 hi + lo (22 bits), so precision is that of fp32 dot products.
// One CTA of 12 warps per SM: every warp keeps its own running maximum / sum / O over every 12th block of 16 rows with
// the next block's 8 KB on its way (96 KB in flight per SM); the warps meet once, in shared memory.
// Positions are cut into `splits` ranges per key/value head.  Up to 8 ranges are the CTAs of a thread-block cluster and
// meet in the first one's shared memory; more store their partial results, take a ticket, and the CTA that arrives last
// combines them.  Either way the order is fixed, so results are bitwise repeatable, and no CTA waits for one that may not
// be running.
// What bounds it: the chain wait -> queries (1 us) -> rows -> meeting (0.5 us) -> ranges (1 to 3 us); the rows themselves
// come at 85 GB/s per SM.
// (64 query heads on 8 key/value heads, 8192 rows, 33.6 MB, in a chain of launches: 45.0 us with one CTA per query head and
// FFMA dot products, which read every row eight times and were bound by instructions; 11.4 us now.  32 heads of their own,
// 2049 rows, 33.6 MB: 11.5 -> 9.1 us.)
// Infinities: an infinite key makes its score infinite, an infinite value its dimension of the result; the lo halves are kept
// from making NaN of either (where scores are formed, and sum_infinite_values).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <string>

#include "nnf_internal.h"

namespace
{
constexpr int kD = 128;       // head dimension
constexpr int kWarps = 12;    // 168 registers a thread: 12 warps fill an SM's register file
constexpr int kFewWarps = 4;  // for a sequence of a few rows that is not cut: less to launch and to add up
constexpr int kRows = 16;     // cache rows per warp and step
constexpr int kQ = 8;         // query heads per CTA
constexpr int kSlot = kQ * (kD + 2); // floats per (head block, split): weighted value sums, maxima, sums
constexpr int kQPitch = kD + 32; // elements per row of queries in shared memory: 16-byte reads of eight rows without conflicts
constexpr int kMaxCluster = 8; // ranges that may form a cluster
constexpr int kMaxSplits = 512; // the ranges' weights fit where the warps' O was
constexpr int kPartBytes = kWarps * kQ * kD * (int)sizeof(float); // the warps' O in shared memory

constexpr int kSmemBytes = kPartBytes + kMaxCluster * kSlot * (int)sizeof(float);
static_assert(kMaxSplits * kQ * 2 * (int)sizeof(float) <= kPartBytes, "weights of the ranges");

struct AttnParams
{
    const __half* q;     // [heads][128], before the rotary embedding
    const __half* k_new; // [kv_heads][128], before the rotary embedding
    const __half* v_new; // [kv_heads][128]
    __half* k_cache;     // [kv_heads][capacity][128]
    __half* v_cache;
    __half* out;         // [heads][128]
    float* ws_part;      // [head blocks][splits][kSlot]
    unsigned* ws_count;  // [head blocks]
    int heads, kv_heads, group, qblocks, capacity, position, splits, chunk, rotary;
    int cluster; // the ranges of a head block are one thread-block cluster: their parts meet in shared memory
    float scale, log2_base; // scale: softmax scale * log2(e)
};

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v)
{
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint4 load_once(const __half* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t h2bits(__half2 h)
{
    return *reinterpret_cast<uint32_t*>(&h);
}
// Two floats as fp16 hi + lo pairs.  (hi saturates, so that a value beyond fp16's range leaves the excess to lo.)
__device__ __forceinline__ void split_hi_lo(float x, float y, uint32_t& hi, uint32_t& lo)
{
    const float cx = fminf(fmaxf(x, -65504.f), 65504.f), cy = fminf(fmaxf(y, -65504.f), 65504.f);
    const __half2 h = __floats2half2_rn(cx, cy);
    const float2 f = __half22float2(h);
    hi = h2bits(h);
    lo = h2bits(__floats2half2_rn(x - f.x, y - f.y));
}
__device__ __forceinline__ uint32_t word(const uint4& v, int i)
{
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

// A query's sums over the rows [begin, end) once more, four dimensions a lane: an infinite value (one that left the fp16
// range) times a weight's lo half is of either sign or NaN.  Here scores and weights are fp32, so that the sums are infinite,
// or NaN if they have to be.  m: what the weights are taken against; qh, ql: the query's halves; knew: the new key.
// Called by a whole warp, and rarely.
__device__ __forceinline__ float4 sum_infinite_values(const AttnParams& p, int kvh, int begin, int end, float m, const __half* qh,
                                                      const __half* ql, const __half* knew)
{
    const int d = 4 * (threadIdx.x & 31);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int row = begin; row < end; row++)
    {
        const size_t at = ((size_t)kvh * p.capacity + row) * kD + d;
        const bool is_new = row == p.position;
        const __half* const k = is_new ? knew + d : p.k_cache + at;
        const __half* const v = is_new ? p.v_new + (size_t)kvh * kD + d : p.v_cache + at;
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++)
            s = fmaf(__half2float(qh[d + j]) + __half2float(ql[d + j]), __half2float(k[j]), s);
#pragma unroll
        for (int x = 1; x < 32; x <<= 1)
            s += __shfl_xor_sync(0xffffffffu, s, x);
        const float w = exp2f(s * p.scale - m);
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[j] = fmaf(w, __half2float(v[j]), acc[j]);
    }
    return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) decode_attention_kernel(const AttnParams p)
{
    constexpr int kThreads = WARPS * 32, kPass = WARPS * kRows;
    extern __shared__ __align__(16) float part_s[]; // [warp][query][128], at the end
    __shared__ __align__(16) __half qh_s[kQ][kQPitch], ql_s[kQ][kQPitch]; // rotated queries, fp16 hi + lo
    __shared__ float cs_s[2][kD / 2];               // cosines and sines of this position
    __shared__ __align__(16) __half knew_s[kD];     // the new key row as it is stored in the cache
    __shared__ float m_s[WARPS][kQ], l_s[WARPS][kQ], f_s[WARPS][kQ];
    __shared__ float mcta_s[kQ];
    __shared__ int last_s;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int block = blockIdx.y, split = blockIdx.x;
    const int kvh = block / p.qblocks, qb = block - kvh * p.qblocks;
    const int head0 = kvh * p.group + qb * kQ;             // first query head of the block
    const int nq = min(kQ, p.group - qb * kQ);             // query heads that exist
    const int n_rows = p.position + 1;
    const int begin = split * p.chunk, end = min(begin + p.chunk, n_rows);
    const bool owns_new = begin <= p.position && p.position < end;
    // Before anything else, and before the launch ahead of this one has finished: ask for the CTA's whole range of
    // both caches to be brought into L2 (a prefetch hands no values to anyone, so it may run ahead of the wait below).
    // HBM then streams from the first microsecond, and the register loads further down see L2 latency.
    if (tid == 0 && end > begin && qb == 0)
    {
        const size_t first = ((size_t)kvh * p.capacity + begin) * kD;
        const uint32_t bytes = (uint32_t)(end - begin) * kD * (uint32_t)sizeof(__half);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.k_cache + first), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.v_cache + first), "r"(bytes) : "memory");
    }
    // A CTA's shared memory may be written from its cluster's other CTAs only once it runs: everybody arrives here and
    // waits before the first such write.
    if (p.cluster)
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    // Rotary embedding, "rotate half": pairs (i, i + 64) are rotated by position * base^(-2i/128).
    if (p.rotary && tid < kD / 2)
    {
        const float inv_freq = exp2f(-(float)(2 * tid) / (float)kD * p.log2_base);
        float sn, cs;
        sincosf((float)p.position * inv_freq, &sn, &cs);
        cs_s[0][tid] = cs, cs_s[1][tid] = sn;
    }
    // The next launch on the stream may start as SMs become free; this one waits for the launch before it (which
    // produced q, k, v; the cache rows it reads were written by earlier steps, but nothing is assumed about those).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- the queries' few bytes, which everything waits for, leave first, then the first block of rows (behind 12 warps'
    // row loads the queries came back 1.5 us later)
    // (lane = 4 neighbouring dimensions of a query)
    constexpr int kQPer = (kQ + WARPS - 1) / WARPS; // a warp takes a query
    const int pd = 4 * lane;
    uint2 qa[kQPer], qb2[kQPer]; // ... and the dimensions they are rotated with
#pragma unroll
    for (int n = 0; n < kQPer; n++)
    {
        const int pq = warp + n * WARPS;
        const __half* x = p.q + (size_t)(head0 + min(pq, nq - 1)) * kD;
        qa[n] = *reinterpret_cast<const uint2*>(x + pd), qb2[n] = *reinterpret_cast<const uint2*>(x + (pd ^ 64));
        if (pq >= nq)
            qa[n] = qb2[n] = make_uint2(0u, 0u);
    }
    const __half* const kbase = p.k_cache + (size_t)kvh * p.capacity * kD + 8 * t;
    const __half* const vbase = p.v_cache + (size_t)kvh * p.capacity * kD + 8 * g;
    uint4 kr[2][4]; // rows g, g + 8; dimensions 32c + 8t .. + 7
    uint4 vr[4][2]; // rows 2t, 2t + 1, 2t + 8, 2t + 9; dimensions 64h + 8g .. + 7
    // Rows past the end of the range read as zeros; the new row is not in the cache yet and is patched in when used.
    auto load_k = [&](int row0) {
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
            const int row = row0 + g + 8 * i;
            const bool live = row < end && row != p.position;
#pragma unroll
            for (int c = 0; c < 4; c++)
                kr[i][c] = live ? load_once(kbase + (size_t)row * kD + 32 * c) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    auto load_v = [&](int row0) {
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            const int row = row0 + 2 * t + (i & 1) + 8 * (i >> 1);
            const bool live = row < end && row != p.position;
#pragma unroll
            for (int h = 0; h < 2; h++)
                vr[i][h] = live ? load_once(vbase + (size_t)row * kD + 64 * h) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    int row0 = begin + warp * kRows;
    if (row0 < end)
        load_k(row0), load_v(row0);

    // ---- queries (and, in the CTA whose range holds the new row, the new key) through the rotary embedding
    __syncthreads(); // cs_s
    auto rotated = [&](__half xa, __half xb, int d) {
        const float a = __half2float(xa), b = __half2float(xb);
        if (!p.rotary)
            return a;
        const float cs = cs_s[0][d & 63], sn = cs_s[1][d & 63];
        return d < 64 ? a * cs - b * sn : a * cs + b * sn;
    };
#pragma unroll
    for (int n = 0; n < kQPer; n++)
    {
        const int pq = warp + n * WARPS;
        if (pq >= kQ)
            break;
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int r = 0; r < 2; r++)
        {
            const __half2 a = *reinterpret_cast<const __half2*>(r == 0 ? &qa[n].x : &qa[n].y);
            const __half2 b = *reinterpret_cast<const __half2*>(r == 0 ? &qb2[n].x : &qb2[n].y);
            split_hi_lo(rotated(__low2half(a), __low2half(b), pd + 2 * r),
                        rotated(__high2half(a), __high2half(b), pd + 2 * r + 1), hi[r], lo[r]);
        }
        *reinterpret_cast<uint2*>(&qh_s[pq][pd]) = make_uint2(hi[0], hi[1]);
        *reinterpret_cast<uint2*>(&ql_s[pq][pd]) = make_uint2(lo[0], lo[1]);
    }
    if (owns_new && tid < kD)
    {
        const __half* kx = p.k_new + (size_t)kvh * kD;
        const __half kn = __float2half_rn(rotated(kx[tid], kx[tid ^ 64], tid));
        knew_s[tid] = kn;
        // append: every block of a group writes the same values
        p.k_cache[((size_t)kvh * p.capacity + p.position) * kD + tid] = kn;
        p.v_cache[((size_t)kvh * p.capacity + p.position) * kD + tid] = p.v_new[(size_t)kvh * kD + tid];
    }
    __syncthreads();
    uint4 qh[4], ql[4]; // per 32 dimensions: [k step][register]
#pragma unroll
    for (int c = 0; c < 4; c++)
        qh[c] = *reinterpret_cast<const uint4*>(&qh_s[g][32 * c + 8 * t]), ql[c] = *reinterpret_cast<const uint4*>(&ql_s[g][32 * c + 8 * t]);

    // ---- running softmax over the warp's blocks of rows; this lane's columns are queries 2t and 2t + 1
    // (m_ref starts at the lowest finite number: rows of score -inf weigh nothing, also before the first finite one)
    float m_ref[2] = {-FLT_MAX, -FLT_MAX}, l_run[2] = {0.f, 0.f};
    float o[2][4][4]; // [64 dimensions][pair of dimensions][dimension 8g + 2j: queries 2t, 2t + 1; 8g + 2j + 1: likewise]
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                o[h][j][e] = 0.f;
    for (; row0 < end; row0 += kPass)
    {
        const bool has_new = owns_new && p.position >= row0 && p.position < row0 + kRows;
        if (has_new)
        {
#pragma unroll
            for (int i = 0; i < 2; i++)
                if (row0 + g + 8 * i == p.position)
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        kr[i][c] = *reinterpret_cast<const uint4*>(knew_s + 32 * c + 8 * t);
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (row0 + 2 * t + (i & 1) + 8 * (i >> 1) == p.position)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        vr[i][h] = *reinterpret_cast<const uint4*>(p.v_new + (size_t)kvh * kD + 64 * h + 8 * g);
        }
        // rows g (queries 2t, 2t + 1) and g + 8; four chains of products, added below
        float s4[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f}, sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int s = 0; s < 2; s++)
            {
                const uint32_t a0 = word(kr[0][c], 2 * s), a2 = word(kr[0][c], 2 * s + 1);
                const uint32_t a1 = word(kr[1][c], 2 * s), a3 = word(kr[1][c], 2 * s + 1);
                mma16816(s == 0 ? s4 : sb, a0, a1, a2, a3, word(qh[c], 2 * s), word(qh[c], 2 * s + 1));
                mma16816(s == 0 ? sc : sd, a0, a1, a2, a3, word(ql[c], 2 * s), word(ql[c], 2 * s + 1));
            }
        const int next = row0 + kPass;
        if (next < end)
            load_k(next);
        // (A score whose hi part is infinite already - a key that left the fp16 range, a row masked by infinities - is that: lo
        // is of either sign or zero, and its product with the infinity would make a NaN of it.)
#pragma unroll
        for (int e = 0; e < 4; e++)
        {
            const float hi = s4[e] + sb[e], sum = fabsf(hi) == INFINITY ? hi : hi + (sc[e] + sd[e]);
            s4[e] = row0 + g + 8 * (e >> 1) < end ? sum * p.scale : -INFINITY;
        }
        // Largest score per query over the block.  The reference value that the exponents are taken against follows only
        // when a score exceeds it by more than 2^8: until then nothing has to be rescaled, and the weights (at most 256)
        // stay well inside fp16.
        float mx[2] = {fmaxf(s4[0], s4[2]), fmaxf(s4[1], s4[3])};
#pragma unroll
        for (int x = 4; x <= 16; x <<= 1)
#pragma unroll
            for (int c = 0; c < 2; c++)
                mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], x));
        if (__any_sync(0xffffffffu, mx[0] > m_ref[0] + 8.f || mx[1] > m_ref[1] + 8.f))
        {
            float corr[2];
#pragma unroll
            for (int c = 0; c < 2; c++)
            {
                const float m = mx[c] > m_ref[c] + 8.f ? mx[c] : m_ref[c];
                corr[c] = exp2f(m_ref[c] - m); // 0 on the first block
                m_ref[c] = m;
                l_run[c] *= corr[c];
            }
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        o[h][j][e] *= corr[e & 1];
        }
        float w[4];
#pragma unroll
        for (int e = 0; e < 4; e++)
        {
            w[e] = exp2f(s4[e] - m_ref[e & 1]); // 0 for rows past the end
            l_run[e & 1] += w[e];
        }
        // P^T as the 8-column operand: rows go from the lane's g to its t
        uint32_t ph[2], pl[2];
#pragma unroll
        for (int i = 0; i < 2; i++)
        {
            uint32_t hi, lo;
            split_hi_lo(w[2 * i], w[2 * i + 1], hi, lo);
            ph[i] = transpose8x8(hi), pl[i] = transpose8x8(lo);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
                const uint32_t w0 = word(vr[0][h], j), w1 = word(vr[1][h], j);
                const uint32_t w2 = word(vr[2][h], j), w3 = word(vr[3][h], j);
                const uint32_t a0 = __byte_perm(w0, w1, 0x5410), a1 = __byte_perm(w0, w1, 0x7632);
                const uint32_t a2 = __byte_perm(w2, w3, 0x5410), a3 = __byte_perm(w2, w3, 0x7632);
                mma16816(o[h][j], a0, a1, a2, a3, ph[0], ph[1]);
                mma16816(o[h][j], a0, a1, a2, a3, pl[0], pl[1]);
            }
        if (next < end)
            load_v(next);
    }

    // ---- the warps meet: weights per (warp, query) first, then sums in warp order
#pragma unroll
    for (int x = 4; x <= 16; x <<= 1)
#pragma unroll
        for (int c = 0; c < 2; c++)
            l_run[c] += __shfl_xor_sync(0xffffffffu, l_run[c], x);
    if (g == 0)
    {
#pragma unroll
        for (int c = 0; c < 2; c++)
            m_s[warp][2 * t + c] = m_ref[c], l_s[warp][2 * t + c] = l_run[c];
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int c = 0; c < 2; c++)
                *reinterpret_cast<float2*>(part_s + (warp * kQ + 2 * t + c) * kD + 64 * h + 8 * g + 2 * j) =
                    make_float2(o[h][j][c], o[h][j][2 + c]);
    __syncthreads();
    if (tid < WARPS * kQ) // the warps' weights, once: thread = (warp, query)
    {
        const int qi = tid % kQ;
        float m = m_s[0][qi];
#pragma unroll
        for (int w = 1; w < WARPS; w++)
            m = fmaxf(m, m_s[w][qi]);
        f_s[tid / kQ][qi] = exp2f(m_s[tid / kQ][qi] - m); // (a warp without rows has sums of zero)
        if (tid < kQ)
            mcta_s[qi] = m;
    }
    __syncthreads();
    float* const mine = p.ws_part + ((size_t)block * p.splits + split) * kSlot;
    float* const slots_s = part_s + WARPS * kQ * kD; // [range][kSlot] of the cluster's first CTA
    uint32_t remote = 0;
    if (p.cluster)
    {
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(remote)
                     : "r"((uint32_t)__cvta_generic_to_shared(slots_s) + (uint32_t)split * (kSlot * 4u)), "r"(0));
    }
    for (int i = tid; i < nq * (kD / 4); i += kThreads) // four dimensions of one query
    {
        const int qi = i / (kD / 4), d4 = i % (kD / 4);
        float l = 0.f;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < WARPS; w++)
        {
            const float f = f_s[w][qi];
            const float4 x = *reinterpret_cast<const float4*>(part_s + (w * kQ + qi) * kD + 4 * d4);
            l = fmaf(l_s[w][qi], f, l);
            v.x = fmaf(x.x, f, v.x), v.y = fmaf(x.y, f, v.y), v.z = fmaf(x.z, f, v.z), v.w = fmaf(x.w, f, v.w);
        }
        if (__any_sync(0xffffffffu, isnan((v.x + v.y) + (v.z + v.w)))) // (a warp has the 32 pieces of one query)
        {
            const float4 e = sum_infinite_values(p, kvh, begin, end, mcta_s[qi], qh_s[qi], ql_s[qi], knew_s);
            v.x = isnan(v.x) ? e.x : v.x, v.y = isnan(v.y) ? e.y : v.y, v.z = isnan(v.z) ? e.z : v.z, v.w = isnan(v.w) ? e.w : v.w;
        }
        if (p.splits == 1)
        {
            uint2 pk;
            pk.x = h2bits(__floats2half2_rn(v.x / l, v.y / l)), pk.y = h2bits(__floats2half2_rn(v.z / l, v.w / l));
            *reinterpret_cast<uint2*>(p.out + (size_t)(head0 + qi) * kD + 4 * d4) = pk;
        }
        else if (p.cluster)
        {
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote + (uint32_t)(qi * kD + 4 * d4) * 4u),
                         "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                         : "memory");
            if (d4 == 0)
                asm volatile("st.shared::cluster.f32 [%0], %1;\n\tst.shared::cluster.f32 [%2], %3;" ::"r"(remote + (uint32_t)(kQ * kD + qi) * 4u),
                             "f"(mcta_s[qi]), "r"(remote + (uint32_t)(kQ * kD + kQ + qi) * 4u), "f"(l)
                             : "memory");
        }
        else
        {
            __stcg(reinterpret_cast<float4*>(mine + qi * kD) + d4, v);
            if (d4 == 0)
            {
                __stcg(mine + kQ * kD + qi, mcta_s[qi]);
                __stcg(mine + kQ * kD + kQ + qi, l);
            }
        }
    }
    if (WARPS < kQ || p.splits == 1) // (the few-warps form is launched for uncut sequences only)
        return;
    if (p.cluster)
    {
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        if (split != 0)
            return;
        for (int i = tid; i < nq * (kD / 4); i += kThreads)
        {
            const int qi = i / (kD / 4), d4 = i % (kD / 4);
            float m = -INFINITY, l = 0.f;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int s = 0; s < p.splits; s++)
                m = fmaxf(m, slots_s[s * kSlot + kQ * kD + qi]);
            for (int s = 0; s < p.splits; s++) // fixed order: repeatable; an empty range adds zero times zero
            {
                const float* part = slots_s + s * kSlot;
                const float f = exp2f(part[kQ * kD + qi] - m);
                const float4 x = *reinterpret_cast<const float4*>(part + qi * kD + 4 * d4);
                l = fmaf(part[kQ * kD + kQ + qi], f, l);
                v.x = fmaf(x.x, f, v.x), v.y = fmaf(x.y, f, v.y), v.z = fmaf(x.z, f, v.z), v.w = fmaf(x.w, f, v.w);
            }
            uint2 pk;
            pk.x = h2bits(__floats2half2_rn(v.x / l, v.y / l)), pk.y = h2bits(__floats2half2_rn(v.z / l, v.w / l));
            *reinterpret_cast<uint2*>(p.out + (size_t)(head0 + qi) * kD + 4 * d4) = pk;
        }
        return;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0)
    {
        const unsigned old = atomicAdd(p.ws_count + block, 1u);
        last_s = old == (unsigned)(p.splits - 1);
        if (last_s)
            p.ws_count[block] = 0u; // leave the counter zeroed for the next call
    }
    __syncthreads();
    if (!last_s)
        return;
    __threadfence();
    // The parts of the first 16 ranges and every range's maximum and sum are asked for at once (the warps' shared memory
    // is free again for the latter), then the sums follow in the order of the ranges: repeatable.
    static_assert(WARPS < kQ || kQ * (kD / 4) <= kThreads, "one position per thread");
    const float* const parts = p.ws_part + (size_t)block * p.splits * kSlot;
    const int qi = tid / (kD / 4), d4 = tid % (kD / 4);
    const float* const my_part = parts + min(qi, kQ - 1) * kD + 4 * d4;
    constexpr int kBatch = 16;
    float4 x[kBatch];
#pragma unroll
    for (int s = 0; s < kBatch; s++)
        x[s] = s < p.splits && qi < nq ? __ldcg(reinterpret_cast<const float4*>(my_part + (size_t)s * kSlot)) : make_float4(0.f, 0.f, 0.f, 0.f);
    float* const wm_s = part_s;                      // [split][query] maxima, then weights
    float* const wl_s = part_s + p.splits * kQ;      // [split][query] sums
    for (int i = tid; i < p.splits * kQ; i += kThreads)
    {
        const float* part = parts + (size_t)(i / kQ) * kSlot + kQ * kD + i % kQ;
        wm_s[i] = __ldcg(part), wl_s[i] = __ldcg(part + kQ);
    }
    __syncthreads();
    if (warp < nq)
    {
        float m = -INFINITY;
        for (int s = lane; s < p.splits; s += 32)
            m = fmaxf(m, wm_s[s * kQ + warp]);
#pragma unroll
        for (int o2 = 1; o2 < 32; o2 <<= 1)
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o2));
        for (int s = lane; s < p.splits; s += 32)
            wm_s[s * kQ + warp] = exp2f(wm_s[s * kQ + warp] - m); // 0 for an empty range
    }
    __syncthreads();
    if (qi >= nq)
        return;
    float l = 0.f;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < p.splits; s0 += kBatch)
    {
        if (s0 > 0)
        {
#pragma unroll
            for (int s = 0; s < kBatch; s++)
                if (s0 + s < p.splits)
                    x[s] = __ldcg(reinterpret_cast<const float4*>(my_part + (size_t)(s0 + s) * kSlot));
        }
#pragma unroll
        for (int s = 0; s < kBatch; s++)
            if (s0 + s < p.splits)
            {
                const float f = wm_s[(s0 + s) * kQ + qi];
                l = fmaf(wl_s[(s0 + s) * kQ + qi], f, l);
                v.x = fmaf(x[s].x, f, v.x), v.y = fmaf(x[s].y, f, v.y), v.z = fmaf(x[s].z, f, v.z), v.w = fmaf(x[s].w, f, v.w);
            }
    }
    uint2 pk;
    pk.x = h2bits(__floats2half2_rn(v.x / l, v.y / l)), pk.y = h2bits(__floats2half2_rn(v.z / l, v.w / l));
    *reinterpret_cast<uint2*>(p.out + (size_t)(head0 + qi) * kD + 4 * d4) = pk;
}

// A sequence of up to 32 rows, one CTA of four warps per query head: a lane has 8 dimensions of one row per round, so that all
// rows are in registers at once, the products are fp32, and the rows are added up in one go.  It is a chain of dependent
// steps throughout, and this is the shortest one (the rows of shared key/value heads come from L2): 1 to 32 rows 1.5 us in a
// chain of launches, where the kernel above takes 2.9 to 3.1.
constexpr int kShortRows = 32;
constexpr int kShortThreads = 128;
__global__ void __launch_bounds__(kShortThreads) short_attention_kernel(const AttnParams p)
{
    constexpr int kRounds = kShortRows / 8; // a round is 8 rows: two a warp, 16 lanes each
    __shared__ __align__(16) float q_s[kD]; // rotated query, times the softmax scale
    __shared__ __align__(16) __half knew_s[kD];
    __shared__ float red_s[4][kD], m_s[4], l_s[4];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int half = lane >> 4, dg = lane & 15; // which of the warp's two rows, which 8 dimensions
    const int head = blockIdx.x, kvh = head / p.group;
    const int rows = p.position + 1;
    const size_t cache0 = (size_t)kvh * p.capacity * kD;
    if (tid == 0)
    {
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.k_cache + cache0), "r"(rows * kD * 2) : "memory");
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.v_cache + cache0), "r"(rows * kD * 2) : "memory");
    }
    float cs = 1.f, sn = 0.f; // of dimensions tid and tid ^ 64
    if (p.rotary)
        sincosf((float)p.position * exp2f(-(float)(2 * (tid & 63)) / (float)kD * p.log2_base), &sn, &cs);
    if (tid < 64)
        sn = -sn;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const __half* const q = p.q + (size_t)head * kD;
    const __half* const kx = p.k_new + (size_t)kvh * kD;
    const __half* const vx = p.v_new + (size_t)kvh * kD;
    const __half qa = q[tid], qb = q[tid ^ 64], ka = kx[tid], kb = kx[tid ^ 64], vn = vx[tid];
    uint4 kr[kRounds], vr[kRounds];
    auto row_of = [&](int r) { return r * 8 + warp * 2 + half; };
#pragma unroll
    for (int r = 0; r < kRounds; r++)
    {
        const size_t at = cache0 + (size_t)row_of(r) * kD + 8 * dg;
        const bool live = row_of(r) < p.position; // (the new row is patched in below)
        kr[r] = live ? load_once(p.k_cache + at) : make_uint4(0u, 0u, 0u, 0u);
        vr[r] = live ? load_once(p.v_cache + at) : make_uint4(0u, 0u, 0u, 0u);
    }
    auto rotated = [&](__half a, __half b) {
        return p.rotary ? fmaf(__half2float(b), sn, __half2float(a) * cs) : __half2float(a);
    };
    q_s[tid] = rotated(qa, qb) * p.scale;
    const __half kn = __float2half_rn(rotated(ka, kb));
    knew_s[tid] = kn;
    // append: every head of a group writes the same values
    p.k_cache[cache0 + (size_t)p.position * kD + tid] = kn;
    p.v_cache[cache0 + (size_t)p.position * kD + tid] = vn;
    __syncthreads();
    float qv[8];
    *reinterpret_cast<float4*>(qv) = *reinterpret_cast<const float4*>(q_s + 8 * dg);
    *reinterpret_cast<float4*>(qv + 4) = *reinterpret_cast<const float4*>(q_s + 8 * dg + 4);
    float s[kRounds], m = -INFINITY;
#pragma unroll
    for (int r = 0; r < kRounds; r++)
    {
        if (row_of(r) == p.position)
        {
            kr[r] = *reinterpret_cast<const uint4*>(knew_s + 8 * dg);
            vr[r] = *reinterpret_cast<const uint4*>(vx + 8 * dg);
        }
        const __half2* k = reinterpret_cast<const __half2*>(&kr[r]);
        float d = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const float2 f = __half22float2(k[j]);
            d = fmaf(qv[2 * j], f.x, d), d = fmaf(qv[2 * j + 1], f.y, d);
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1)
            d += __shfl_xor_sync(0xffffffffu, d, x);
        s[r] = row_of(r) < rows ? d : -INFINITY;
        m = fmaxf(m, s[r]);
    }
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
    if (lane == 0)
        m_s[warp] = m;
    __syncthreads();
    m = fmaxf(fmaxf(m_s[0], m_s[1]), fmaxf(m_s[2], m_s[3]));
    float l = 0.f, acc[8];
#pragma unroll
    for (int j = 0; j < 8; j++)
        acc[j] = 0.f;
#pragma unroll
    for (int r = 0; r < kRounds; r++)
    {
        const float w = exp2f(s[r] - m); // 0 for rows past the end
        l += w;
        const __half2* v = reinterpret_cast<const __half2*>(&vr[r]);
#pragma unroll
        for (int j = 0; j < 4; j++)
        {
            const float2 f = __half22float2(v[j]);
            acc[2 * j] = fmaf(w, f.x, acc[2 * j]), acc[2 * j + 1] = fmaf(w, f.y, acc[2 * j + 1]);
        }
    }
    // the two rows of a warp, then the four warps
    l += __shfl_xor_sync(0xffffffffu, l, 16);
#pragma unroll
    for (int j = 0; j < 8; j++)
        acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
    if (half == 0)
    {
        *reinterpret_cast<float4*>(&red_s[warp][8 * dg]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        *reinterpret_cast<float4*>(&red_s[warp][8 * dg + 4]) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    }
    if (lane == 0)
        l_s[warp] = l;
    __syncthreads();
    const float sum = (red_s[0][tid] + red_s[1][tid]) + (red_s[2][tid] + red_s[3][tid]);
    p.out[(size_t)head * kD + tid] = __float2half_rn(sum / ((l_s[0] + l_s[1]) + (l_s[2] + l_s[3])));
}

int head_blocks(const nnf_b200_attn_desc& d)
{
    return d.kv_heads * ((d.heads / d.kv_heads + kQ - 1) / kQ);
}

// Ranges per head block, one CTA per SM.  Up to 8 ranges meet in the shared memory of a cluster (about 1 us), more in the
// workspace (about 3 us: store, fence, ticket, read back).  Measured: a sequence of up to 128 rows is fastest uncut (128 rows,
// 8 heads on 8: 4.20 us, 2 ranges 4.59, 3 ranges 4.40, 4 ranges 4.36; 64 on 8: 4.46, 4.92, 4.76, 4.77); a
// range pays from 64 rows on (563 rows on 2 key/value heads: 3 ranges 6.2 us, 8 ranges 5.3 us, since one SM takes in no
// more than about 85 GB/s); up to about 600 rows a range the cluster wins (4097 rows on 8 heads: 8 ranges 9.2 us, 16
// through the workspace 9.6 us; 8192 rows: 16.0 and 13.1 us), beyond that as many ranges as one wave holds, of 256 rows at
// least.
int pick_splits(const nnf_b200_ctx* ctx, const nnf_b200_attn_desc& d)
{
    const int sms = ctx ? ctx->sm_count : 148;
    const int rows = d.position + 1;
    if (d.splits > 0)
        return std::min(std::min(d.splits, std::max(1, rows / 16)), kMaxSplits);
    const int wave = std::max(1, sms / head_blocks(d));
    if (rows <= 128 || wave == 1)
        return 1;
    // clusters of n one-per-SM CTAs that the 148 SMs hold at once (the occupancy calculator's answers; the launch asks
    // again and falls back to the workspace)
    static const int held[kMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    int in_cluster = std::min(wave, kMaxCluster);
    while (in_cluster > 1 && held[in_cluster] < head_blocks(d))
        in_cluster--;
    if (rows <= in_cluster * 608)
        return std::min(in_cluster, (rows + 63) / 64);
    return std::min(std::max(std::min(wave, (rows + 255) / 256), in_cluster), kMaxSplits);
}

// Whether the device holds a launch's clusters (one per head block, of `splits` CTAs) all at once, asked once per number
// of ranges and device.
bool clusters_fit(int dev, int splits, int blocks)
{
    if (splits < 2 || splits > kMaxCluster || dev < 0 || dev >= nnf::kMaxDevices)
        return false;
    static std::mutex mu;
    static int held[nnf::kMaxDevices][kMaxCluster + 1] = {}; // clusters + 1; 0: not asked yet
    std::lock_guard<std::mutex> lock(mu);
    int& h = held[dev][splits];
    if (h == 0)
    {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(splits, 1);
        c.blockDim = dim3(kWarps * 32);
        c.dynamicSmemBytes = kSmemBytes;
        cudaLaunchAttribute a[1];
        a[0].id = cudaLaunchAttributeClusterDimension;
        a[0].val.clusterDim.x = (unsigned)splits, a[0].val.clusterDim.y = 1, a[0].val.clusterDim.z = 1;
        c.attrs = a, c.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, decode_attention_kernel<kWarps>, &c) != cudaSuccess)
            n = 0;
        (void)cudaGetLastError();
        h = n + 1;
    }
    return h - 1 >= blocks;
}
} // namespace

namespace nnf
{
int attn_check(const nnf_b200_attn_desc& d, std::string* why)
{
    if (d.heads < 1 || d.kv_heads < 1 || d.heads % d.kv_heads != 0 || d.position < 0 || d.capacity <= d.position ||
        d.splits < 0 || d.reserved[0] || d.reserved[1] || d.reserved[2] || d.reserved[3])
    {
        *why = "heads must be a positive multiple of kv_heads, 0 <= position < capacity, splits >= 0, reserved zero";
        return NNF_B200_EINVAL;
    }
    if (d.head_dim != kD || d.dtype != NNF_B200_F16)
    {
        *why = "decode attention is built for head_dim 128 and fp16 tensors";
        return NNF_B200_ENOTSUP;
    }
    return NNF_B200_OK;
}

size_t attn_workspace_bytes(const nnf_b200_ctx* ctx, const nnf_b200_attn_desc& d)
{
    const int splits = pick_splits(ctx, d);
    if (splits == 1)
        return 0;
    const size_t cnt = ((size_t)head_blocks(d) * sizeof(unsigned) + 255) / 256 * 256;
    return cnt + (size_t)head_blocks(d) * splits * kSlot * sizeof(float);
}

int attn_launch(nnf_b200_ctx* ctx, cudaStream_t stream, const nnf_b200_attn_desc& d, const void* q, const void* k_new,
                const void* v_new, void* k_cache, void* v_cache, void* out, void* workspace)
{
    AttnParams p{};
    p.q = static_cast<const __half*>(q);
    p.k_new = static_cast<const __half*>(k_new);
    p.v_new = static_cast<const __half*>(v_new);
    p.k_cache = static_cast<__half*>(k_cache);
    p.v_cache = static_cast<__half*>(v_cache);
    p.out = static_cast<__half*>(out);
    p.heads = d.heads, p.kv_heads = d.kv_heads, p.capacity = d.capacity, p.position = d.position;
    p.rotary = d.rotary != 0;
    p.group = d.heads / d.kv_heads;
    p.qblocks = (p.group + kQ - 1) / kQ;
    p.scale = (d.softmax_scale > 0.f ? d.softmax_scale : 1.0f / sqrtf((float)kD)) * 1.44269504f; // exponents base 2
    p.log2_base = log2f(d.rotary_base > 0.f ? d.rotary_base : 10000.f);
    p.splits = pick_splits(ctx, d);
    const int rows = d.position + 1;
    // whole blocks of rows per range; ranges left without rows store an empty partial result
    p.chunk = ((rows + p.splits - 1) / p.splits + kRows - 1) / kRows * kRows;
    if (p.splits > 1)
    {
        const size_t cnt = ((size_t)head_blocks(d) * sizeof(unsigned) + 255) / 256 * 256;
        p.ws_count = static_cast<unsigned*>(workspace);
        p.ws_part = reinterpret_cast<float*>(static_cast<char*>(workspace) + cnt);
    }
    static bool configured[kMaxDevices] = {}; // the shared-memory limit belongs to the device that is current
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev < 0 || dev >= kMaxDevices))
        e = cudaErrorInvalidDevice;
    if (e == cudaSuccess && !configured[dev])
    {
        e = cudaFuncSetAttribute(decode_attention_kernel<kWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        configured[dev] = e == cudaSuccess;
    }
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("decode_attention set-up: ") + cudaGetErrorString(e));
    (void)cudaGetLastError();
    cudaLaunchConfig_t cfg = {};
    const bool short_one = p.splits == 1 && rows <= kShortRows;
    cfg.gridDim = short_one ? dim3(d.heads) : dim3(p.splits, head_blocks(d));
    // an uncut sequence of up to two passes of four warps: 61 rows 4.1 -> 3.5 us
    const bool few = p.splits == 1 && rows <= 2 * kFewWarps * kRows;
    cfg.blockDim = dim3(short_one ? kShortThreads : (few ? kFewWarps : kWarps) * 32);
    cfg.dynamicSmemBytes = short_one ? 0 : few ? kFewWarps * kQ * kD * sizeof(float) : kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    overlap_attribute(attr, &cfg.numAttrs);
    p.cluster = clusters_fit(dev, p.splits, head_blocks(d));
    if (p.cluster)
    {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = (unsigned)p.splits;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    cfg.attrs = attr;
    e = short_one ? cudaLaunchKernelEx(&cfg, short_attention_kernel, p)
        : few     ? cudaLaunchKernelEx(&cfg, decode_attention_kernel<kFewWarps>, p)
                  : cudaLaunchKernelEx(&cfg, decode_attention_kernel<kWarps>, p);
    if (e != cudaSuccess)
        return set_error(ctx, NNF_B200_ECUDA, std::string("decode_attention launch: ") + cudaGetErrorString(e));
    ctx->launches++;
    return NNF_B200_OK;
}
} // namespace nnf
