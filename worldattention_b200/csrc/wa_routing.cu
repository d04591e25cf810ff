// HSA block routing on the GPU: block-mean pooling, block attention map, Gini-adaptive selection.
//
// Stands in for wan/modules/hsa/routing.py.  The work is bandwidth- and latency-bound (one read
// of Q and K, then a few hundred short rows), so the kernels are plain coalesced / warp-shuffle
// code; every reduction that feeds the discrete selection accumulates in float64 and rounds once,
// which makes the chosen block ids independent of the summation order.
#include <cooperative_groups.h>

#include <type_traits>

#include "wa_internal.cuh"

namespace wa {

// ------------------------------------------------------------------------------------------------
// Pooling.  One CTA per (batch, block, head): block_size token rows of D contiguous elements.
// ------------------------------------------------------------------------------------------------
constexpr int POOL_THREADS = 256;

template <bool VEC_BF16>
__global__ void __launch_bounds__(POOL_THREADS)
pool_blocks_kernel(View4 x, int L, int H, int D, int block_size, int num_blocks, int aligned,
                   float *__restrict__ pooled, View4 x2, int L2, int num_blocks2, int aligned2,
                   float *__restrict__ pooled2, int out_blocks2, int *__restrict__ zero, int n_zero) {
    int nb = blockIdx.x;
    const int h = blockIdx.y, b = blockIdx.z;
    if (n_zero && nb == 0 && h == 0 && b == 0)   // counters of the kernel that follows on the stream
        for (int i = threadIdx.x; i < n_zero; i += POOL_THREADS) zero[i] = 0;
    int out_blocks = num_blocks;   // rows per (batch, head) of the output buffer
    if (nb >= num_blocks) {   // second tensor (keys) pooled by the same launch
        nb -= num_blocks;
        x = x2; L = L2; num_blocks = num_blocks2; aligned = aligned2; pooled = pooled2; out_blocks = out_blocks2;
    }
    const int t0 = nb * block_size;
    const int n_real = min(block_size, L - t0);
    extern __shared__ double pool_smem[];  // [rows_in_flight][D]

    const long long base = (long long)b * x.sb + (long long)h * x.sh;
    float *dst = pooled + (((long long)b * H + h) * out_blocks + nb) * (long long)D;

    if (VEC_BF16) {
        // 8 bf16 per thread per token; lanes_per_row threads cover one token row.
        const int lanes_per_row = D >> 3;
        const int rows = POOL_THREADS / lanes_per_row;
        const int lane = threadIdx.x % lanes_per_row, row = threadIdx.x / lanes_per_row;
        double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // float64: exact for a block of bf16 values, so order-free
        if (row < rows) {
            const __nv_bfloat16 *p = (const __nv_bfloat16 *)x.ptr + base + lane * 8;
            // eight row loads in flight per thread; rows past the end contribute zeros
            for (int t = row; t < n_real; t += 8 * rows) {
                uint4 raw[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int tt = t + u * rows;
                    raw[u] = tt < n_real ? *reinterpret_cast<const uint4 *>(p + (long long)(t0 + tt) * x.sl)
                                         : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&raw[u]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float2 f = __bfloat1622float2(h2[i]);
                        acc[2 * i] += (double)f.x;
                        acc[2 * i + 1] += (double)f.y;
                    }
                }
            }
        }
        double *sm = pool_smem;  // [rows][D]
        if (row < rows) {
#pragma unroll
            for (int i = 0; i < 8; ++i) sm[row * D + lane * 8 + i] = acc[i];
        }
        __syncthreads();
        for (int d = threadIdx.x; d < D; d += POOL_THREADS) {
            double s = 0.0;
            for (int r = 0; r < rows; ++r) s += sm[r * D + d];
            float out;
            if (aligned) out = bf16_round_f((float)(s / (double)block_size));
            else out = __fdiv_rn(bf16_round_f((float)s), (float)n_real);
            dst[d] = out;
        }
    } else {
        // generic: thread per channel (strided), float64 accumulation.
        const int rows = max(1, POOL_THREADS / D);
        const int per_row = min(D, POOL_THREADS);
        const int row = threadIdx.x / per_row, lane = threadIdx.x % per_row;
        for (int d0 = 0; d0 < D; d0 += per_row) {
            const int d = d0 + lane;
            double acc = 0.0;
            if (row < rows && d < D) {
                // sixteen loads in flight per thread (25 + 74 blocks of 64 float32 rows, 12 heads: 20.5 -> 13.3 us)
                for (int t = row; t < n_real; t += 16 * rows) {
                    float v[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u)
                        v[u] = t + u * rows < n_real ? load_elem(x.ptr, x.dtype, base + (long long)(t0 + t + u * rows) * x.sl + d) : 0.f;
#pragma unroll
                    for (int u = 0; u < 16; ++u) acc += (double)v[u];
                }
                pool_smem[row * per_row + lane] = acc;
            }
            __syncthreads();
            if (row == 0 && d < D) {
                double s = 0.0;
                for (int r = 0; r < rows; ++r) s += pool_smem[r * per_row + lane];
                float out;
                if (aligned) {
                    out = (float)(s / (double)block_size);
                    if (x.dtype == WA_BF16) out = bf16_round_f(out);
                } else {
                    float sum32 = (float)s;
                    if (x.dtype == WA_BF16) sum32 = bf16_round_f(sum32);
                    out = __fdiv_rn(sum32, (float)n_real);
                }
                dst[d] = out;
            }
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Pooling, streaming form for bf16 rows of 8..256 channels (a power of two): SPLIT warps per (batch,
// block, head), no block-level synchronisation on the load path.  The D/8 lanes that cover one token
// row form a group; the groups of the item's warps take token rows round-robin.  Every lane keeps
// UNROLL 16-byte row loads in flight and issues the next batch before it consumes the current one.
// Sums are float64: a sum of a few hundred bf16 values is exact there, so the result does not depend
// on the order of the additions (the routing decision downstream is discrete).
// ------------------------------------------------------------------------------------------------
#ifndef WA_POOL_SPLIT
#define WA_POOL_SPLIT 2
#endif
#ifndef WA_POOL_UNROLL
#define WA_POOL_UNROLL 4
#endif

#ifndef WA_POOL_MIN_CTAS
#define WA_POOL_MIN_CTAS 3
#endif

template <int UNROLL, int SPLIT>
__global__ void __launch_bounds__(POOL_THREADS, WA_POOL_MIN_CTAS)
pool_warp_kernel(View4 x, int L, int H, int D, int block_size, int num_blocks, int aligned, float *__restrict__ pooled,
                 View4 x2, int L2, int num_blocks2, int aligned2, float *__restrict__ pooled2, int out_blocks2, int B,
                 int *__restrict__ zero, int n_zero) {
    constexpr int ITEMS_PER_CTA = POOL_THREADS / 32 / SPLIT;
    __shared__ double partial[ITEMS_PER_CTA][SPLIT > 1 ? SPLIT - 1 : 1][256];   // [item][warp - 1][channel]
    if (n_zero && blockIdx.x == 0)   // counters of the kernel that follows on the stream
        for (int i = threadIdx.x; i < n_zero; i += POOL_THREADS) zero[i] = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = warp / SPLIT, part = warp % SPLIT;   // item of this CTA, this warp's share of its rows
    long long item = (long long)blockIdx.x * ITEMS_PER_CTA + slot;   // ((b, block), head), head fastest
    const long long items1 = (long long)B * num_blocks * H;
    int out_blocks = num_blocks;   // rows per (batch, head) of the output buffer
    bool live = true;
    if (item >= items1) {   // second tensor (keys) pooled by the same launch
        item -= items1;
        live = item < (long long)B * num_blocks2 * H;
        x = x2; L = L2; num_blocks = num_blocks2; aligned = aligned2; pooled = pooled2; out_blocks = out_blocks2;
    }
    if (!live) item = 0;   // keeps the CTA's barrier below unconditional; nothing is stored
    const int h = (int)(item % H);
    const int nb = (int)((item / H) % num_blocks);
    const int b = (int)(item / ((long long)H * num_blocks));
    const int t0 = nb * block_size;
    const int n_real = live ? min(block_size, L - t0) : 0;
    const int lanes_per_row = D >> 3, groups = 32 / lanes_per_row;
    const int col = (lane % lanes_per_row) * 8, group = lane / lanes_per_row;
    const int stride = groups * SPLIT;               // token rows between two loads of one lane
    const __nv_bfloat16 *p = (const __nv_bfloat16 *)x.ptr + (long long)b * x.sb + (long long)h * x.sh +
                             (long long)t0 * x.sl + col;
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint4 cur[UNROLL], nxt[UNROLL];
    auto fetch = [&](uint4 (&dst)[UNROLL], int t) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int tt = t + u * stride;
            dst[u] = tt < n_real ? __ldg(reinterpret_cast<const uint4 *>(p + (long long)tt * x.sl)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    const int first = part * groups + group;
    fetch(cur, first);
    for (int t = first; t < n_real; t += UNROLL * stride) {
        fetch(nxt, t + UNROLL * stride);   // rows past the end load nothing
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const __nv_bfloat162 *h2 = reinterpret_cast<const __nv_bfloat162 *>(&cur[u]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __bfloat1622float2(h2[i]);
                acc[2 * i] += (double)f.x;
                acc[2 * i + 1] += (double)f.y;
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) cur[u] = nxt[u];
    }
    // the groups of a warp, then the warps of the item
    for (int step = lanes_per_row; step < 32; step <<= 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], step);
    }
    if (SPLIT > 1) {
        if (part > 0 && group == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) partial[slot][part - 1][col + i] = acc[i];
        }
        __syncthreads();
        if (part == 0 && group == 0) {
#pragma unroll
            for (int w = 0; w < SPLIT - 1; ++w)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i] += partial[slot][w][col + i];
        }
    }
    if (live && part == 0 && group == 0) {
        float out[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            out[i] = aligned ? bf16_round_f((float)(acc[i] / (double)block_size))
                             : __fdiv_rn(bf16_round_f((float)acc[i]), (float)n_real);
        float4 *dst = reinterpret_cast<float4 *>(pooled + (((long long)b * H + h) * out_blocks + nb) * (long long)D + col);
        dst[0] = make_float4(out[0], out[1], out[2], out[3]);
        dst[1] = make_float4(out[4], out[5], out[6], out[7]);
    }
}

// ------------------------------------------------------------------------------------------------
// Block attention map.  One CTA per (b, h, query block) row; a warp per key block for the dot.
// ------------------------------------------------------------------------------------------------
constexpr int SCORE_THREADS = 256;

#ifdef WA_ROUTE_TRACE   // tuning aid: per-CTA phase timestamps (ns) of the fused routing kernel
__device__ long long g_route_trace[4096 * 12];
#define ROUTE_STAMP(i)                                                                         \
    do {                                                                                       \
        if (threadIdx.x == 0 && blockIdx.x < 4096) {                                           \
            long long t_;                                                                      \
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                            \
            g_route_trace[blockIdx.x * 12 + (i)] = t_;                                          \
        }                                                                                      \
    } while (0)
#else
#define ROUTE_STAMP(i)
#endif

// One row of logits: out[j] = fl32(q . k_j) * scale, the dot accumulated in float64 and rounded once.  `out` may be
// shared or global memory.  Called by every thread of the CTA; no barrier at the end.
__device__ __forceinline__ void row_logits(const float *__restrict__ q, const float *__restrict__ k, int Nkv, int D, float scale,
                                           float *out) {
    const int T = blockDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = T >> 5;
    const bool vec = (D & 3) == 0;
    for (int j0 = warp * 8; j0 < Nkv; j0 += nwarps * 8) {   // eight independent dot products in flight
        double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (vec) {
            for (int d = lane * 4; d < D; d += 128) {
                const float4 qv = *reinterpret_cast<const float4 *>(q + d);
                float4 kv[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    kv[u] = j0 + u < Nkv ? *reinterpret_cast<const float4 *>(k + (long long)(j0 + u) * D + d)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    acc[u] = fma((double)qv.x, (double)kv[u].x, acc[u]);
                    acc[u] = fma((double)qv.y, (double)kv[u].y, acc[u]);
                    acc[u] = fma((double)qv.z, (double)kv[u].z, acc[u]);
                    acc[u] = fma((double)qv.w, (double)kv[u].w, acc[u]);
                }
            }
        } else {
            for (int d = lane; d < D; d += 32) {
                const double qd = (double)q[d];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (j0 + u < Nkv) acc[u] = fma(qd, (double)k[(long long)(j0 + u) * D + d], acc[u]);
            }
        }
        // transposed reduction: halve the number of live sums at each of the first three exchange steps,
        // so the eight 32-lane sums cost 9 exchanges instead of 40; lane l ends with dot (l >> 2) & 7
        const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4;
        double r4[4], r2[2];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double keep = b16 ? acc[u + 4] : acc[u], give = b16 ? acc[u] : acc[u + 4];
            r4[u] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const double keep = b8 ? r4[u + 2] : r4[u], give = b8 ? r4[u] : r4[u + 2];
            r2[u] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
        }
        double t = (b4 ? r2[1] : r2[0]) + __shfl_xor_sync(0xffffffffu, b4 ? r2[0] : r2[1], 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        const int u = (lane >> 2) & 7;
        if ((lane & 3) == 0 && j0 + u < Nkv) out[j0 + u] = __fmul_rn((float)t, scale);
    }
}

// Softmax of one row of logits in place: float64 sum, each value rounded once to float32.  `out` may be shared or global
// memory; `red` holds >= 32 doubles.  Called by every thread of the CTA after the logits are complete (and a barrier).
__device__ __forceinline__ void row_softmax(int Nkv, float *out, double *red, float *bcast) {
    const int T = blockDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = T >> 5;
    float m = -INFINITY;
    for (int j = threadIdx.x; j < Nkv; j += T) m = fmaxf(m, out[j]);
    m = warp_max(m);
    if (lane == 0) red[warp] = (double)m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float mm = -INFINITY;
        for (int w = 0; w < nwarps; ++w) mm = fmaxf(mm, (float)red[w]);
        *bcast = mm;
    }
    __syncthreads();
    m = *bcast;
    __syncthreads();

    double s = 0.0;
    for (int j = threadIdx.x; j < Nkv; j += T) {
        float e = (float)exp((double)__fsub_rn(out[j], m));
        out[j] = e;
        s += (double)e;
    }
    s = warp_sum_d(s);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < nwarps; ++w) t += red[w];
        *bcast = (float)t;
    }
    __syncthreads();
    const float denom = *bcast;
    for (int j = threadIdx.x; j < Nkv; j += T) out[j] = __fdiv_rn(out[j], denom);
    __syncthreads();
}

// One row: out[j] = softmax_j(q . k_j * scale) with float64 dots and sums, each rounded once to float32.
__device__ __forceinline__ void row_block_attention(const float *__restrict__ q, const float *__restrict__ k, int Nkv, int D,
                                                    float scale, float *out, double *red, float *bcast) {
    row_logits(q, k, Nkv, D, scale, out);
    __syncthreads();
    ROUTE_STAMP(1);
    row_softmax(Nkv, out, red, bcast);
}

// ------------------------------------------------------------------------------------------------
// Logits of all rows on the float64 matrix instruction (head_dim 128): out[row][key] = fl32(q . k) * scale, float64 products
// and sums, rounded once, like row_logits.  With a row per CTA every row streams its head's pooled keys from L2 and converts
// them to float64 for itself (a quarter of a product's rate); here a CTA holds up to 80 query rows of a head as float64
// operands in shared memory, in the instruction's own order (16-byte loads without conflicts), and a warp reads 16 keys from
// L2 once for all of them.  A lane's four dimensions of a step of 16 are neighbours in memory (its k indices of both operands
// are permuted alike).  Bound by the float64 pipe: 65 multiply-adds per clock and SM measured for this instruction, 55 for scalar
// ones.  One CTA of eight warps per SM: two warps per scheduler keep the pipe busy.
// 12 heads, 74 rows, 11 700 keys: 103 us (12.9 T multiply-adds/s of the 18.4 measured); with eight rows per CTA on scalar float64 and
// the row steps in the same kernel the routing took 655 us, now 103 + 119.
// ------------------------------------------------------------------------------------------------
constexpr int RL_WARPS = 8, RL_KEYS = 16, RL_TILE = RL_WARPS * RL_KEYS, RL_MAX_MT = 5;   // keys per warp and per tile; 16-row tiles per CTA

__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

template <int MT>
__global__ void __launch_bounds__(RL_WARPS * 32, 1)
route_logits_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int Nq, int Nkv, float scale, float *__restrict__ out,
                    int groups, int tiles, long long units) {
    extern __shared__ __align__(16) unsigned char logits_smem[];
    double2 *qfrag = reinterpret_cast<double2 *>(logits_smem);        // [MT][8 steps][4 dimensions][32 lanes] of (row g, row g + 8)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    pdl_wait();
    // unit = (batch and head, group of MT * 16 rows, tile of keys), tile fastest; a CTA takes a run of them
    const long long first = units * blockIdx.x / gridDim.x, last = units * (blockIdx.x + 1) / gridDim.x;
    long long staged = -1;
    for (long long u = first; u < last; ++u) {
        const long long rows = u / tiles, bh = rows / groups;
        const int key0 = (int)(u - rows * tiles) * RL_TILE + warp * RL_KEYS, i0 = (int)(rows - bh * groups) * MT * 16;
        if (rows != staged) {
            __syncthreads();
            for (int i = threadIdx.x; i < MT * 8 * 32; i += RL_WARPS * 32) {
                const int l = i & 31, row = i0 + (i >> 8) * 16 + (l >> 2), dim = ((i >> 5) & 7) * 16 + (l & 3) * 4;
                const float *q = qp + (bh * Nq + row) * 128 + dim;
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 lo = row < Nq ? *reinterpret_cast<const float4 *>(q) : zero;
                const float4 hi = row + 8 < Nq ? *reinterpret_cast<const float4 *>(q + 8 * 128) : zero;
                double2 *dst = qfrag + (i >> 5) * 128 + l;
                dst[0] = make_double2(lo.x, hi.x);
                dst[32] = make_double2(lo.y, hi.y);
                dst[64] = make_double2(lo.z, hi.z);
                dst[96] = make_double2(lo.w, hi.w);
            }
            __syncthreads();
            staged = rows;
        }
        if (key0 >= Nkv) continue;
        const float4 *ka = reinterpret_cast<const float4 *>(kp + (bh * Nkv + min(key0 + g, Nkv - 1)) * 128) + t;
        const float4 *kb = reinterpret_cast<const float4 *>(kp + (bh * Nkv + min(key0 + 8 + g, Nkv - 1)) * 128) + t;
        float4 na = __ldg(ka), nb = __ldg(kb);
        double acc[MT][2][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][0][i] = acc[m][1][i] = 0.0;
#pragma unroll 2
        for (int step = 0; step < 8; ++step) {
            const double ba[4] = {na.x, na.y, na.z, na.w}, bb[4] = {nb.x, nb.y, nb.z, nb.w};
            const int next = min(step + 1, 7) * 4;
            na = __ldg(ka + next);
            nb = __ldg(kb + next);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                double a[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const double2 q2 = qfrag[((m * 8 + step) * 4 + e) * 32 + lane];
                    a[2 * e] = q2.x;
                    a[2 * e + 1] = q2.y;
                }
                mma_f64(acc[m][0], a, ba);
                mma_f64(acc[m][1], a, bb);
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int half = 0; half < 2; ++half)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = i0 + m * 16 + g + 8 * (i >> 1), key = key0 + half * 8 + 2 * t + (i & 1);
                    if (row < Nq && key < Nkv) out[(bh * Nq + row) * Nkv + key] = __fmul_rn((float)acc[m][half][i], scale);
                }
    }
}

__global__ void __launch_bounds__(SCORE_THREADS)
route_scores_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int Nq, int Nkv,
                    int D, float scale, float *__restrict__ attn) {
    const long long row = blockIdx.x;  // (b*H + h)*Nq + i
    const long long bh = row / Nq;
    __shared__ double red[32];
    __shared__ float bcast;
    row_block_attention(qp + row * D, kp + bh * (long long)Nkv * D, Nkv, D, scale, attn + row * Nkv, red, &bcast);
}

// ------------------------------------------------------------------------------------------------
// Selection, pass A: per row, sort (probability descending, id ascending) and the row's Gini term.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t descending_key(float p) {
    if (p == 0.0f) p = 0.0f;  // -0 -> +0
    uint32_t u = __float_as_uint(p);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // ascending-orderable
    return ~u;                                        // descending
}

__global__ void route_sort_kernel(const float *__restrict__ attn, int Nkv, int n_pow2,
                                  int32_t *__restrict__ index, float *__restrict__ gini_rows) {
    extern __shared__ unsigned long long keys[];  // n_pow2
    __shared__ double red[32];
    const long long row = blockIdx.x;
    const float *p = attn + row * Nkv;
    const int T = blockDim.x;

    for (int j = threadIdx.x; j < n_pow2; j += T)
        keys[j] = j < Nkv ? (((unsigned long long)descending_key(p[j]) << 32) | (unsigned)j)
                          : 0xFFFFFFFFFFFFFFFFull;
    __syncthreads();
    for (int k = 2; k <= n_pow2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n_pow2; i += T) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long a = keys[i], b = keys[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) {
                        keys[i] = b;
                        keys[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    // index + Gini: sum_m fp32((N + 1 - 2m) * p_(m)), m 1-based, accumulated in float64.
    int32_t *idx = index + row * Nkv;
    double acc = 0.0;
    for (int m = threadIdx.x; m < Nkv; m += T) {
        const int id = (int)(keys[m] & 0xFFFFFFFFull);
        idx[m] = id;
        const float w = __fsub_rn((float)(Nkv + 1), __fmul_rn(2.0f, (float)(m + 1)));
        acc += (double)__fmul_rn(w, p[id]);
    }
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (T + 31) / 32; ++w) t += red[w];
        gini_rows[row] = __fdiv_rn((float)t, (float)Nkv);
    }
}

// Mean of a head's Gini rows over (batch, query block) -> the head's cumulative-mass threshold.  256 strided
// float64 partials, a shuffle tree inside each warp, the eight warp totals added in order.  Called by every
// thread of a CTA of >= 256 threads; `red` holds >= 8 doubles; the result is valid in every thread.
__device__ __forceinline__ float head_threshold(const float *gini_rows, int B, int H, int Nq, int h, float tau_min,
                                                float tau_span, double *red, float *bcast) {
    const int count = B * Nq, tid = threadIdx.x;
    if (tid < 256) {
        double g = 0.0;
        for (int r = tid; r < count; r += 256) {
            const int bb = r / Nq, ii = r % Nq;
            g += (double)__ldcg(&gini_rows[((long long)bb * H + h) * Nq + ii]);
        }
        g = warp_sum_d(g);
        if ((tid & 31) == 0) red[tid >> 5] = g;
    }
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        const float head_gini = (float)(t / (double)count);
        *bcast = __fadd_rn(tau_min, __fmul_rn(head_gini, tau_span));
    }
    __syncthreads();
    return *bcast;
}

// ------------------------------------------------------------------------------------------------
// Selection, pass B: per-head threshold, float64 cumulative mass, count (and optional mask).
// ------------------------------------------------------------------------------------------------
constexpr int SELECT_THREADS = 256;

__global__ void __launch_bounds__(SELECT_THREADS)
route_count_kernel(const float *__restrict__ attn, const int32_t *__restrict__ index,
                   const float *__restrict__ gini_rows, int B, int H, int Nq, int Nkv,
                   float tau_min, float tau_span, const int32_t *__restrict__ fixed_num,
                   int32_t *__restrict__ num, uint8_t *__restrict__ mask,
                   float *__restrict__ thresholds) {
    const long long row = blockIdx.x;
    const int i = (int)(row % Nq);
    const int h = (int)((row / Nq) % H);
    const int b = (int)(row / ((long long)Nq * H));
    __shared__ double part[SELECT_THREADS];
    __shared__ float thr_s;
    __shared__ int cnt_s;

    if (threadIdx.x == 0) cnt_s = 0;
    const float thr = head_threshold(gini_rows, B, H, Nq, h, tau_min, tau_span, part, &thr_s);
    if (threadIdx.x == 0 && b == 0 && i == 0) thresholds[h] = thr;
    const float *p = attn + row * Nkv;
    const int32_t *idx = index + row * Nkv;
    uint8_t *mrow = mask ? mask + row * Nkv : nullptr;

    if (fixed_num) {
        const int n = max(0, min(fixed_num[h], Nkv));
        if (threadIdx.x == 0) num[row] = n;
        if (mrow)
            for (int m = threadIdx.x; m < Nkv; m += SELECT_THREADS) mrow[idx[m]] = m < n;
        return;
    }

    // contiguous chunk per thread, float64 running sums, exclusive scan of the chunk totals
    const int chunk = (Nkv + SELECT_THREADS - 1) / SELECT_THREADS;
    const int m0 = threadIdx.x * chunk, m1 = min(Nkv, m0 + chunk);
    double local = 0.0;
    for (int m = m0; m < m1; ++m) local += (double)p[idx[m]];
    __syncthreads();
    part[threadIdx.x] = local;
    __syncthreads();
    double offset = 0.0;
    for (int w = 0; w < threadIdx.x; ++w) offset += part[w];  // fixed order prefix
    int kept = 0;
    double run = offset;
    for (int m = m0; m < m1; ++m) {
        const float pm = p[idx[m]];
        run += (double)pm;
        const bool keep = __fsub_rn((float)run, pm) < thr;
        kept += keep;
        if (mrow) mrow[idx[m]] = keep;
    }
    if (kept) atomicAdd(&cnt_s, kept);
    __syncthreads();
    if (threadIdx.x == 0) num[row] = cnt_s;
}

// ------------------------------------------------------------------------------------------------
// The forward's routing, a CTA per (batch, head, query block) row (route_row, route_fused_kernel): scores where
// route_logits_kernel has not left them, softmax, sort and the row's Gini term, with the probabilities kept in shared memory.  The CTA that
// finishes a head last (a counter per head) turns the head's Gini rows into its threshold and counts
// every row of that head, a warp per row over the sorted probabilities; the CTA that finishes the
// last head prepares the attention kernel's launch (work order, counters).  Same arithmetic as the
// three separate kernels above; no CTA ever waits for another.
// ------------------------------------------------------------------------------------------------
// one key per thread, bitonic: exchange distances below 32 go through shuffles, the rest through `keys` (one entry per thread)
__device__ __forceinline__ unsigned long long sort_key_per_thread(unsigned long long key, unsigned long long *keys, int n_pow2) {
    const int tid = threadIdx.x;
    for (int k = 2; k <= n_pow2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            unsigned long long other;
            if (j >= 32) {
                keys[tid] = key;
                __syncthreads();
                other = keys[tid ^ j];
                __syncthreads();
            } else {
                other = __shfl_xor_sync(0xffffffffu, key, j);
            }
            const bool keep_min = ((tid & j) == 0) == ((tid & k) == 0);
            key = (other < key) == keep_min ? other : key;
        }
    }
    return key;
}

__device__ __forceinline__ void sort_keys_smem(unsigned long long *keys, int n_pow2) {   // ascending bitonic sort, whole CTA
    const int T = blockDim.x;
    for (int k = 2; k <= n_pow2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n_pow2; i += T) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long a = keys[i], b = keys[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) {
                        keys[i] = b;
                        keys[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// The k best blocks of a row, in order, WITHOUT sorting the row: for a fixed per-head count over thousands of key blocks
// the full bitonic sort (105 passes over 16384 keys) was two thirds of the routing kernel.  Keys are the sort's own
// 64-bit keys (descending probability, then ascending id; all distinct).  A most-significant-byte-first radix select
// narrows down the k-th smallest key (histogram passes over the row: it stops as soon as one histogram bin holds exactly the
// keys still needed, or the keys at or below the bin are no more than the CTA's threads), the keys at or below it are collected
// and only they are sorted.  `idx[0..k)` receive the same ids in the same order as the full sort; slots past k are not written.
// `keys` is shared memory for `key_slots` >= max(threads, pow2(k)) entries.  Called by every thread of the CTA (256 to 1024 of them).
// A larger k is selected in pieces: `from` is the smallest key still to be had and `n_left` how many there are of those; returns
// the largest key taken.
__device__ __forceinline__ unsigned long long select_top_blocks(const float *probs, int Nkv, int k, unsigned long long *keys, int key_slots,
                                                                int32_t *idx, int id_offset, unsigned long long *keys_out,
                                                                unsigned long long from, int n_left) {
    __shared__ unsigned int hist[256];
    __shared__ unsigned long long prefix_s, mask_s;
    __shared__ int need_s, done_s;
    __shared__ unsigned int taken_s;
    const int T = blockDim.x, tid = threadIdx.x;
    if (k <= 0) return 0ull;
    auto key_of = [&](int j) { return ((unsigned long long)descending_key(probs[j]) << 32) | (unsigned)(id_offset + j); };
    // the keys of a row usually agree in their leading bytes (probabilities of one softmax share sign and most of the
    // exponent; near-uniform attention agrees much further): find the common prefix with one min/max pass and start the
    // digit passes below it
    __shared__ unsigned long long lo_s[32], hi_s[32];
    unsigned long long lo = 0xFFFFFFFFFFFFFFFFull, hi = 0ull;
    for (int j = tid; j < Nkv; j += T) {
        const unsigned long long key = key_of(j);
        if (key < from) continue;
        lo = key < lo ? key : lo;
        hi = key > hi ? key : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if ((tid & 31) == 0) {
        lo_s[tid >> 5] = lo;
        hi_s[tid >> 5] = hi;
    }
    __syncthreads();
    int first_byte = 7;
    if (tid == 0) {
        for (int w = 1; w < (T >> 5); ++w) {
            lo = lo_s[w] < lo ? lo_s[w] : lo;
            hi = hi_s[w] > hi ? hi_s[w] : hi;
        }
        const unsigned long long diff = lo ^ hi;
        const int top = diff ? (63 - __clzll((long long)diff)) >> 3 : 0;      // highest byte in which two keys differ
        const unsigned long long mask = top >= 7 ? 0ull : (0xFFFFFFFFFFFFFFFFull << (8 * (top + 1)));
        prefix_s = lo & mask;
        mask_s = mask;
        need_s = k;
        done_s = k >= n_left;     // every block is kept: nothing to select
        taken_s = 0u;
        lo_s[0] = (unsigned long long)top;
    }
    __syncthreads();
    first_byte = (int)lo_s[0];
    // a histogram per warp (in the keys' memory, idle until the collection below): the probabilities of a row share their
    // leading bits, so in the first passes every warp adds to the same bin, and one shared bin serialised them
    unsigned int *warp_hist = reinterpret_cast<unsigned int *>(keys);
    const int copies = min(T >> 5, key_slots / 128), wid = (tid >> 5) % copies;      // 256 counters of 4 bytes per copy
    for (int byte = first_byte; byte >= 0 && !done_s; --byte) {
        for (int i = tid; i < copies * 256; i += T) warp_hist[i] = 0u;
        __syncthreads();
        const unsigned long long prefix = prefix_s, mask = mask_s;
        for (int j0 = 0; j0 < Nkv; j0 += T) {      // whole warps iterate together: the votes below need every lane
            const int j = j0 + tid;
            const unsigned long long key = j < Nkv ? key_of(j) : 0ull;
            const bool cand = j < Nkv && key >= from && (key & mask) == prefix;
            const unsigned int voters = __ballot_sync(0xffffffffu, cand);
            if (voters) {
                // the probabilities of a row share their leading bits: the digit of the warp's first candidate is usually
                // the digit of most of them; those are counted with one addition, the others add for themselves
                const unsigned int digit = (unsigned)(key >> (8 * byte)) & 255u;
                const int leader = __ffs(voters) - 1;
                const unsigned int common = __shfl_sync(0xffffffffu, digit, leader);
                const unsigned int same = __ballot_sync(0xffffffffu, cand && digit == common);
                if ((tid & 31) == leader) atomicAdd(&warp_hist[wid * 256 + common], (unsigned)__popc(same));
                else if (cand && digit != common) atomicAdd(&warp_hist[wid * 256 + digit], 1u);
            }
        }
        __syncthreads();
        if (tid < 256) {
            unsigned int total = 0;
            for (int w = 0; w < copies; ++w) total += warp_hist[w * 256 + tid];
            hist[tid] = total;
        }
        __syncthreads();
        if (tid < 32) {      // first digit at which the running count reaches what is still needed
            unsigned int mine[8], sum = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                mine[i] = hist[tid * 8 + i];
                sum += mine[i];
            }
            unsigned int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += v;
            }
            const unsigned int need = (unsigned)need_s, before = incl - sum;
            if (before < need && need <= incl) {      // exactly one lane
                unsigned int run = before, in_bin = 0;
                int d = -1;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (d < 0) {
                        if (need <= run + mine[i]) {
                            d = i;
                            in_bin = mine[i];
                        } else {
                            run += mine[i];
                        }
                    }
                }
                prefix_s = prefix | ((unsigned long long)(tid * 8 + d) << (8 * byte));
                mask_s = mask | (0xFFull << (8 * byte));
                need_s = (int)(need - run);
                // stop refining when the whole bin is wanted, or when the keys at or below this bin are few enough to sort
                // with a key per thread (every further digit would cost another pass over the whole row)
                if (in_bin == need - run || (unsigned)k - (need - run) + in_bin <= (unsigned)min(T, 1024)) done_s = 1;
            }
        }
        __syncthreads();
    }
    ROUTE_STAMP(11);
    // collect the keys at or below the k-th (with all keys kept when k >= Nkv: mask 0, prefix 0), then sort just those
    const unsigned long long prefix = prefix_s, mask = mask_s;
    for (int j = tid; j < Nkv; j += T) {
        const unsigned long long key = key_of(j);
        if (key >= from && (key & mask) <= prefix) keys[atomicAdd(&taken_s, 1u)] = key;
    }
    __syncthreads();
    const int kept = (int)taken_s;      // >= min(k, Nkv): the k best and, when the selection stopped early, the rest of the last bin
    int k_pow2 = 1;
    while (k_pow2 < kept) k_pow2 <<= 1;
    for (int j = kept + tid; j < k_pow2; j += T) keys[j] = 0xFFFFFFFFFFFFFFFFull;
    __syncthreads();
    if (k_pow2 <= T && T <= key_slots) {
        const unsigned long long key = sort_key_per_thread(tid < k_pow2 ? keys[tid] : 0xFFFFFFFFFFFFFFFFull, keys, k_pow2);
        __syncthreads();
        keys[tid] = key;
        __syncthreads();
    } else {
        sort_keys_smem(keys, k_pow2);
    }
    for (int m = tid; m < min(k, kept); m += T) {
        if (idx) idx[m] = (int32_t)(keys[m] & 0xFFFFFFFFull);
        if (keys_out) keys_out[m] = keys[m];      // the sortable keys themselves (ids offset by `id_offset`)
    }
    const unsigned long long taken = keys[max(0, min(k, kept) - 1)];
    __syncthreads();
    return taken;
}

// One (batch, head, query block) row of the fused routing; called by every thread of the CTA.  With `logits_ready`
// the row's scaled logits already lie in `sorted + row * Nkv`.
template <bool READY>
__device__ __forceinline__ void route_row(const long long row, const float *__restrict__ qp,
                                          const float *__restrict__ kp, int B, int H, int Nq, int Nkv, int n_pow2, int D, float scale,
                                          float tau_min, float tau_span, const int32_t *__restrict__ fixed_num, float *sorted,
                                          int32_t *__restrict__ index, int32_t *num, float *__restrict__ thresholds, float *gini_rows,
                                          int *counters, const SchedJob &job, unsigned long long *keys, float *probs, double *red,
                                          float &bcast, int &last_flag) {
    const int T = blockDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = T >> 5;
    const long long bh = row / Nq;
    const int h = (int)(bh % H);

    if constexpr (READY) {
        const float *lrow = sorted + row * Nkv;
        for (int j = tid; j < Nkv; j += T) probs[j] = lrow[j];
    } else {
        row_logits(qp + row * D, kp + bh * (long long)Nkv * D, Nkv, D, scale, probs);
    }
    __syncthreads();
    ROUTE_STAMP(1);
    row_softmax(Nkv, probs, red, &bcast);
    ROUTE_STAMP(2);

    if (n_pow2 <= T) {
        unsigned long long key = sort_key_per_thread(
            tid < Nkv ? (((unsigned long long)descending_key(probs[tid]) << 32) | (unsigned)tid) : 0xFFFFFFFFFFFFFFFFull, keys, n_pow2);
        keys[tid] = key;
        __syncthreads();
    } else {
        for (int j = tid; j < n_pow2; j += T)
            keys[j] = j < Nkv ? (((unsigned long long)descending_key(probs[j]) << 32) | (unsigned)j)
                              : 0xFFFFFFFFFFFFFFFFull;
        __syncthreads();
        sort_keys_smem(keys, n_pow2);
    }
    ROUTE_STAMP(3);
    int32_t *idx = index + row * Nkv;
    double acc = 0.0;
    for (int m = tid; m < Nkv; m += T) {
        const int id = (int)(keys[m] & 0xFFFFFFFFull);
        idx[m] = id;
        const float w = __fsub_rn((float)(Nkv + 1), __fmul_rn(2.0f, (float)(m + 1)));
        acc += (double)__fmul_rn(w, probs[id]);
    }
    acc = warp_sum_d(acc);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < nwarps; ++w) t += red[w];
        gini_rows[row] = __fdiv_rn((float)t, (float)Nkv);
    }
    __syncthreads();
    if (!fixed_num) {
        // What the count needs of this row once the head's threshold is known: for every sorted position the
        // cumulative mass before it, fl32(fl64 prefix including m) - p_m.  A contiguous run of positions per thread,
        // float64 run totals scanned over the CTA (lane order inside a warp, warp order across warps).
        float *crow = sorted + row * Nkv;
        const int chunk = (Nkv + T - 1) / T;
        const int m0 = min(Nkv, tid * chunk), m1 = min(Nkv, m0 + chunk);
        double local = 0.0;
        for (int m = m0; m < m1; ++m) local += (double)probs[(int)(keys[m] & 0xFFFFFFFFull)];
        double incl = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) red[warp] = incl;
        __syncthreads();
        double run = incl - local;
        for (int w = 0; w < warp; ++w) run += red[w];
        for (int m = m0; m < m1; ++m) {
            const float pm = probs[(int)(keys[m] & 0xFFFFFFFFull)];
            run += (double)pm;
            crow[m] = __fsub_rn((float)run, pm);
        }
    }

    // ---- last CTA of this head? ------------------------------------------------------------------
    const int rows_per_head = B * Nq;
    ROUTE_STAMP(4);
    __threadfence();
    __syncthreads();
    if (tid == 0) last_flag = atomicAdd(&counters[1 + h], 1) == rows_per_head - 1;
    __syncthreads();
    ROUTE_STAMP(5);
    // experiment: let the attention kernel's CTAs become resident while only the heads' last CTAs are still at work
    if (job.release_dependents_after_rows) pdl_release_dependents();
    if (!last_flag) return;
    __threadfence();

    const float thr = head_threshold(gini_rows, B, H, Nq, h, tau_min, tau_span, red, &bcast);
    if (tid == 0) thresholds[h] = thr;
    ROUTE_STAMP(8);
    if (fixed_num) {
        const int n = max(0, min(fixed_num[h], Nkv));
        for (int r = tid; r < rows_per_head; r += T) num[((long long)(r / Nq) * H + h) * Nq + r % Nq] = n;
    } else {
        // kept blocks of a row = positions whose mass-before is under the threshold.  All rows of the head are
        // counted together, a batch of independent loads per thread at a time: the loop is one CTA's, so it is the
        // memory round trips, not the arithmetic, that it has to keep few.
        constexpr int ROWS_AT_ONCE = 128, LOADS = 8;
        __shared__ int row_count[ROWS_AT_ONCE];
        __shared__ long long row_base[ROWS_AT_ONCE];
        const int step_r = T / Nkv, step_m = T % Nkv;   // element e -> (row e / Nkv, position e % Nkv), advanced without dividing
        for (int r0 = 0; r0 < rows_per_head; r0 += ROWS_AT_ONCE) {
            const int nr = min(ROWS_AT_ONCE, rows_per_head - r0);
            for (int r = tid; r < nr; r += T) {
                const int rg = r0 + r;
                row_count[r] = 0;
                row_base[r] = (((long long)(rg / Nq) * H + h) * Nq + rg % Nq) * Nkv;
            }
            __syncthreads();
            if ((Nkv & 3) == 0) {
                // four positions per load; a thread's loads are all issued before the first is used
                const int quads_per_row = Nkv >> 2, total = nr * quads_per_row;
                constexpr int QLOADS = 8;
                for (int e0 = 0; e0 < total; e0 += QLOADS * T) {
                    float4 c[QLOADS];
                    int rr[QLOADS];
#pragma unroll
                    for (int u = 0; u < QLOADS; ++u) {
                        const int e = e0 + u * T + tid;
                        rr[u] = -1;
                        if (e < total) {
                            const int r = e / quads_per_row;
                            rr[u] = r;
                            c[u] = __ldcg(reinterpret_cast<const float4 *>(sorted + row_base[r]) + (e - r * quads_per_row));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < QLOADS; ++u) {
                        const int n = rr[u] >= 0 ? (c[u].x < thr) + (c[u].y < thr) + (c[u].z < thr) + (c[u].w < thr) : 0;
                        const int first = __shfl_sync(0xffffffffu, rr[u], 0);
                        if (__all_sync(0xffffffffu, rr[u] == first)) {   // the warp is inside one row: one addition for all lanes
                            const int all = __reduce_add_sync(0xffffffffu, n);
                            if (lane == 0 && all) atomicAdd(&row_count[first], all);
                        } else if (n) {
                            atomicAdd(&row_count[rr[u]], n);
                        }
                    }
                }
            } else {
            const int total = nr * Nkv;   // <= 128 * 16384
            int r = tid / Nkv, m = tid % Nkv;
            for (int e0 = 0; e0 < total; e0 += LOADS * T) {
                float c[LOADS];
                int rr[LOADS];
#pragma unroll
                for (int u = 0; u < LOADS; ++u) {
                    const bool in = e0 + u * T + tid < total;
                    rr[u] = in ? r : -1;
                    c[u] = in ? __ldcg(sorted + row_base[r] + m) : 0.f;
                    r += step_r;
                    m += step_m;
                    if (m >= Nkv) {
                        m -= Nkv;
                        ++r;
                    }
                }
#pragma unroll
                for (int u = 0; u < LOADS; ++u) {
                    const bool keep = rr[u] >= 0 && c[u] < thr;
                    const int first = __shfl_sync(0xffffffffu, rr[u], 0);
                    if (__all_sync(0xffffffffu, rr[u] == first)) {   // the warp is inside one row: one atomic for all lanes
                        const int n = __popc(__ballot_sync(0xffffffffu, keep));
                        if (lane == 0 && first >= 0 && n) atomicAdd(&row_count[first], n);
                    } else if (keep) {
                        atomicAdd(&row_count[rr[u]], 1);
                    }
                }
            }
            }
            __syncthreads();
            ROUTE_STAMP(9);
            for (int r2 = tid; r2 < nr; r2 += T) num[row_base[r2] / Nkv] = row_count[r2];
            __syncthreads();
        }
    }

    // ---- last head? ------------------------------------------------------------------------------
    ROUTE_STAMP(6);
    __threadfence();
    __syncthreads();
    if (tid == 0) last_flag = atomicAdd(&counters[0], 1) == H - 1;
    __syncthreads();
    if (!last_flag || !job.order) return;
    __threadfence();
    schedule_items(num, B * H * Nq, Nq, Nkv, job);
    ROUTE_STAMP(7);
}

// ------------------------------------------------------------------------------------------------
// The forward's routing: a row per CTA, from its logits on where route_logits_kernel has left them in `sorted` (READY).  Then up to 512
// threads a row run with 32 registers, four CTAs to an SM instead of two: the kernel is a chain of barriers, and several rows cover each
// other (74 rows of 12 heads, the whole call: over 147 blocks 194.1 -> 191.6 us, over 293 346 -> 337, over 585 696 -> 688).
// ------------------------------------------------------------------------------------------------
template <bool READY, int THREADS>
__global__ void __launch_bounds__(THREADS, READY && THREADS <= 512 ? 4 : 1)
route_fused_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int B, int H, int Nq, int Nkv, int n_pow2,
                   int D, float scale, float tau_min, float tau_span, const int32_t *__restrict__ fixed_num,
                   float *sorted, int32_t *__restrict__ index, int32_t *num, float *__restrict__ thresholds,
                   float *gini_rows, int *counters, SchedJob job, int gate_per_cta, int sm_count, int slots, int key_slots) {
    extern __shared__ __align__(16) unsigned char fused_smem[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(fused_smem);   // key_slots
    float *probs = reinterpret_cast<float *>(keys + key_slots);                      // Nkv
    __shared__ double red[256];
    __shared__ float bcast;
    __shared__ int last_flag;

    // CTAs are dealt to the SMs round-robin, so CTAs b, b + sm_count, ... tend to share an SM: give them
    // neighbouring rows (same head, same pooled keys) so that their key reads can meet in L1
    const long long row = (long long)(blockIdx.x % sm_count) * slots + blockIdx.x / sm_count;
    // No early release of the attention kernel here: its CTAs, once resident and waiting, slowed the tail of this
    // kernel (the per-head count and the work order are a few CTAs' work) by about 5 us.
    pdl_wait();                 // pooled means and zeroed counters come from the launch before
    if (job.release_at_start) pdl_release_dependents();
    if (row >= (long long)B * H * Nq) return;

    ROUTE_STAMP(0);
    if (job.order) convert_gate_slice(job, (int)row * gate_per_cta, gate_per_cta);
    route_row<READY>(row, qp, kp, B, H, Nq, Nkv, n_pow2, D, scale, tau_min, tau_span, fixed_num, sorted, index, num, thresholds,
              gini_rows, counters, job, keys, probs, red, bcast, last_flag);
}

// ------------------------------------------------------------------------------------------------
// The whole routing of short rows (head_dim 128, up to 64 query blocks of a head over the batch and 128 key blocks; with a batch 64, or
// 128 where one round of the CTA's warps does): a cluster, or a CTA, per head.  There the kernel above is a chain of waits: some twenty
// barriers of a row, a counter per head, the last CTA's walk over all rows of the head, a second counter.  Here the logits come from the float64 matrix instruction, a 16 x 8 tile per
// warp, a row's softmax, sort and sums stay inside a warp (K keys per lane, exchanges by shuffles), and the head's threshold
// and counts need two barriers.  Same sums (float64, rounded where the reference rounds) and the same order.
// 12 heads, the whole call: 7 query blocks over 19 key blocks 40.5 -> 37.0 us, 37 over 37 100.1 -> 96.2 (the routing itself 20.6 -> 11.5 and
// 22.6 -> 15.9).
// ------------------------------------------------------------------------------------------------
// Without a batch the rows of a head are spread over a cluster of up to eight CTAs, so that every row has a warp of its own and the whole
// chip fetches its instructions at once; the Gini terms go to all of them through distributed shared memory (37 query blocks over 37:
// 17.8 -> 11.1 us, the call 87.5 -> 81.5; 63 over 125, which the row kernel took before, 166 -> 149 us a call).
constexpr int RH_WARPS = 32, RH_MAX_KEYS = 128, RH_MAX_ROWS = 64;

__device__ __forceinline__ float value_of_key(unsigned long long key) {      // the probability that descending_key was given
    const uint32_t u = ~(uint32_t)(key >> 32);
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

template <int K, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
route_head_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int B, int H, int Nq, int Nkv, float scale, float tau_min,
                  float tau_span, const int32_t *__restrict__ fixed_num, int32_t *__restrict__ index, int32_t *num,
                  float *__restrict__ thresholds, int *counters, SchedJob job, int gate_per_cta) {
    constexpr int W = K * 32;
    extern __shared__ __align__(16) float row_values[];      // [rows of the head][W]: logits, then the mass before each sorted position
    __shared__ float gini[RH_MAX_ROWS], threshold;
    __shared__ int last_flag;
    const auto cluster = cooperative_groups::this_cluster();
    const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank(), h = blockIdx.x / parts;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, rows = B * Nq;
    // this CTA's rows of the head (a batch has one CTA per head)
    const int per = (rows + parts - 1) / parts, first = part * per, mine_n = max(0, min(per, rows - first));
    if (parts > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // everybody is there before anything is left with others
    pdl_wait();                 // pooled means and zeroed counters come from the launch before
    if (job.release_at_start) pdl_release_dependents();
    if (job.order) convert_gate_slice(job, (int)blockIdx.x * gate_per_cta, gate_per_cta);

    const int in_item = B == 1 ? mine_n : Nq, row_tiles = (in_item + 15) / 16, key_tiles = (Nkv + 7) / 8;      // in_item: rows of a batch item here
    for (int u = warp; u < B * row_tiles * key_tiles; u += WARPS) {
        const int b = u / (row_tiles * key_tiles), rest = u - b * row_tiles * key_tiles, i0 = first + rest / key_tiles * 16, j0 = rest % key_tiles * 8;
        const float *qb = qp + (long long)(b * H + h) * Nq * 128;
        const float4 *qa = reinterpret_cast<const float4 *>(qb + min(i0 + g, Nq - 1) * 128) + t;
        const float4 *qc = reinterpret_cast<const float4 *>(qb + min(i0 + g + 8, Nq - 1) * 128) + t;
        const float4 *kv = reinterpret_cast<const float4 *>(kp + ((long long)(b * H + h) * Nkv + min(j0 + g, Nkv - 1)) * 128) + t;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll(WARPS < 32 ? 8 : 2)
        for (int step = 0; step < 8; ++step) {
            const float4 x = __ldg(qa + 4 * step), y = __ldg(qc + 4 * step), z = __ldg(kv + 4 * step);
            const double a[8] = {x.x, y.x, x.y, y.y, x.z, y.z, x.w, y.w}, k[4] = {z.x, z.y, z.z, z.w};
            mma_f64(acc, a, k);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = i0 + g + 8 * (i >> 1), key = j0 + 2 * t + (i & 1);
            if (row < first + in_item && key < Nkv) row_values[(b * Nq + row - first) * W + key] = __fmul_rn((float)acc[i], scale);
        }
    }
    __syncthreads();

    if (parts > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int i = warp; i < mine_n; i += WARPS) {
        const int r = first + i;
        float *mine = row_values + i * W + lane;
        const long long row = (long long)(r / Nq * H + h) * Nq + r % Nq;
        float e[K], m = -INFINITY;
#pragma unroll
        for (int u = 0; u < K; ++u) {
            e[u] = u * 32 + lane < Nkv ? mine[u * 32] : -INFINITY;
            m = fmaxf(m, e[u]);
        }
        m = warp_max(m);
        double sum = 0.0;
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (u * 32 + lane < Nkv) {
                e[u] = (float)exp((double)__fsub_rn(e[u], m));
                sum += (double)e[u];
            }
        const float denom = (float)warp_sum_d(sum);
        unsigned long long key[K];      // position u * 32 + lane
#pragma unroll
        for (int u = 0; u < K; ++u)
            key[u] = u * 32 + lane < Nkv ? ((unsigned long long)descending_key(__fdiv_rn(e[u], denom)) << 32) | (unsigned)(u * 32 + lane)
                                         : 0xFFFFFFFFFFFFFFFFull;
#pragma unroll
        for (int k = 2; k <= W; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
                for (int u = 0; u < K; ++u) {
                    if (j >= 32) {
                        const int v = u ^ (j >> 5);
                        if (v > u) {
                            const bool up = ((u * 32) & k) == 0;
                            const unsigned long long a = key[u], c = key[v];
                            key[u] = (a < c) == up ? a : c;
                            key[v] = (a < c) == up ? c : a;
                        }
                    } else {
                        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key[u], j);
                        const bool keep_min = ((lane & j) == 0) == (((u * 32 + lane) & k) == 0);
                        key[u] = (other < key[u]) == keep_min ? other : key[u];
                    }
                }
            }
        double spread = 0.0, before = 0.0;
#pragma unroll
        for (int u = 0; u < K; ++u) {
            const int at = u * 32 + lane;
            const bool real = at < Nkv;
            const float p = real ? value_of_key(key[u]) : 0.f;
            if (real) {
                index[row * Nkv + at] = (int32_t)(key[u] & 0xFFFFFFFFull);
                spread += (double)__fmul_rn(__fsub_rn((float)(Nkv + 1), __fmul_rn(2.0f, (float)(at + 1))), p);
            }
            double mass = (double)p;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double v = __shfl_up_sync(0xffffffffu, mass, o);
                if (lane >= o) mass += v;
            }
            mass += before;
            before = __shfl_sync(0xffffffffu, mass, 31);
            mine[u * 32] = real ? __fsub_rn((float)mass, p) : INFINITY;
        }
        spread = warp_sum_d(spread);
        if (lane < parts) *cluster.map_shared_rank(&gini[r], lane) = __fdiv_rn((float)spread, (float)Nkv);
    }
    if (parts > 1) cluster.sync(); else __syncthreads();
    if (warp == 0) {
        double total = 0.0;
        for (int r = lane; r < rows; r += 32) total += (double)gini[r];
        total = warp_sum_d(total);
        if (lane == 0) threshold = __fadd_rn(tau_min, __fmul_rn((float)(total / (double)rows), tau_span));
        if (lane == 0 && part == 0) thresholds[h] = threshold;
    }
    __syncthreads();
    for (int i = warp; i < mine_n; i += WARPS) {
        const int r = first + i;
        int n = 0;
        if (fixed_num) {
            n = max(0, min(fixed_num[h], Nkv));
        } else {
#pragma unroll
            for (int u = 0; u < K; ++u) n += __popc(__ballot_sync(0xffffffffu, row_values[i * W + u * 32 + lane] < threshold));
        }
        if (lane == 0) num[(long long)(r / Nq * H + h) * Nq + r % Nq] = n;
    }
    // the CTA that finishes the last head prepares the attention kernel's launch
    __threadfence();
    __syncthreads();
    if (tid == 0) last_flag = atomicAdd(&counters[0], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last_flag || !job.order) return;
    __threadfence();
    schedule_items(num, B * H * Nq, Nq, Nkv, job);
}

// ------------------------------------------------------------------------------------------------
// Routing with a fixed count per head where nobody reads the whole order or the thresholds: a row per CTA, up to 2048 blocks in
// registers (V per thread) from the logit to the key, more in shared memory, and only the best blocks are ordered.  Every warp sorts its lanes' best keys; with
// W warps and c = ceil(count / W), at least W * c >= count blocks lie at or below the worst of the warps' c-th keys, so what lies
// above it cannot be among the best.  The few blocks at or below it (26 of 256 for a count of 16, about 90 of 11 700 for 32) are
// collected and each counts how many of them come before it, which is its place.  Same probabilities and keys as route_row,
// hence the same ids in the same order.  The counts are known without the routing, so the attention kernel's work order is
// made by a CTA of its own (the first) beside the rows instead of by the last one after them.
// Bound by latency (a row is a chain of four block-wide exchanges) and, over thousands of blocks, by the float64 exponentials.
// 128 threads a row up to 512 blocks; 256 where the row makes its own logits (a warp per eight dot products) or has up to
// 2048; beyond, 512 threads with three CTAs per SM (two from some 12 500 blocks on, by their shared memory).
// Before, a row was sorted (or, beyond 1024 blocks, selected by radix passes) with its Gini term, and two counters led to the last CTA.
// 12 heads, 37 rows over 256 blocks: 16.7 -> 7.8 us, the call 134.0 -> 128.6; 74 rows over 11 700: 117 -> 78 with the values in registers (two
// CTAs per SM and spills), 56 in shared memory.
// Rows of few blocks, which were route_head_kernel's, the whole call: 4 over 4 26.5 -> 21.0, 7 over 19 34.1 -> 29.8, 37 over 37 78.6 -> 68.7,
// 37 over 74 88.3 -> 75.3, 25 over 49 of a batch of two 102.1 -> 94.7.
// ------------------------------------------------------------------------------------------------
template <int T, int V>      // V = 0: the row's values in shared memory, any number of them
__global__ void __launch_bounds__(T, V ? 1024 / T : 3)
route_topk_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int H, int Nq, int Nkv, int D, float scale,
                  const int32_t *__restrict__ fixed_num, float *logits, int32_t *__restrict__ index, int32_t *__restrict__ num, SchedJob job,
                  int rows, int gate_per_cta, int sm_count, int per_sm, int logits_ready) {
    constexpr int W = T / 32, SLOTS = V == 0 ? 1024 : V * T < 2048 ? V * T : 2048, N = V ? V : 1;
    extern __shared__ float own_logits[];                // Nkv, where the row makes them or keeps its values
    __shared__ __align__(16) unsigned long long keys[SLOTS];
    __shared__ float top[W];
    __shared__ double sums[W];
    __shared__ uint32_t bounds[W];
    __shared__ int n_near;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();                 // pooled means, or logits, come from the launch before
    if (job.release_at_start) pdl_release_dependents();
    if (blockIdx.x == 0) {
        const int each = job.paired ? (Nq + 1) >> 1 : Nq;      // items of a head
        if (job.order && (!job.paired || job.by_counts))
            schedule_rows([&](int item) { return __ldg(fixed_num + (item / each) % H); }, rows / Nq * each, Nkv, job);
        return;
    }
    // neighbouring rows (same head, same pooled keys) on one SM, as in route_fused_kernel
    const int at = blockIdx.x - 1, row = (at % sm_count) * per_sm + at / sm_count;
    if (row >= rows) return;
    if (job.order) convert_gate_slice(job, row * gate_per_cta, gate_per_cta);

    const int want = max(0, min(fixed_num[(row / Nq) % H], Nkv));
    if (tid == 0) {
        num[row] = want;
        n_near = 0;
    }
    if (want == 0) return;
    float *lrow = logits + (long long)row * Nkv;
    if (!logits_ready) {
        row_logits(qp + (long long)row * D, kp + (long long)(row / Nq) * Nkv * D, Nkv, D, scale, own_logits);
        __syncthreads();
    }
    float e[N], m = -INFINITY;
    uint32_t key[N], best = 0xFFFFFFFFu;                 // upper half of the sort's key; the id is the lower one
    double sum = 0.0;
    auto total_of = [&]() -> float {                     // the row's sum, rounded once
        sum = warp_sum_d(sum);
        if (lane == 0) sums[warp] = sum;
        __syncthreads();
        sum = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) sum += sums[w];
        return (float)sum;
    };
    auto largest_of = [&]() {
        m = warp_max(m);
        if (lane == 0) top[warp] = m;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) m = fmaxf(m, top[w]);
    };
    auto exponential = [&](float x) { return (float)exp((double)__fsub_rn(x, m)); };
    if constexpr (V > 0) {
#pragma unroll
        for (int u = 0; u < V; ++u) {
            const int j = u * T + tid;
            e[u] = j < Nkv ? (logits_ready ? __ldcg(lrow + j) : own_logits[j]) : -INFINITY;
        }
#pragma unroll
        for (int u = 0; u < V; ++u) m = fmaxf(m, e[u]);
        largest_of();
#pragma unroll
        for (int u = 0; u < V; ++u)
            if (u * T + tid < Nkv) {
                e[u] = exponential(e[u]);
                sum += (double)e[u];
            }
        const float denom = total_of();
#pragma unroll
        for (int u = 0; u < V; ++u) {
            key[u] = u * T + tid < Nkv ? descending_key(__fdiv_rn(e[u], denom)) : 0xFFFFFFFFu;
            best = min(best, key[u]);
        }
    } else {
        // a thread only touches its own places
        if (logits_ready) {
#pragma unroll 8
            for (int j = tid; j < Nkv; j += T) own_logits[j] = __ldcg(lrow + j);
        }
#pragma unroll 8
        for (int j = tid; j < Nkv; j += T) m = fmaxf(m, own_logits[j]);
        largest_of();
#pragma unroll 2
        for (int j = tid; j < Nkv; j += T) {
            const float x = exponential(own_logits[j]);
            own_logits[j] = x;
            sum += (double)x;
        }
        const float denom = total_of();
#pragma unroll 2
        for (int j = tid; j < Nkv; j += T) {
            const uint32_t x = descending_key(__fdiv_rn(own_logits[j], denom));
            own_logits[j] = __uint_as_float(x);
            best = min(best, x);
        }
    }
    const int nth = (want + W - 1) / W;
    uint32_t bound = 0xFFFFFFFFu;
    if (nth <= 32) {
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const uint32_t other = __shfl_xor_sync(0xffffffffu, best, j);
                const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
                best = keep_min ? min(best, other) : max(best, other);
            }
        bound = __shfl_sync(0xffffffffu, best, nth - 1);
    }
    if (lane == 0) bounds[warp] = bound;
    __syncthreads();
    bound = 0u;
#pragma unroll
    for (int w = 0; w < W; ++w) bound = max(bound, bounds[w]);
    auto collect = [&](int j, uint32_t x) {
        const bool near = j < Nkv && x <= bound;
        const unsigned voters = __ballot_sync(0xffffffffu, near);
        if (voters) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&n_near, __popc(voters));
            const int pos = __shfl_sync(0xffffffffu, base, 0) + __popc(voters & ((1u << lane) - 1u));
            if (near && pos < SLOTS) keys[pos] = ((unsigned long long)x << 32) | (unsigned)j;
        }
    };
    if constexpr (V > 0) {
#pragma unroll
        for (int u = 0; u < V; ++u) collect(u * T + tid, key[u]);
    } else {
#pragma unroll 4
        for (int j0 = 0; j0 < Nkv; j0 += T) collect(j0 + tid, j0 + tid < Nkv ? __float_as_uint(own_logits[j0 + tid]) : 0xFFFFFFFFu);
    }
    __syncthreads();
    const int n = n_near;        // >= want
    int32_t *idx = index + (long long)row * Nkv;
    if (n <= T) {
        if (tid < n) {
            const unsigned long long mine = keys[tid];
            int place = 0;
            for (int j = 0; j < n; ++j) place += keys[j] < mine;
            if (place < want) idx[place] = (int32_t)(mine & 0xFFFFFFFFull);
        }
    } else if ((V > 0 && V * T <= SLOTS) || n <= SLOTS) {        // a large count, or many equal probabilities
        int n_pow2 = 1;
        while (n_pow2 < n) n_pow2 <<= 1;                 // <= SLOTS, a power of two
        for (int j = n + tid; j < n_pow2; j += T) keys[j] = 0xFFFFFFFFFFFFFFFFull;
        __syncthreads();
        sort_keys_smem(keys, n_pow2);
        for (int j = tid; j < want; j += T) idx[j] = (int32_t)(keys[j] & 0xFFFFFFFFull);
    } else if constexpr (V == 0) {
        for (int j = tid; j < Nkv; j += T) lrow[j] = value_of_key((unsigned long long)__float_as_uint(own_logits[j]) << 32);
        __syncthreads();
        unsigned long long from = 0ull;
        for (int first = 0; first < want; first += SLOTS)
            from = select_top_blocks(lrow, Nkv, min(want - first, SLOTS), keys, SLOTS, idx + first, 0, nullptr, from, Nkv - first) + 1ull;
    }
}

#ifdef WA_ROUTE_TRACE
}  // namespace wa
extern "C" int wa_route_trace_read(long long *dst, int n_ctas) {
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(dst, wa::g_route_trace, (size_t)n_ctas * 12 * sizeof(long long));
    return 0;
}
namespace wa {
#endif

// ------------------------------------------------------------------------------------------------
// Fixed top-k routing over a SHARDED key cache (no reference counterpart: the reference is single-device).
// Every rank scores only the key blocks it owns and keeps its best `kcap` per row as sortable 64-bit keys
// (descending logit, then ascending global block id); the ranks exchange those keys; each rank then merges
// the W * kcap candidates of a row, takes the head's k best and keeps the ones it owns.  Work and traffic per
// rank fall with the number of ranks, where gathering every pooled key and repeating the whole routing on
// every rank does not.  Selection is by LOGIT: softmax is monotone, so this is the single-device choice
// except where distinct logits round to one probability at the k-th place (there the single-device rule
// orders by block id, this one by logit).
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
route_local_candidates_kernel(const float *__restrict__ qp, const float *__restrict__ kp, int Nq, int Nloc, int n_pow2, int D,
                              float scale, int block_lo, int kcap, unsigned long long *__restrict__ cand) {
    extern __shared__ __align__(16) unsigned char cand_smem[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(cand_smem);   // n_pow2
    float *logits = reinterpret_cast<float *>(keys + n_pow2);                       // Nloc
    const long long row = blockIdx.x;   // (b * H + h) * Nq + i
    const long long bh = row / Nq;
    row_logits(qp + row * D, kp + bh * (long long)Nloc * D, Nloc, D, scale, logits);
    __syncthreads();
    if (n_pow2 > (int)blockDim.x && kcap <= 1024) {
        // a long row: pick the kcap best instead of sorting all of them (same keys, same order)
        const int k = min(kcap, Nloc);
        select_top_blocks(logits, Nloc, k, keys, n_pow2, nullptr, block_lo, cand + row * kcap, 0ull, Nloc);
        for (int j = k + threadIdx.x; j < kcap; j += blockDim.x) cand[row * kcap + j] = 0xFFFFFFFFFFFFFFFFull;
        return;
    }
    for (int j = threadIdx.x; j < n_pow2; j += blockDim.x)
        keys[j] = j < Nloc ? (((unsigned long long)descending_key(logits[j]) << 32) | (unsigned)(block_lo + j))
                           : 0xFFFFFFFFFFFFFFFFull;
    __syncthreads();
    sort_keys_smem(keys, n_pow2);
    for (int j = threadIdx.x; j < kcap; j += blockDim.x) cand[row * kcap + j] = j < n_pow2 ? keys[j] : 0xFFFFFFFFFFFFFFFFull;
}

__global__ void __launch_bounds__(256)
route_merge_candidates_kernel(const unsigned long long *__restrict__ cand, int W, long long rows, int Nq, int H, int kcap,
                              int n_pow2, const int32_t *__restrict__ topk, int Nkv_total, int block_lo, int block_hi,
                              int index_stride, int32_t *__restrict__ local_index, int32_t *__restrict__ local_num) {
    extern __shared__ __align__(16) unsigned char merge_smem[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(merge_smem);   // n_pow2 >= W * kcap
    __shared__ int count;
    const long long row = blockIdx.x;
    const int h = (int)((row / Nq) % H);
    const int n = W * kcap;
    for (int j = threadIdx.x; j < n_pow2; j += blockDim.x)
        keys[j] = j < n ? cand[((long long)(j / kcap) * rows + row) * kcap + (j % kcap)] : 0xFFFFFFFFFFFFFFFFull;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    sort_keys_smem(keys, n_pow2);
    const int k = max(0, min(min(topk[h], Nkv_total), n));
    // the head's k best; the ones this rank owns, in ascending block order (candidates of one rank arrive id-distinct,
    // so an id appears once)
    int32_t *out = local_index + row * index_stride;
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
        const unsigned id = (unsigned)(keys[j] & 0xFFFFFFFFull);
        if (keys[j] != 0xFFFFFFFFFFFFFFFFull && (int)id >= block_lo && (int)id < block_hi) {
            // rank among the owned ones = number of owned selected ids below this one
            int below = 0;
            for (int t = 0; t < k; ++t) {
                const unsigned other = (unsigned)(keys[t] & 0xFFFFFFFFull);
                below += keys[t] != 0xFFFFFFFFFFFFFFFFull && (int)other >= block_lo && (int)other < block_hi && other < id;
            }
            out[below] = (int)id - block_lo;
            atomicAdd(&count, 1);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) local_num[row] = count;
}

// ------------------------------------------------------------------------------------------------
// Mask -> ascending index list.  One warp per row, ballot-ordered compaction.
// ------------------------------------------------------------------------------------------------
__global__ void map_to_index_kernel(const uint8_t *__restrict__ mask, long long rows, int Nkv,
                                    int32_t *__restrict__ index, int32_t *__restrict__ num) {
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const uint8_t *m = mask + row * Nkv;
    int32_t *idx = index + row * Nkv;
    int n = 0;
    for (int j0 = 0; j0 < Nkv; j0 += 32) {
        const int j = j0 + lane;
        const bool on = j < Nkv && m[j] != 0;
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        if (on) idx[n + __popc(bal & ((1u << lane) - 1u))] = j;
        n += __popc(bal);
    }
    for (int j = n + lane; j < Nkv; j += 32) idx[j] = -1;
    if (lane == 0) num[row] = n;
}

// ------------------------------------------------------------------------------------------------
// Selection of one KV shard.  One warp per row: a bitmap of the shard's blocks in shared memory,
// then two ballot-ordered compactions (selected blocks, then the rest).
// ------------------------------------------------------------------------------------------------
constexpr int LOCAL_SEL_WARPS = 8;

__global__ void __launch_bounds__(LOCAL_SEL_WARPS * 32)
local_selection_kernel(const int32_t *__restrict__ index, const int32_t *__restrict__ num, long long rows, int Nkv,
                       int block_lo, int width, int words, int32_t *__restrict__ local_index,
                       int32_t *__restrict__ local_num) {
    extern __shared__ unsigned int sel_bitmap[];   // [warps][words]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * LOCAL_SEL_WARPS + warp;
    if (row >= rows) return;
    unsigned int *bm = sel_bitmap + warp * words;
    for (int w = lane; w < words; w += 32) bm[w] = 0u;
    __syncwarp();
    const int32_t *idx = index + row * Nkv;
    const int n = max(0, min(num[row], Nkv));
    for (int j = lane; j < n; j += 32) {
        const int id = max(0, min(idx[j], Nkv - 1)) - block_lo;
        if (id >= 0 && id < width) atomicOr(&bm[id >> 5], 1u << (id & 31));
    }
    __syncwarp();
    int32_t *out = local_index + row * width;
    int at = 0;
    for (int pass = 0; pass < 2; ++pass) {   // members first, then the rest
        for (int base = 0; base < width; base += 32) {
            const int c = base + lane;
            const bool member = c < width && ((bm[base >> 5] >> lane) & 1u);
            const bool take = c < width && (pass == 0 ? member : !member);
            const unsigned bal = __ballot_sync(0xffffffffu, take);
            if (take) out[at + __popc(bal & ((1u << lane) - 1u))] = c;
            at += __popc(bal);
        }
        if (pass == 0 && lane == 0) local_num[row] = at;
    }
}

}  // namespace wa

using namespace wa;

extern "C" int wa_route_local_selection(const int32_t *index, const int32_t *num, long long rows, int Nkv, int block_lo,
                                        int block_hi, int32_t *local_index, int32_t *local_num, void *stream) {
    WA_REQUIRE(index && num && local_index && local_num, WA_ERR_ARG, "wa_route_local_selection: null pointer");
    WA_REQUIRE(rows > 0 && Nkv > 0 && block_lo >= 0 && block_hi > block_lo, WA_ERR_ARG,
               "wa_route_local_selection: need rows > 0, Nkv > 0 and a non-empty block range");
    const int width = block_hi - block_lo;
    WA_REQUIRE(width <= 16384, WA_ERR_UNSUPPORTED, "wa_route_local_selection: at most 16384 blocks per shard, got %d", width);
    const int words = (width + 31) / 32;
    const long long ctas = (rows + LOCAL_SEL_WARPS - 1) / LOCAL_SEL_WARPS;
    WA_REQUIRE(ctas < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_route_local_selection: too many rows");
    local_selection_kernel<<<(unsigned)ctas, LOCAL_SEL_WARPS * 32, (size_t)LOCAL_SEL_WARPS * words * sizeof(unsigned int),
                             (cudaStream_t)stream>>>(index, num, rows, Nkv, block_lo, width, words, local_index, local_num);
    return check_launch("wa_route_local_selection");
}

namespace wa {
static bool pool_vec_ok(const wa_tensor4 *x, int D) {
    return x->dtype == WA_BF16 && D % 8 == 0 && D / 8 <= POOL_THREADS && ((uintptr_t)x->ptr % 16 == 0) &&
           x->stride_b % 8 == 0 && x->stride_l % 8 == 0 && x->stride_h % 8 == 0;
}

// Pools `x` (and, when given, `y`, e.g. queries and keys of one forward) in a single launch.
int pool_launch(const wa_tensor4 *x, int Lx, float *px, const wa_tensor4 *y, int Ly, float *py, int B, int H, int D,
                int block_size, cudaStream_t stream, int *zero, int n_zero, int y_first_block, int *status_mirror) {
    const int nbx = ceil_div(Lx, block_size);
    const int nby_all = y ? ceil_div(Ly, block_size) : 0;   // rows per (batch, head) of py
    const int y_aligned = y ? Ly % block_size == 0 : 0;
    wa_tensor4 y_tail;
    if (y && y_first_block >= nby_all) y = nullptr;   // every key block is pooled already
    if (y && y_first_block > 0) {   // the first blocks of y are pooled already: start at token y_first_block * block_size
        y_tail = *y;
        y_tail.ptr = (char *)y->ptr + (size_t)y_first_block * block_size * y->stride_l * dtype_size(y->dtype);
        y = &y_tail;
        Ly -= y_first_block * block_size;
        py += (size_t)y_first_block * D;
    }
    const int nby = y ? ceil_div(Ly, block_size) : 0;
    if (pool_sm100_supported(x, y, H, D, block_size) && (uintptr_t)px % 8 == 0 && (!y || (uintptr_t)py % 8 == 0))
        return pool_sm100_launch(x, Lx, px, y, Ly, py, nby_all, B, H, D, block_size, stream, zero, n_zero, status_mirror);
    View4 vx = make_view(x), vy = y ? make_view(y) : vx;
    dim3 grid(nbx + nby, H, B);
    const bool vec = pool_vec_ok(x, D) && (!y || pool_vec_ok(y, D));
    const int lanes = D / 8;
    if (vec && D % 8 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && ((uintptr_t)px % 16 == 0) &&
        (!y || (uintptr_t)py % 16 == 0)) {
        constexpr int items_per_cta = POOL_THREADS / 32 / WA_POOL_SPLIT;
        const long long items = (long long)B * H * (nbx + nby);
        const long long ctas = (items + items_per_cta - 1) / items_per_cta;
        WA_REQUIRE(ctas < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_pool_blocks: too many blocks");
        pool_warp_kernel<WA_POOL_UNROLL, WA_POOL_SPLIT><<<(unsigned)ctas, POOL_THREADS, 0, stream>>>(
            vx, Lx, H, D, block_size, nbx, Lx % block_size == 0, px, vy, Ly, nby, y_aligned, py, nby_all, B, zero, n_zero);
    } else if (vec) {
        const int rows = POOL_THREADS / (D / 8);
        const size_t smem = (size_t)rows * D * sizeof(double);
        WA_REQUIRE(smem <= 48 * 1024, WA_ERR_UNSUPPORTED, "wa_pool_blocks: D=%d too large", D);
        pool_blocks_kernel<true><<<grid, POOL_THREADS, smem, stream>>>(vx, Lx, H, D, block_size, nbx, Lx % block_size == 0,
                                                                       px, vy, Ly, nby, y_aligned, py, nby_all, zero, n_zero);
    } else {
        const int rows = D >= POOL_THREADS ? 1 : POOL_THREADS / D;
        const size_t smem = (size_t)rows * (D < POOL_THREADS ? D : POOL_THREADS) * sizeof(double);
        pool_blocks_kernel<false><<<grid, POOL_THREADS, smem, stream>>>(vx, Lx, H, D, block_size, nbx, Lx % block_size == 0,
                                                                        px, vy, Ly, nby, y_aligned, py, nby_all, zero, n_zero);
    }
    return check_launch("wa_pool_blocks");
}
}  // namespace wa

extern "C" int wa_pool_blocks(const wa_tensor4 *x, int B, int L, int H, int D, int block_size,
                              float *pooled, void *stream) {
    WA_REQUIRE(x && x->ptr && pooled, WA_ERR_ARG, "wa_pool_blocks: null pointer");
    WA_REQUIRE(valid_dtype(x->dtype), WA_ERR_ARG, "wa_pool_blocks: bad dtype %d", x->dtype);
    WA_REQUIRE(B > 0 && L > 0 && H > 0 && D > 0 && block_size > 0, WA_ERR_ARG,
               "wa_pool_blocks: sizes must be positive (B=%d L=%d H=%d D=%d block=%d)", B, L, H, D,
               block_size);
    WA_REQUIRE(H <= 65535 && B <= 65535, WA_ERR_UNSUPPORTED, "wa_pool_blocks: B, H must be <= 65535");
    return pool_launch(x, L, pooled, nullptr, 0, nullptr, B, H, D, block_size, (cudaStream_t)stream, nullptr, 0, 0);
}

extern "C" int wa_route_scores(const float *q_pooled, const float *k_pooled, int B, int H, int Nq,
                               int Nkv, int D, float *block_attn, void *stream) {
    WA_REQUIRE(q_pooled && k_pooled && block_attn, WA_ERR_ARG, "wa_route_scores: null pointer");
    WA_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nkv > 0 && D > 0, WA_ERR_ARG,
               "wa_route_scores: sizes must be positive");
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_route_scores: too many rows");
    const float scale = (float)pow((double)D, -0.5);
    route_scores_kernel<<<(unsigned)rows, SCORE_THREADS, 0, (cudaStream_t)stream>>>(
        q_pooled, k_pooled, Nq, Nkv, D, scale, block_attn);
    return check_launch("wa_route_scores");
}

namespace wa {
int route_select_launch(const float *block_attn, int B, int H, int Nq, int Nkv, double tau_min,
                        double tau_max, const int32_t *fixed_num_per_head, int32_t *index,
                        int32_t *num, uint8_t *mask, float *thresholds, float *gini_scratch,
                        cudaStream_t stream) {
    int n_pow2 = 1;
    while (n_pow2 < Nkv) n_pow2 <<= 1;
    WA_REQUIRE(n_pow2 <= 16384, WA_ERR_UNSUPPORTED,
               "wa_route_select: at most 16384 key blocks per row, got %d", Nkv);
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_route_select: too many rows");
    const size_t smem = (size_t)n_pow2 * sizeof(unsigned long long);
    int threads = n_pow2 / 2;
    threads = threads < 32 ? 32 : (threads > 1024 ? 1024 : threads);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(route_sort_kernel,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail((int)e, "wa_route_select: %s", cudaGetErrorString(e));
    }
    route_sort_kernel<<<(unsigned)rows, threads, smem, stream>>>(block_attn, Nkv, n_pow2, index,
                                                                 gini_scratch);
    int rc = check_launch("wa_route_select(sort)");
    if (rc) return rc;
    route_count_kernel<<<(unsigned)rows, SELECT_THREADS, 0, stream>>>(
        block_attn, index, gini_scratch, B, H, Nq, Nkv, (float)tau_min, (float)(tau_max - tau_min),
        fixed_num_per_head, num, mask, thresholds);
    return check_launch("wa_route_select(count)");
}
}  // namespace wa

namespace wa {
// With a batch a CTA takes 32 rows and 32 tiles of logits at a time.  Two rounds of rows pay up to 64 keys (37 rows over 37: 16.5 us against 22.6);
// beyond, one round of rows or of tiles does (25 rows over 74: 14.7 against 20; whole calls: 37 over 74 144.9 against 147.8,
// but 37 over 110, two rounds of both, 108.7 against 101.6).
// Without, a warp per row, up to eight rows per CTA.  While K and V are compressed beside it, two CTAs at most, of sixteen warps (36 rows over
// 36 of 12 heads, whole calls: 70.1 us with four of eight warps, 62.3 with one of 32, 61.6), but one of 32 where the compression
// is cut into more shares beside that, or fits beside that only (SchedJob::one_part; of 16 heads 18 rows over 18 46.9 -> 44.0, 17 over 34
// 68.4 -> 62.7), and one of sixteen where that is a row per warp
// of few keys (10 rows over 20 of 8 heads 51.6 us with two, 49.3 with one; 11 over 33 of 12 44.2 and 42.9; but 14 over 56 79.7 and 80.8).
int route_short_parts(int B, int Nq, int Nkv, int D, bool beside) {
    const bool one_round = (long long)B * Nq <= RH_WARPS || (long long)B * ((Nq + 15) / 16) * ((Nkv + 7) / 8) <= RH_WARPS;
    if (D != 128 || Nkv > RH_MAX_KEYS || (long long)B * Nq > RH_MAX_ROWS || (B > 1 && Nkv > 64 && !one_round)) return 0;
    int parts = 1;
    while (B == 1 && parts * (beside && Nkv <= 48 && Nq > 8 ? 16 : 8) < Nq && parts < (beside ? 2 : 8)) parts <<= 1;
    return parts;
}

int route_fused_launch(const float *q_pooled, const float *k_pooled, int B, int H, int Nq, int Nkv, int D, double tau_min,
                       double tau_max, const int32_t *fixed_num_per_head, float *sorted, int32_t *index, int32_t *num,
                       float *thresholds, float *gini, int *counters, const SchedJob &job_in, cudaStream_t stream, bool whole_order) {
    int n_pow2 = 1;
    while (n_pow2 < Nkv) n_pow2 <<= 1;
    WA_REQUIRE(n_pow2 <= 16384, WA_ERR_UNSUPPORTED, "wa_hsa_forward(routing): at most 16384 key blocks per row, got %d", Nkv);
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_hsa_forward(routing): too many rows");
    int threads = n_pow2 / 2;
    threads = threads < 256 ? 256 : (threads > 1024 ? 1024 : threads);
    // A key per thread up to 512 key blocks: 45 passes through shared memory took 13 of a row's 19 us there, with shuffles 4 (whole calls
    // with 256 and 512 threads, 74 rows of 12 heads over 257 blocks: 190 and 175 us; over 512: 242 and 229).  Beyond, a row's CTA
    // of 1024 threads fills half an SM, and what the sort gains is lost on the other steps (512 and 1024 threads, 74 over 585: 301 and
    // 299 us; over 700: 316 and 315; over 1024: 388 and 389; 37 over 513: 201 and 192).
    if (n_pow2 == 512) threads = 512;
    const int key_slots = n_pow2 > threads ? n_pow2 : threads;
    const size_t smem = (size_t)key_slots * sizeof(unsigned long long) + (size_t)Nkv * sizeof(float);
    int sms = sm_count();
    const float scale = (float)pow((double)D, -0.5), span = (float)(tau_max - tau_min);
    const long long bh = (long long)B * H;

    const int two_parts = ((uintptr_t)q_pooled % 16 == 0) && ((uintptr_t)k_pooled % 16 == 0) ? route_short_parts(B, Nq, Nkv, D, job_in.release_at_start) : 0;
    const int parts = job_in.one_part && two_parts > 0 ? 1 : two_parts;
    const bool short_rows = parts > 0;
    // route_topk_kernel, whatever the size -- unless the call's keys and values are compressed meanwhile, which is the longer of the two for
    // short rows: a CTA per row takes room on most SMs from its clusters (8 heads, 10 query blocks over 30, whole calls: 42.0 us, with a
    // CTA per head 39.4; 12 heads, 7 over 19 38.3 and 35.4; 2 items of 24 heads, 6 over 22 68.8 and 67.4)
    const bool by_count = fixed_num_per_head && !whole_order && !(short_rows && job_in.release_at_start);
    if (!by_count && short_rows) {
        const auto launch = [&](auto width, auto warps) -> cudaError_t {
            constexpr int K = decltype(width)::value, WARPS = decltype(warps)::value, ALONE = 190 * 1024;
            const auto kernel = route_head_kernel<K, WARPS>;
            static PerDeviceOnce attr_set;
            if (!attr_set.done()) {
                const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ALONE);
                if (e != cudaSuccess) return e;
                attr_set.mark();
            }
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(H * parts);
            cfg.blockDim = dim3(WARPS * 32);
            cfg.dynamicSmemBytes = (size_t)B * ((Nq + parts - 1) / parts) * K * 32 * sizeof(float);      // at most 32 KB
            // Where the chip has room for every CTA of the compression beside these, they keep their SMs to themselves: they are the longer chain
            // (12 heads, 6 query blocks over 6 29.3 -> 28.8 us a call, 36 over 36 of 64 tokens 62.7 -> 61.5).
            if (job_in.beside_sms > 0 && H * parts + job_in.beside_sms <= sm_count()) cfg.dynamicSmemBytes = ALONE;
            cfg.stream = stream;
            cudaLaunchAttribute attr[2];
            cfg.attrs = attr;
            cfg.numAttrs = 0;
            if (parts > 1) {      // a cluster of one costs the launches around it (8 rows over 8, whole call: 30.1 us with, 27.4 without)
                attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
                attr[cfg.numAttrs].val.clusterDim.x = parts;
                attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
                ++cfg.numAttrs;
            }
            if (pdl_enabled()) {
                attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
                attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
                ++cfg.numAttrs;
            }
            return cudaLaunchKernelEx(&cfg, kernel, q_pooled, k_pooled, B, H, Nq, Nkv, scale, (float)tau_min, span, fixed_num_per_head, index, num,
                                      thresholds, counters, job_in, (128 * 128 / 4 + H * parts - 1) / (H * parts) * 4);
        };
        // Eight warps, or sixteen where a row has up to sixteen tiles of logits (4 rows over 79: 14.4 us with eight, 12.4 with sixteen).
        const auto launch_width = [&](auto few, auto many) {
            return Nkv <= 32 ? launch(std::integral_constant<int, 1>(), few)
                             : Nkv <= 64 ? launch(std::integral_constant<int, 2>(), few) : launch(std::integral_constant<int, 4>(), many);
        };
        const std::integral_constant<int, 8> w8;
        const std::integral_constant<int, 16> w16;
        const std::integral_constant<int, RH_WARPS> w32;
        const cudaError_t e = B > 1 || job_in.one_part ? launch_width(w32, w32) : job_in.release_at_start && Nq > 8 ? launch_width(w16, w16) : launch_width(w8, w16);
        if (e != cudaSuccess) return fail((int)e, "wa_hsa_forward(routing of short rows): %s", cudaGetErrorString(e));
        return check_launch("wa_hsa_forward(routing of short rows)");
    }

    // Scoring in a launch of its own costs about 2 us and saves every row its pass over the head's keys: from 65 536 logits on it
    // pays (444 rows over 256 key blocks, the whole call: 130.7 -> 127.8 us; 888 over 122: 227.9 -> 222.9; 888 over 512: 706.6 ->
    // 686.4), at 444 rows over 37 the row kernel alone is 2.7 us faster.
    const bool logits_ready = D == 128 && rows * Nkv >= 65536 && ((uintptr_t)q_pooled % 16 == 0) && ((uintptr_t)k_pooled % 16 == 0);
    if (logits_ready) {
        // rows per CTA: those that finish first, a tile of 128 keys being 2.1 us per 16 rows and about 1 us besides
        const int tiles = (Nkv + RL_TILE - 1) / RL_TILE, row_tiles = (Nq + 15) / 16;
        auto cost = [&](int mt) { return ((bh * ((row_tiles + mt - 1) / mt) * tiles + sms - 1) / sms) * (21 * mt + 10); };
        int mt = RL_MAX_MT;
        for (int m = RL_MAX_MT - 1; m >= 1; --m)
            if (cost(m) < cost(mt)) mt = m;
        const int groups = (row_tiles + mt - 1) / mt;
        const long long units = bh * groups * tiles;
        const auto launch = [&](auto width) -> cudaError_t {
            constexpr int MT = decltype(width)::value, BYTES = MT * 16 * 128 * (int)sizeof(double);
            const auto kernel = route_logits_kernel<MT>;
            static PerDeviceOnce attr_set;
            if (!attr_set.done()) {
                const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES);
                if (e != cudaSuccess) return e;
                attr_set.mark();
            }
            return launch_dependent(kernel, dim3((unsigned)(units < sms ? units : sms)), dim3(RL_WARPS * 32), BYTES, stream, q_pooled, k_pooled, Nq, Nkv,
                                    scale, sorted, groups, tiles, units);
        };
        const cudaError_t e = mt == 1 ? launch(std::integral_constant<int, 1>()) : mt == 2 ? launch(std::integral_constant<int, 2>())
                            : mt == 3 ? launch(std::integral_constant<int, 3>()) : mt == 4 ? launch(std::integral_constant<int, 4>())
                                      : launch(std::integral_constant<int, 5>());
        if (e != cudaSuccess) return fail((int)e, "wa_hsa_forward(logits): %s", cudaGetErrorString(e));
        if (const int rc = check_launch("wa_hsa_forward(logits)")) return rc;
    }
    const int gate_per_cta = (int)((128 * 128 / 4 + rows - 1) / rows) * 4;
    if (rows < sms) sms = (int)rows;
    const int slots = (int)((rows + sms - 1) / sms);
    if (by_count) {
        const auto launch = [&](auto threads_c, auto values_c) -> cudaError_t {
            constexpr int T = decltype(threads_c)::value, V = decltype(values_c)::value;
            const size_t bytes = V > 0 && logits_ready ? 0 : (size_t)Nkv * sizeof(float);       // at most 64 KB
            const auto kernel = route_topk_kernel<T, V>;
            static PerDeviceOnce attr_set;
            if (!attr_set.done()) {
                const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (V > 0 ? T * V : 16384) * (int)sizeof(float));
                if (e != cudaSuccess) return e;
                attr_set.mark();
            }
            return launch_dependent(kernel, dim3((unsigned)((long long)sms * slots) + 1), dim3(T), bytes, stream, q_pooled, k_pooled, H, Nq, Nkv, D,
                                    scale, fixed_num_per_head, sorted, index, num, job_in, (int)rows, gate_per_cta, sms, slots, logits_ready ? 1 : 0);
        };
        using std::integral_constant;
        const cudaError_t e = logits_ready && Nkv <= 256    ? launch(integral_constant<int, 128>(), integral_constant<int, 2>())
                              : logits_ready && Nkv <= 512  ? launch(integral_constant<int, 128>(), integral_constant<int, 4>())
                              : Nkv <= 256                  ? launch(integral_constant<int, 256>(), integral_constant<int, 1>())
                              : Nkv <= 2048                 ? launch(integral_constant<int, 256>(), integral_constant<int, 8>())
                                                            : launch(integral_constant<int, 512>(), integral_constant<int, 0>());
        if (e != cudaSuccess) return fail((int)e, "wa_hsa_forward(routing by count): %s", cudaGetErrorString(e));
        return check_launch("wa_hsa_forward(routing by count)");
    }
    const dim3 grid((unsigned)((long long)sms * slots));
    SchedJob job = job_in;
    job.release_dependents_after_rows = pdl_mode() == 2;
    const auto kernel = !logits_ready ? route_fused_kernel<false, 1024> : threads <= 512 ? route_fused_kernel<true, 512> : route_fused_kernel<true, 1024>;
    if (smem > 24 * 1024) {   // static shared memory of the kernel takes ~22 KB of the default 48 KB
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail((int)e, "wa_hsa_forward(routing): %s", cudaGetErrorString(e));
    }
    const cudaError_t le = launch_dependent(kernel, grid, dim3(threads), smem, stream, q_pooled, k_pooled, B, H, Nq, Nkv, n_pow2, D, scale,
                                            (float)tau_min, span, fixed_num_per_head, sorted, index, num, thresholds, gini, counters, job,
                                            gate_per_cta, sms, slots, key_slots);
    if (le != cudaSuccess) return fail((int)le, "wa_hsa_forward(routing): %s", cudaGetErrorString(le));
    return check_launch("wa_hsa_forward(routing)");
}
}  // namespace wa

extern "C" int wa_route_select(const float *block_attn, int B, int H, int Nq, int Nkv,
                               double tau_min, double tau_max, const int32_t *fixed_num_per_head,
                               int32_t *index, int32_t *num, uint8_t *mask, float *thresholds,
                               float *gini_scratch, void *stream) {
    WA_REQUIRE(block_attn && index && num && thresholds && gini_scratch, WA_ERR_ARG,
               "wa_route_select: null pointer");
    WA_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nkv > 0, WA_ERR_ARG,
               "wa_route_select: sizes must be positive");
    return route_select_launch(block_attn, B, H, Nq, Nkv, tau_min, tau_max, fixed_num_per_head,
                               index, num, mask, thresholds, gini_scratch, (cudaStream_t)stream);
}

extern "C" int wa_map_to_index(const uint8_t *mask, int B, int H, int Nq, int Nkv, int32_t *index,
                               int32_t *num, void *stream) {
    WA_REQUIRE(mask && index && num, WA_ERR_ARG, "wa_map_to_index: null pointer");
    WA_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nkv > 0, WA_ERR_ARG,
               "wa_map_to_index: sizes must be positive");
    const long long rows = (long long)B * H * Nq;
    const int warps = 4;
    map_to_index_kernel<<<(unsigned)((rows + warps - 1) / warps), warps * 32, 0,
                          (cudaStream_t)stream>>>(mask, rows, Nkv, index, num);
    return check_launch("wa_map_to_index");
}

// ------------------------------------------------------------------------------------------------
// wa_route_select_static: the same selection with its per-row scratch inside the library.
//
// For callers that are not allowed to allocate device memory at the point where routing runs: a
// serving process that hands out its whole HBM budget at start-up and forbids later allocation, a
// plugin whose host owns the allocator, or a loop that must not call anything that can synchronise
// the device (cudaMalloc / cudaFree do).  Such a caller has nowhere to get the B*H*Nq floats of
// Gini scratch from, so this entry point keeps them in a file-scope device array of fixed size.
// Every GPU that loads the library carries that array (256 KiB) until the process exits.
// ------------------------------------------------------------------------------------------------
namespace wa {
constexpr int STATIC_SELECT_MAX_ROWS = WA_ROUTE_SELECT_STATIC_MAX_ROWS;
static __device__ __align__(256) float g_select_scratch[STATIC_SELECT_MAX_ROWS];

// The array's name is only a host-side handle; the device address comes from the runtime, once
// per device, with that device current.
static float *select_scratch_address() {
    constexpr int MAX_DEVICES = 64;
    static float *cached[MAX_DEVICES] = {nullptr};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
        fail(WA_ERR_DEVICE, "wa_route_select_static: no usable current device");
        return nullptr;
    }
    if (!cached[dev]) {
        float *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_select_scratch);
        if (e != cudaSuccess || !ptr) {
            fail((int)e, "wa_route_select_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return nullptr;
        }
        cached[dev] = ptr;
    }
    return cached[dev];
}
}  // namespace wa

extern "C" int wa_route_select_static(const float *block_attn, int B, int H, int Nq, int Nkv, double tau_min,
                                      double tau_max, const int32_t *fixed_num_per_head, int32_t *index,
                                      int32_t *num, uint8_t *mask, float *thresholds, void *stream) {
    WA_REQUIRE(block_attn && index && num && thresholds, WA_ERR_ARG, "wa_route_select_static: null pointer");
    WA_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nkv > 0, WA_ERR_ARG, "wa_route_select_static: sizes must be positive");
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows <= STATIC_SELECT_MAX_ROWS, WA_ERR_UNSUPPORTED,
               "wa_route_select_static: %lld rows (B*H*Nq) exceed the built-in scratch of %d rows; "
               "use wa_route_select with caller-provided scratch",
               rows, STATIC_SELECT_MAX_ROWS);
    float *scratch = select_scratch_address();
    if (!scratch) return WA_ERR_DEVICE;
    // Nothing in the scratch has to start at zero: pass A writes every row's Gini term before pass B reads it.
    return route_select_launch(block_attn, B, H, Nq, Nkv, tau_min, tau_max, fixed_num_per_head, index, num, mask,
                               thresholds, scratch, (cudaStream_t)stream);
}

extern "C" int wa_route_local_candidates(const float *q_pooled, const float *k_pooled_local, int B, int H, int Nq, int Nloc, int D,
                                         int block_lo, int kcap, unsigned long long *candidates, void *stream) {
    const char *what = "wa_route_local_candidates";
    WA_REQUIRE(q_pooled && candidates && (k_pooled_local || Nloc == 0), WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(B > 0 && H > 0 && Nq > 0 && Nloc >= 0 && D > 0 && kcap > 0 && block_lo >= 0, WA_ERR_ARG, "%s: bad sizes", what);
    int n_pow2 = 1;
    while (n_pow2 < Nloc) n_pow2 <<= 1;
    WA_REQUIRE(n_pow2 <= 16384, WA_ERR_UNSUPPORTED, "%s: at most 16384 key blocks per shard, got %d", what, Nloc);
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many rows", what);
    int threads = n_pow2 / 2;
    threads = threads < 256 ? 256 : (threads > 1024 ? 1024 : threads);
    const size_t smem = (size_t)n_pow2 * sizeof(unsigned long long) + (size_t)(Nloc > 0 ? Nloc : 1) * sizeof(float);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(route_local_candidates_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
    }
    route_local_candidates_kernel<<<(unsigned)rows, threads, smem, (cudaStream_t)stream>>>(
        q_pooled, k_pooled_local, Nq, Nloc, n_pow2, D, (float)pow((double)D, -0.5), block_lo, kcap, candidates);
    return check_launch(what);
}

extern "C" int wa_route_merge_candidates(const unsigned long long *candidates, int W, int B, int H, int Nq, int kcap,
                                         const int32_t *topk_per_head, int Nkv_total, int block_lo, int block_hi, int index_stride,
                                         int32_t *local_index, int32_t *local_num, void *stream) {
    const char *what = "wa_route_merge_candidates";
    WA_REQUIRE(candidates && topk_per_head && local_index && local_num, WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(W > 0 && B > 0 && H > 0 && Nq > 0 && kcap > 0 && Nkv_total > 0 && block_lo >= 0 && block_hi >= block_lo, WA_ERR_ARG,
               "%s: bad sizes", what);
    WA_REQUIRE(index_stride >= kcap || index_stride >= block_hi - block_lo, WA_ERR_ARG,
               "%s: index rows of %d entries cannot hold the selection", what, index_stride);
    int n_pow2 = 1;
    while (n_pow2 < W * kcap) n_pow2 <<= 1;
    WA_REQUIRE(n_pow2 <= 4096, WA_ERR_UNSUPPORTED, "%s: at most 4096 candidates per row, got %d", what, W * kcap);
    const long long rows = (long long)B * H * Nq;
    WA_REQUIRE(rows < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many rows", what);
    route_merge_candidates_kernel<<<(unsigned)rows, 256, (size_t)n_pow2 * sizeof(unsigned long long), (cudaStream_t)stream>>>(
        candidates, W, rows, Nq, H, kcap, n_pow2, topk_per_head, Nkv_total, block_lo, block_hi, index_stride, local_index,
        local_num);
    return check_launch(what);
}
