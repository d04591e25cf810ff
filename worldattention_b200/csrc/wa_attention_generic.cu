// Shape-generic SIMT attention kernels: block-sparse branch, compressed ("linear") branch, gate and
// combine, shard-partial merge.
//
// These accept any head_dim <= 256, any block size, float32 or bf16 tensors in either
// `[B, L, H, D]` or `[B, H, N, D]` layout, and compute in float32.  They serve the shapes the
// tcgen05 kernel does not cover and are the in-library cross-check for it.  Stand-ins for
// wan/modules/hsa/block_sparse_torch.py:16-64 and wan/modules/hsa/attention.py:113-118, 246-259.
#include "wa_common.cuh"

namespace wa {

constexpr int GA_THREADS = 256;
constexpr int GA_WARPS = GA_THREADS / 32;
constexpr int GA_ROWS_PER_WARP = 4;
constexpr int GA_QT = GA_WARPS * GA_ROWS_PER_WARP;  // 32 query rows per CTA
constexpr int GA_TK = 32;                           // key tokens per shared-memory chunk
constexpr int GA_MAXD = 256;
constexpr int GA_DC = GA_MAXD / 32;                 // channels per lane

struct GenericAttnParams {
    View4 q, k, v;
    void *out;
    int out_dtype;
    long long osb, osl, osh;
    int H, Lq, Lkv, D;
    int q_block;    // query rows per routing block
    int q_tile;     // query rows per CTA (<= GA_QT, divides the work inside one routing block)
    int tiles_per_block;
    int kv_block;   // key tokens per block
    int n_kv_blocks;
    int dense;      // 1: visit every key block in order (no index / num)
    const int32_t *index;
    const int32_t *num;
    int index_stride;
    const int32_t *block_sizes;
    int round_in, round_out;
    float scale;
    float *lse;
    const int32_t *order;   // split kernel, not dense: routing rows in the order in which CTAs take them, or null
    int ahead, beside;      // split kernel: the next launch may start while this one runs; this one started while the one before it ran
};

__global__ void __launch_bounds__(GA_THREADS)
generic_attention_kernel(GenericAttnParams p) {
    extern __shared__ float ga_smem[];
    const int D = p.D;
    const int ldk = D + 1;
    float *qs = ga_smem;                 // [GA_QT][D]
    float *ks = qs + GA_QT * D;          // [GA_TK][D + 1]
    float *vs = ks + GA_TK * ldk;        // [GA_TK][D]

    const int qb = blockIdx.x / p.tiles_per_block;
    const int tile = blockIdx.x % p.tiles_per_block;
    const int h = blockIdx.y, b = blockIdx.z;
    const int row0 = qb * p.q_block + tile * p.q_tile;
    const int rows_here = max(0, min(min(p.q_tile, p.q_block - tile * p.q_tile), p.Lq - row0));
    if (rows_here <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // stage the query rows
    const long long qbase = (long long)b * p.q.sb + (long long)h * p.q.sh;
    for (int e = threadIdx.x; e < rows_here * D; e += GA_THREADS) {
        const int r = e / D, d = e % D;
        float x = load_elem(p.q.ptr, p.q.dtype, qbase + (long long)(row0 + r) * p.q.sl + d);
        qs[r * D + d] = p.round_in ? bf16_round_f(x) : x;
    }

    float m_i[GA_ROWS_PER_WARP], l_i[GA_ROWS_PER_WARP], acc[GA_ROWS_PER_WARP][GA_DC];
#pragma unroll
    for (int r = 0; r < GA_ROWS_PER_WARP; ++r) {
        m_i[r] = -INFINITY;
        l_i[r] = 0.f;
#pragma unroll
        for (int c = 0; c < GA_DC; ++c) acc[r][c] = 0.f;
    }

    const long long meta = ((long long)b * p.H + h) * (long long)((p.Lq + p.q_block - 1) / p.q_block) + qb;
    const int n_sel = p.dense ? p.n_kv_blocks : max(0, min(p.num[meta], p.index_stride));
    const int32_t *ids = p.dense ? nullptr : p.index + meta * (long long)p.index_stride;
    const long long kbase = (long long)b * p.k.sb + (long long)h * p.k.sh;
    const long long vbase = (long long)b * p.v.sb + (long long)h * p.v.sh;

    for (int s = 0; s < n_sel; ++s) {
        int id = p.dense ? s : ids[s];
        id = max(0, min(id, p.n_kv_blocks - 1));
        int size = p.block_sizes ? p.block_sizes[id] : p.Lkv - id * p.kv_block;
        size = max(0, min(size, min(p.kv_block, p.Lkv - id * p.kv_block)));
        for (int c0 = 0; c0 < size; c0 += GA_TK) {
            const int n_tok = min(GA_TK, size - c0);
            __syncthreads();
            for (int e = threadIdx.x; e < GA_TK * D; e += GA_THREADS) {
                const int t = e / D, d = e % D;
                float kx = 0.f, vx = 0.f;
                if (t < n_tok) {
                    const long long tok = (long long)id * p.kv_block + c0 + t;
                    kx = load_elem(p.k.ptr, p.k.dtype, kbase + tok * p.k.sl + d);
                    vx = load_elem(p.v.ptr, p.v.dtype, vbase + tok * p.v.sl + d);
                    if (p.round_in) {
                        kx = bf16_round_f(kx);
                        vx = bf16_round_f(vx);
                    }
                }
                ks[t * ldk + d] = kx;
                vs[t * D + d] = vx;
            }
            __syncthreads();

            // scores: lane = key token, four query rows per warp share each K element
            float sc[GA_ROWS_PER_WARP] = {0.f, 0.f, 0.f, 0.f};
            const float *krow = ks + lane * ldk;
            const float *q0 = qs + (warp * GA_ROWS_PER_WARP) * D;
            for (int d = 0; d < D; ++d) {
                const float kx = krow[d];
#pragma unroll
                for (int r = 0; r < GA_ROWS_PER_WARP; ++r) sc[r] = fmaf(q0[r * D + d], kx, sc[r]);
            }
#pragma unroll
            for (int r = 0; r < GA_ROWS_PER_WARP; ++r) {
                const float sv = lane < n_tok ? sc[r] * p.scale : -INFINITY;
                const float m_new = fmaxf(m_i[r], warp_max(sv));
                const float pr = lane < n_tok ? expf(sv - m_new) : 0.f;
                const float alpha = m_i[r] == -INFINITY ? 0.f : expf(m_i[r] - m_new);
                l_i[r] = l_i[r] * alpha + warp_sum(pr);
                m_i[r] = m_new;
#pragma unroll
                for (int c = 0; c < GA_DC; ++c) acc[r][c] *= alpha;
                sc[r] = pr;
            }
            for (int t = 0; t < n_tok; ++t) {
                float pt[GA_ROWS_PER_WARP];
#pragma unroll
                for (int r = 0; r < GA_ROWS_PER_WARP; ++r) pt[r] = __shfl_sync(0xffffffffu, sc[r], t);
#pragma unroll
                for (int c = 0; c < GA_DC; ++c) {
                    const int d = lane + 32 * c;
                    if (d < D) {
                        const float vx = vs[t * D + d];
#pragma unroll
                        for (int r = 0; r < GA_ROWS_PER_WARP; ++r) acc[r][c] = fmaf(pt[r], vx, acc[r][c]);
                    }
                }
            }
        }
    }

#pragma unroll
    for (int r = 0; r < GA_ROWS_PER_WARP; ++r) {
        const int lr = warp * GA_ROWS_PER_WARP + r;
        if (lr >= rows_here) continue;
        const int row = row0 + lr;
        const float inv = l_i[r] > 0.f ? 1.0f / l_i[r] : 0.f;
        const long long obase = (long long)b * p.osb + (long long)row * p.osl + (long long)h * p.osh;
#pragma unroll
        for (int c = 0; c < GA_DC; ++c) {
            const int d = lane + 32 * c;
            if (d < D) {
                float o = acc[r][c] * inv;
                if (p.round_out) o = bf16_round_f(o);
                store_elem(p.out, p.out_dtype, obase + d, o);
            }
        }
        if (p.lse && lane == 0)
            p.lse[((long long)b * p.H + h) * p.Lq + row] = l_i[r] > 0.f ? m_i[r] + logf(l_i[r]) : -INFINITY;
    }
}

// ------------------------------------------------------------------------------------------------
// head_dim 128: the same contract on the warp-level matrix instructions, with the accuracy of the float32 kernel above.
//
// Two warps share 16 of the CTA's 64 query rows, each with one half of a chunk's keys and sums of its own (merged at the
// end); chunks may span several routing blocks.  Operands are sums of bf16 parts without a remainder, and every product of
// parts is taken:
//   NS = 1  q, k and v are bf16 values (bf16 tensors, or `round_in`): one product for the scores; the float32
//           probabilities are three bf16 parts (8 + 8 + 8 bits of the significand), so P V takes three.
//   NS = 3  float32 operands, three parts each: nine products, of which the smallest still matter: a part is cut off, so
//           the second is up to 2^-7 and the third up to 2^-15 of its value and a product of both 2^-22.
// Parts are cut off, not rounded, so they keep the sign of their value, and a part that would be zero is a tiny
// number instead: infinities in V or K then give what a float32 product gives and not 0 * inf.
// The instruction's own accumulator cuts what does not fit its 24 bits, always toward zero: a sum carried in it through all
// products and keys was up to 2.6e-5 too small.  So each accumulation starts at zero and takes only the products of one
// 16-term step, smallest first; the steps are added with rounding in registers.
// Error against float64 (2-norm of the result), SIMT kernel -> this one: 75 float32 slots 3.8e-7 -> 1.8e-7, 2000 slots
// 9.2e-7 -> 2.6e-7, 4680 rounded keys 1.25e-6 -> 2.9e-7; the log-sum-exp has the same error within 6 % or less.
// The SIMT kernel above is bound by shared-memory reads (one per four multiply-adds).  12 heads, 1560 queries: a third of
// 4680 keys in 64-token blocks 1480 -> 238 us, 75 float32 slots 92 -> 57 us.
//
// DIRECT: keys and values that are bf16 in memory (aligned rows) go to shared memory by asynchronous copies, the next chunk
// while one is at work, with one barrier a chunk.  Float32 layers get there by rounding keys and values once (round_kv_kernel, see
// wa_hsa_forward) instead of in every CTA that selects them: 238 -> 202 us.  Rows of
// different counts then left a third of the chip idle at the end (mean 240 of 368 kcycles per SM): they are taken heaviest first
// (-> 156 us), and the linear branch's launch starts on what the last of them leave free (`ahead`, `beside`: the two branches
// 261 -> 216 us from the first's start to the second's end).
// ------------------------------------------------------------------------------------------------
constexpr int SA_ROWS = 64;                  // query rows of a CTA
constexpr int SA_THREADS = 256;
constexpr int SA_D = 128;
constexpr int SA_LD = SA_D + 8;              // bf16 elements of a shared-memory row: ldmatrix without bank conflicts
constexpr int sa_keys(int ns) { return ns == 1 ? 64 : 32; }
constexpr size_t sa_smem(int ns, int stages) { return (size_t)ns * (SA_ROWS + stages * 2 * sa_keys(ns)) * SA_LD * 2 + stages * 32; }

__device__ __forceinline__ uint32_t sa_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {   // from zero
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// two 8-column products of one step, from zero or onto what the step has summed up
__device__ __forceinline__ void mma_step(bool first, float (&x0)[4], float (&x1)[4], const uint32_t (&a)[4], const uint32_t (&b)[4]) {
    if (first) {
        mma16816_new(x0, a, b[0], b[1]);
        mma16816_new(x1, a, b[2], b[3]);
    } else {
        mma16816(x0, a, b[0], b[1]);
        mma16816(x1, a, b[2], b[3]);
    }
}
__device__ __forceinline__ void add4(float (&c)[4], const float (&x)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += x[i];
}

constexpr float SA_TINY = 2.3509887e-38f;    // 2^-125, a bf16 number
__device__ __forceinline__ float plain_nan(float x) { return x == x ? x : NAN; }   // one whose upper half is a NaN by itself
__device__ __forceinline__ float top_part(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ float rest_of(float x, float hi) {
    const float r = x - hi;
    return isinf(hi) || (r == 0.f && x != 0.f) ? copysignf(SA_TINY, x) : r;
}
// the upper halves of two floats as a bf16 pair (x in the low half)
__device__ __forceinline__ uint32_t top_pair(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }

template <int NS>
__device__ __forceinline__ void stage4(__nv_bfloat16 *dst, size_t part_stride, float4 x) {   // four elements of a row, NS parts
    if constexpr (NS == 1) {
        __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
        *reinterpret_cast<uint2 *>(dst) = make_uint2(*reinterpret_cast<uint32_t *>(&a), *reinterpret_cast<uint32_t *>(&b));
    } else {
        x = make_float4(plain_nan(x.x), plain_nan(x.y), plain_nan(x.z), plain_nan(x.w));
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            *reinterpret_cast<uint2 *>(dst + i * part_stride) = make_uint2(top_pair(x.x, x.y), top_pair(x.z, x.w));
            x = make_float4(rest_of(x.x, top_part(x.x)), rest_of(x.y, top_part(x.y)), rest_of(x.z, top_part(x.z)), rest_of(x.w, top_part(x.w)));
        }
    }
}
__device__ __forceinline__ float4 fetch4(const void *base, int dtype, long long off) {
    if (dtype == WA_F32) return *reinterpret_cast<const float4 *>((const float *)base + off);
    const uint2 raw = *reinterpret_cast<const uint2 *>((const __nv_bfloat16 *)base + off);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src, bool real) {      // zeros if not real
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}

template <int NS, bool DIRECT>
__global__ void __launch_bounds__(SA_THREADS, NS == 1 ? 2 : 1)
split_attention_kernel(GenericAttnParams p) {
    static_assert(!DIRECT || NS == 1, "asynchronous copies bring bf16 values");
    constexpr int KC = sa_keys(NS), KW = KC / 2, NT = KW / 8, RW = KC / 8;   // keys of a chunk and of a warp; 8-key tiles; rows a warp stages
    extern __shared__ __align__(16) uint8_t sa_raw[];
    __nv_bfloat16 *qs = reinterpret_cast<__nv_bfloat16 *>(sa_raw);   // [NS][SA_ROWS][SA_LD]
    __nv_bfloat16 *ks = qs + NS * SA_ROWS * SA_LD;                    // [NS][KC][SA_LD]
    __nv_bfloat16 *vs = ks + NS * KC * SA_LD;                         // [NS][KC][SA_LD]
    constexpr int STAGES = DIRECT ? 2 : 1, STAGE_ELEMS = 2 * NS * KC * SA_LD;
    unsigned *real = reinterpret_cast<unsigned *>(ks + STAGES * STAGE_ELEMS);   // per stage and warp: which of the rows it staged are real keys

    if (p.ahead) pdl_release_dependents();
    // what is left of the chip at the end of the launch before this one is used; whoever waits for this launch waits for both
    struct Both {
        int beside;
        __device__ ~Both() { if (beside) pdl_wait(); }
    } both{p.beside};
    int qb = blockIdx.x / p.tiles_per_block, h = blockIdx.y, b = blockIdx.z;
    const int tile = blockIdx.x % p.tiles_per_block, n_qb = (p.Lq + p.q_block - 1) / p.q_block;
    if (p.order) {
        const int item = p.order[qb];
        qb = item % n_qb;
        h = item / n_qb % p.H;
        b = item / n_qb / p.H;
    }
    const int row0 = qb * p.q_block + tile * p.q_tile;
    const int rows_here = max(0, min(min(p.q_tile, p.q_block - tile * p.q_tile), p.Lq - row0));
    if (rows_here <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, c2 = 2 * (lane & 3);
    const int rg = warp & 3, half_keys = warp >> 2;   // row group; which half of every chunk's keys

    const long long qbase = (long long)b * p.q.sb + (long long)h * p.q.sh;
    for (int r = warp; r < SA_ROWS; r += SA_THREADS / 32) {
        const float4 x = r < rows_here ? fetch4(p.q.ptr, p.q.dtype, qbase + (long long)(row0 + r) * p.q.sl + 4 * lane)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
        stage4<NS>(qs + r * SA_LD + 4 * lane, (size_t)SA_ROWS * SA_LD, x);
    }

    float o[SA_D / 8][4];
#pragma unroll
    for (int j = 0; j < SA_D / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    float mA = -INFINITY, mB = -INFINITY, lA = 0.f, lB = 0.f;   // rows g and g + 8 of the warp; l: this thread's columns only

    const long long meta = ((long long)b * p.H + h) * (long long)((p.Lq + p.q_block - 1) / p.q_block) + qb;
    const int n_sel = p.dense ? p.n_kv_blocks : max(0, min(p.num[meta], p.index_stride));
    const int32_t *ids = p.dense ? nullptr : p.index + meta * (long long)p.index_stride;
    const long long kbase = (long long)b * p.k.sb + (long long)h * p.k.sh, vbase = (long long)b * p.v.sb + (long long)h * p.v.sh;
    const long long total = (long long)n_sel * p.kv_block;
    const bool rows_mine = 16 * rg < rows_here;
    unsigned any_key = 0;   // this warp's half had a real key

    // ldmatrix addresses of this lane (A operand; B operand of the scores; B operand of P V, transposed)
    const uint32_t qa = sa_u32(qs + (16 * rg + (lane & 15)) * SA_LD + (lane >> 4) * 8);
    const uint32_t ka = sa_u32(ks + (half_keys * KW + (lane & 7) + (lane >> 4) * 8) * SA_LD + ((lane >> 3) & 1) * 8);
    const uint32_t va = sa_u32(vs + (half_keys * KW + (lane & 15)) * SA_LD + (lane >> 4) * 8);
    constexpr uint32_t Q_PART = SA_ROWS * SA_LD * 2, K_PART = KC * SA_LD * 2;   // bytes between the parts of an operand

    // this warp stages rows warp * RW ... of a chunk; lane i looks up the block of the i-th of them, then its token
    auto block_of = [&](long long c0) -> int {
        const long long j = c0 + warp * RW + lane;
        if (lane >= RW || j >= total) return -1;
        const int s = (int)(j / p.kv_block);
        return max(0, min(p.dense ? s : ids[s], p.n_kv_blocks - 1));
    };
    auto token_of = [&](long long c0, int id) -> int {
        if (id < 0) return -1;
        const int off = (int)((c0 + warp * RW + lane) % p.kv_block);
        int size = p.block_sizes ? p.block_sizes[id] : p.Lkv - id * p.kv_block;
        size = max(0, min(size, min(p.kv_block, p.Lkv - id * p.kv_block)));
        return off < size ? id * p.kv_block + off : -1;
    };
    int stage = 0, next_block = block_of(0);
    // DIRECT: the chunk at c0 into a stage; the blocks of the chunk behind it are looked up on the way
    auto copy_chunk = [&](long long c0, int to) {
        const int token = token_of(c0, next_block);
        next_block = block_of(c0 + KC);
        const unsigned found = __ballot_sync(0xffffffffu, token >= 0);
        if (lane == 0) real[to * 8 + warp] = found;
        const uint32_t dst = sa_u32(ks + to * STAGE_ELEMS + (warp * RW + (lane >> 4)) * SA_LD + (lane & 15) * 8);
#pragma unroll
        for (int r = 0; r < RW; r += 2) {
            const int t = __shfl_sync(0xffffffffu, token, r + (lane >> 4));
            const long long row = max(t, 0);
            copy16_async(dst + r * SA_LD * 2, (const __nv_bfloat16 *)p.k.ptr + kbase + row * p.k.sl + (lane & 15) * 8, t >= 0);
            copy16_async(dst + (KC + r) * SA_LD * 2, (const __nv_bfloat16 *)p.v.ptr + vbase + row * p.v.sl + (lane & 15) * 8, t >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (DIRECT && total > 0) copy_chunk(0, 0);

    for (long long c0 = 0; c0 < total; c0 += KC, stage ^= DIRECT ? 1 : 0) {
        if (DIRECT) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();      // this chunk has arrived, and the one before it, in the other stage, has been read
            if (c0 + KC < total) copy_chunk(c0 + KC, stage ^ 1);
        } else {
        __syncthreads();   // the chunk before this one has been read
        const int token = token_of(c0, block_of(c0));
        const unsigned found = __ballot_sync(0xffffffffu, token >= 0);
        if (lane == 0) real[warp] = found;
#pragma unroll
        for (int r0 = 0; r0 < RW; r0 += 4) {
            float4 kx[4], vx[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = __shfl_sync(0xffffffffu, token, r0 + i);
                kx[i] = vx[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (t >= 0) {
                    kx[i] = fetch4(p.k.ptr, p.k.dtype, kbase + (long long)t * p.k.sl + 4 * lane);
                    vx[i] = fetch4(p.v.ptr, p.v.dtype, vbase + (long long)t * p.v.sl + 4 * lane);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = warp * RW + r0 + i;
                stage4<NS>(ks + r * SA_LD + 4 * lane, (size_t)KC * SA_LD, kx[i]);
                stage4<NS>(vs + r * SA_LD + 4 * lane, (size_t)KC * SA_LD, vx[i]);
            }
        }
        __syncthreads();
        }
        const uint32_t at = stage * STAGE_ELEMS * 2;      // bytes
        if (!rows_mine) continue;
        unsigned keep = 0;   // this warp's keys that are real
#pragma unroll
        for (int w = 0; w < 4; ++w) keep |= real[stage * 8 + 4 * half_keys + w] << (w * RW);
        if (keep == 0) continue;
        any_key = 1;
        const bool full = keep == (KW == 32 ? ~0u : (1u << (KW & 31)) - 1);

        float sc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) sc[j][0] = sc[j][1] = sc[j][2] = sc[j][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < SA_D / 16; ++kk) {
            uint32_t a[NS][4];
#pragma unroll
            for (int i = 0; i < NS; ++i) ldsm4(a[i], qa + i * Q_PART + kk * 32);
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                float x0[4], x1[4];   // this step's 16 channels
#pragma unroll
                for (int i = NS - 1; i >= 0; --i) {
                    uint32_t kb[4];
                    ldsm4(kb, ka + at + i * K_PART + (uint32_t)(j * 8 * SA_LD + kk * 16) * 2);
#pragma unroll
                    for (int u = NS - 1; u >= 0; --u) mma_step(i == NS - 1 && u == NS - 1, x0, x1, a[u], kb);
                }
                add4(sc[j], x0);
                add4(sc[j + 1], x1);
            }
        }
        // scale, mask, running maximum
        float xA = -INFINITY, xB = -INFINITY;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
#pragma unroll
            for (int u = 0; u < 4; ++u) sc[j][u] *= p.scale;
            if (!full) {
                if (!((keep >> (8 * j + c2)) & 1)) sc[j][0] = sc[j][2] = -INFINITY;
                if (!((keep >> (8 * j + c2 + 1)) & 1)) sc[j][1] = sc[j][3] = -INFINITY;
            }
            xA = fmaxf(xA, fmaxf(sc[j][0], sc[j][1]));
            xB = fmaxf(xB, fmaxf(sc[j][2], sc[j][3]));
        }
#pragma unroll
        for (int w = 1; w < 4; w <<= 1) {
            xA = fmaxf(xA, __shfl_xor_sync(0xffffffffu, xA, w));
            xB = fmaxf(xB, __shfl_xor_sync(0xffffffffu, xB, w));
        }
        const float nA = fmaxf(mA, xA), nB = fmaxf(mB, xB);
        const float fA = mA == -INFINITY ? 0.f : expf(mA - nA), fB = mB == -INFINITY ? 0.f : expf(mB - nB);
        mA = nA; mB = nB;
        lA *= fA; lB *= fB;
        const float eA = nA == -INFINITY ? 0.f : nA, eB = nB == -INFINITY ? 0.f : nB;   // only scores of -inf so far: weights of zero
#pragma unroll
        for (int j = 0; j < SA_D / 8; ++j) { o[j][0] *= fA; o[j][1] *= fA; o[j][2] *= fB; o[j][3] *= fB; }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            sc[j][0] = expf(sc[j][0] - eA); sc[j][1] = expf(sc[j][1] - eA);
            sc[j][2] = expf(sc[j][2] - eB); sc[j][3] = expf(sc[j][3] - eB);
            if (!full) {
                if (!((keep >> (8 * j + c2)) & 1)) sc[j][0] = sc[j][2] = 0.f;
                if (!((keep >> (8 * j + c2 + 1)) & 1)) sc[j][1] = sc[j][3] = 0.f;
            }
            lA += sc[j][0] + sc[j][1];
            lB += sc[j][2] + sc[j][3];
        }
        // O += P V, 16 keys at a time
#pragma unroll
        for (int kk = 0; kk < KW / 16; ++kk) {
            uint32_t a[3][4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {   // a0: row g, first 8 keys; a1: row g + 8; a2, a3: the same of the last 8 keys
                float x = sc[2 * kk + (u >> 1)][2 * (u & 1)], y = sc[2 * kk + (u >> 1)][2 * (u & 1) + 1];
                const float tx = x > 0.f ? SA_TINY : 0.f, ty = y > 0.f ? SA_TINY : 0.f;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    a[i][u] = top_pair(x, y);
                    x = fmaxf(x - top_part(x), tx);
                    y = fmaxf(y - top_part(y), ty);
                }
            }
#pragma unroll
            for (int j = 0; j < SA_D / 8; j += 2) {
                float x0[4], x1[4];   // this step's 16 keys
#pragma unroll
                for (int i = NS - 1; i >= 0; --i) {
                    uint32_t vb[4];
                    ldsm4_t(vb, va + at + i * K_PART + (uint32_t)(kk * 16 * SA_LD + j * 8) * 2);
#pragma unroll
                    for (int u = 2; u >= 0; --u) mma_step(i == NS - 1 && u == 2, x0, x1, a[u], vb);
                }
                add4(o[j], x0);
                add4(o[j + 1], x1);
            }
        }
    }
#pragma unroll
    for (int w = 1; w < 4; w <<= 1) {
        lA += __shfl_xor_sync(0xffffffffu, lA, w);
        lB += __shfl_xor_sync(0xffffffffu, lB, w);
    }
    // merge the halves: the second one leaves maximum, sum and accumulator of its rows where the keys and values were
    __syncthreads();
    float4 *left = reinterpret_cast<float4 *>(ks) + (size_t)rg * (SA_D / 8 + 1) * 32 + lane;   // [SA_D / 8 + 1][32 lanes]
    static_assert(4 * (SA_D / 8 + 1) * 32 * 16 <= NS * 2 * KC * SA_LD * 2, "the accumulators fit where the keys and values were");
    if (lane == 0) real[warp] = any_key;
    if (half_keys && rows_mine) {
#pragma unroll
        for (int j = 0; j < SA_D / 8; ++j) left[j * 32] = make_float4(o[j][0], o[j][1], o[j][2], o[j][3]);
        left[SA_D / 8 * 32] = make_float4(mA, mB, lA, lB);
    }
    __syncthreads();
    if (half_keys || !rows_mine) return;
    any_key |= real[warp + 4];
    {
        const float4 other = left[SA_D / 8 * 32];
        const float nA = fmaxf(mA, other.x), nB = fmaxf(mB, other.y);
        const float fA = mA == -INFINITY ? 0.f : expf(mA - nA), fB = mB == -INFINITY ? 0.f : expf(mB - nB);
        const float hA = other.x == -INFINITY ? 0.f : expf(other.x - nA), hB = other.y == -INFINITY ? 0.f : expf(other.y - nB);
        mA = nA; mB = nB;
        lA = lA * fA + other.z * hA;
        lB = lB * fB + other.w * hB;
#pragma unroll
        for (int j = 0; j < SA_D / 8; ++j) {
            const float4 x = left[j * 32];
            o[j][0] = o[j][0] * fA + x.x * hA; o[j][1] = o[j][1] * fA + x.y * hA;
            o[j][2] = o[j][2] * fB + x.z * hB; o[j][3] = o[j][3] * fB + x.w * hB;
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int lr = 16 * rg + g + 8 * half, row = row0 + lr;
        if (lr >= rows_here) continue;
        const float l = half ? lB : lA, m = half ? mB : mA;
        // no key: zeros; keys, but every score -inf: not a number, as a softmax of them is
        const float inv = l > 0.f ? 1.0f / l : any_key && m == -INFINITY ? NAN : 0.f;
        const long long at = (long long)b * p.osb + (long long)row * p.osl + (long long)h * p.osh + c2;
#pragma unroll
        for (int j = 0; j < SA_D / 8; ++j) {
            float x = o[j][2 * half] * inv, y = o[j][2 * half + 1] * inv;
            __nv_bfloat162 xy = __floats2bfloat162_rn(x, y);
            if (p.out_dtype == WA_BF16) {
                *reinterpret_cast<__nv_bfloat162 *>((__nv_bfloat16 *)p.out + at + 8 * j) = xy;
            } else {
                if (p.round_out) {
                    x = __low2float(xy);
                    y = __high2float(xy);
                }
                *reinterpret_cast<float2 *>((float *)p.out + at + 8 * j) = make_float2(x, y);
            }
        }
        if (p.lse && c2 == 0) p.lse[((long long)b * p.H + h) * p.Lq + row] = l > 0.f ? m + logf(l) : -INFINITY;
    }
}

template <int NS, bool DIRECT>
int launch_split_attention(GenericAttnParams &p, int B, int n_q_blocks, cudaStream_t stream, const char *what) {
    p.q_tile = p.q_block < SA_ROWS ? p.q_block : SA_ROWS;
    p.tiles_per_block = ceil_div(p.q_block, p.q_tile);
    const long long gx = (long long)n_q_blocks * p.tiles_per_block;
    if (p.order && gx * p.H * B >= (1ll << 31)) p.order = nullptr;
    WA_REQUIRE(gx < (1ll << 31) && p.H <= 65535 && B <= 65535, WA_ERR_UNSUPPORTED, "%s: grid too large", what);
    static PerDeviceOnce attr_set;
    if (!attr_set.done()) {
        const cudaError_t e = cudaFuncSetAttribute(split_attention_kernel<NS, DIRECT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sa_smem(NS, DIRECT ? 2 : 1));
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
        attr_set.mark();
    }
    const dim3 grid = p.order ? dim3((unsigned)(gx * p.H * B)) : dim3((unsigned)gx, p.H, B);
    const size_t smem = sa_smem(NS, DIRECT ? 2 : 1);
    if (p.beside) {
        const cudaError_t e = launch_dependent(split_attention_kernel<NS, DIRECT>, grid, dim3(SA_THREADS), smem, stream, p);
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
    } else {
        split_attention_kernel<NS, DIRECT><<<grid, SA_THREADS, smem, stream>>>(p);
    }
    return check_launch(what);
}

// four consecutive elements of every row as one load or store
static bool rows_of_four(const void *ptr, int dtype, long long sb, long long sl, long long sh) {
    return (uintptr_t)ptr % (4 * dtype_size(dtype)) == 0 && sb % 4 == 0 && sl % 4 == 0 && sh % 4 == 0;
}

// Float32 keys and values -> bf16, contiguous `[B, L, H, D]` one behind the other at `dst`: what every CTA of the sparse branch would
// round for itself.  One pass over memory: 2 x 4680 tokens of 1536 channels (57 MB read, 29 written) 13.3 us
// alone; it runs beside the compression of the call's keys and values.
constexpr int RK_THREADS = 256, RK_AT_ONCE = 4;
__global__ void __launch_bounds__(RK_THREADS)
round_kv_kernel(View4 k, View4 v, long long pieces, int L, int H, int D8, uint4 *__restrict__ dst, int beside) {
    const View4 &src = blockIdx.y ? v : k;
    uint4 *out = dst + blockIdx.y * pieces;                      // a piece: eight channels
    float4 x[RK_AT_ONCE][2];
    const long long first = (long long)blockIdx.x * RK_THREADS * RK_AT_ONCE + threadIdx.x;
#pragma unroll
    for (int u = 0; u < RK_AT_ONCE; ++u) {
        const long long i = first + u * RK_THREADS;
        if (i < pieces) {
            const long long head = i / D8, token = head / H, b = token / L;
            const float4 *at = reinterpret_cast<const float4 *>((const float *)src.ptr + b * src.sb + (token - b * L) * src.sl + (head - token * H) * src.sh) +
                               2 * (i - head * D8);
            x[u][0] = __ldg(at);
            x[u][1] = __ldg(at + 1);
        }
    }
#pragma unroll
    for (int u = 0; u < RK_AT_ONCE; ++u) {
        const long long i = first + u * RK_THREADS;
        if (i < pieces) {
            const __nv_bfloat162 a = __floats2bfloat162_rn(x[u][0].x, x[u][0].y), b = __floats2bfloat162_rn(x[u][0].z, x[u][0].w);
            const __nv_bfloat162 c = __floats2bfloat162_rn(x[u][1].x, x[u][1].y), d = __floats2bfloat162_rn(x[u][1].z, x[u][1].w);
            out[i] = make_uint4(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b),
                                *reinterpret_cast<const uint32_t *>(&c), *reinterpret_cast<const uint32_t *>(&d));
        }
    }
    if (beside) pdl_wait();
}

bool round_kv_supported(const wa_tensor4 *k, const wa_tensor4 *v, int D) {
    const auto ok = [](const wa_tensor4 *t) {
        return t->dtype == WA_F32 && rows_of_four(t->ptr, t->dtype, t->stride_b, t->stride_l, t->stride_h);
    };
    return D == SA_D && ok(k) && ok(v);
}

int round_kv_launch(const wa_tensor4 *k, const wa_tensor4 *v, int B, int L, int H, int D, void *dst, bool beside, cudaStream_t stream) {
    const long long pieces = (long long)B * L * H * (D / 8), blocks = (pieces + RK_THREADS * RK_AT_ONCE - 1) / (RK_THREADS * RK_AT_ONCE);
    WA_REQUIRE(blocks < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_hsa_forward(rounding): too many keys");
    const View4 kv = make_view(k), vv = make_view(v);
    if (beside) {
        const cudaError_t e = launch_dependent(round_kv_kernel, dim3((unsigned)blocks, 2), dim3(RK_THREADS), 0, stream, kv, vv, pieces, L, H, D / 8, (uint4 *)dst, 1);
        if (e != cudaSuccess) return fail((int)e, "wa_hsa_forward(rounding): %s", cudaGetErrorString(e));
    } else {
        round_kv_kernel<<<dim3((unsigned)blocks, 2), RK_THREADS, 0, stream>>>(kv, vv, pieces, L, H, D / 8, (uint4 *)dst, 0);
    }
    return check_launch("wa_hsa_forward(rounding)");
}

int launch_generic_attention(GenericAttnParams &p, int B, int n_q_blocks, cudaStream_t stream,
                             const char *what) {
    WA_REQUIRE(p.D <= GA_MAXD, WA_ERR_UNSUPPORTED, "%s: head_dim %d > %d", what, p.D, GA_MAXD);
    if (p.D == SA_D && rows_of_four(p.q.ptr, p.q.dtype, p.q.sb, p.q.sl, p.q.sh) && rows_of_four(p.k.ptr, p.k.dtype, p.k.sb, p.k.sl, p.k.sh) &&
        rows_of_four(p.v.ptr, p.v.dtype, p.v.sb, p.v.sl, p.v.sh) && rows_of_four(p.out, p.out_dtype, p.osb, p.osl, p.osh)) {
        if (p.dense) {   // every block, any grouping of the rows
            n_q_blocks = ceil_div(p.Lq, SA_ROWS);
            p.q_block = SA_ROWS;
        }
        const bool exact = p.round_in || (p.q.dtype == WA_BF16 && p.k.dtype == WA_BF16 && p.v.dtype == WA_BF16);
        const auto rows_of_eight = [](const View4 &t) {      // 16 bytes at a time
            return t.dtype == WA_BF16 && (uintptr_t)t.ptr % 16 == 0 && t.sb % 8 == 0 && t.sl % 8 == 0 && t.sh % 8 == 0;
        };
        if (exact && rows_of_eight(p.k) && rows_of_eight(p.v)) return launch_split_attention<1, true>(p, B, n_q_blocks, stream, what);
        return exact ? launch_split_attention<1, false>(p, B, n_q_blocks, stream, what) : launch_split_attention<3, false>(p, B, n_q_blocks, stream, what);
    }
    p.q_tile = p.q_block < GA_QT ? p.q_block : GA_QT;
    p.tiles_per_block = ceil_div(p.q_block, p.q_tile);
    const long long gx = (long long)n_q_blocks * p.tiles_per_block;
    WA_REQUIRE(gx < (1ll << 31) && p.H <= 65535 && B <= 65535, WA_ERR_UNSUPPORTED, "%s: grid too large", what);
    const size_t smem = ((size_t)GA_QT * p.D + (size_t)GA_TK * (p.D + 1) + (size_t)GA_TK * p.D) * sizeof(float);
    static PerDeviceOnce attr_set;
    if (smem > 48 * 1024 && !attr_set.done()) {
        cudaError_t e = cudaFuncSetAttribute(generic_attention_kernel,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024);
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
        attr_set.mark();
    }
    dim3 grid((unsigned)gx, p.H, B);
    generic_attention_kernel<<<grid, GA_THREADS, smem, stream>>>(p);
    return check_launch(what);
}

// ------------------------------------------------------------------------------------------------
// Gate + combine.  One warp per (batch, token, head) vector.
// ------------------------------------------------------------------------------------------------
constexpr int GC_WARPS = 8;

__global__ void __launch_bounds__(GC_WARPS * 32)
gate_combine_kernel(View4 q, View4 sp, View4 li, void *out, int out_dtype, long long osb, long long osl,
                    long long osh, long long n_vec, int L, int H, int D, const void *gw, const void *gb,
                    int gdt, int round_gate) {
    extern __shared__ float gc_smem[];  // [GC_WARPS][D]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long vec = (long long)blockIdx.x * GC_WARPS + warp;
    if (vec >= n_vec) return;
    const int h = (int)(vec % H);
    const int l = (int)((vec / H) % L);
    const int b = (int)(vec / ((long long)H * L));
    float *qv = gc_smem + warp * D;
    const long long qoff = (long long)b * q.sb + (long long)l * q.sl + (long long)h * q.sh;
    for (int d = lane; d < D; d += 32) qv[d] = load_elem(q.ptr, q.dtype, qoff + d);
    __syncwarp();
    const long long soff = (long long)b * sp.sb + (long long)l * sp.sl + (long long)h * sp.sh;
    const long long loff = (long long)b * li.sb + (long long)l * li.sl + (long long)h * li.sh;
    const long long ooff = (long long)b * osb + (long long)l * osl + (long long)h * osh;
    for (int e = lane; e < D; e += 32) {
        float z;
        if (gw) {
            z = gb ? load_elem(gb, gdt, e) : 0.f;
            float dot = 0.f;
            for (int d = 0; d < D; ++d) dot = fmaf(qv[d], load_elem(gw, gdt, (long long)e * D + d), dot);
            z += dot;
        } else {
            z = qv[e];
        }
        float g = 1.0f / (1.0f + expf(-z));
        if (round_gate) g = bf16_round_f(g);
        const float s = load_elem(sp.ptr, sp.dtype, soff + e);
        const float x = load_elem(li.ptr, li.dtype, loff + e);
        store_elem(out, out_dtype, ooff + e, fmaf(x, g, s));
    }
}

// Same operation with the gate weight staged in shared memory (head_dim <= 128): a persistent grid, each warp takes eight
// (batch, token, head) vectors at a time and a lane produces outputs lane, lane + 32, ... of all of them, so that a weight
// read from shared memory serves eight multiply-adds (the dot products add up in the order of the channels, as before).
// Bound by shared-memory reads and the latency of its loads, which are therefore issued together: 18 720 vectors
// of 128 float32 channels 100 -> 47 us (one vector per warp took a read per multiply-add), -> 30 with the weight in 16-byte loads.
constexpr int GS_WARPS = 8;
constexpr int GS_VECS = 8;
constexpr int GS_MAXD = 128;
inline int gs_ld(int D) { return (D + 3) / 4 * 4 + 4; }   // floats of a staged row: 16-byte reads of neighbouring rows do not collide
inline size_t gs_smem(int D) { return ((size_t)(D + GS_WARPS * GS_VECS) * gs_ld(D) + D) * sizeof(float); }

__global__ void __launch_bounds__(GS_WARPS * 32)
gate_combine_smem_kernel(View4 q, View4 sp, View4 li, void *out, int out_dtype, long long osb, long long osl,
                         long long osh, long long n_vec, int L, int H, int D, int ld, const void *gw, const void *gb, int gdt,
                         int round_gate) {
    extern __shared__ __align__(16) float gs_smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *ws = gs_smem_raw;                                   // [D][ld], zero beyond column D
    float *qv = ws + D * ld + warp * GS_VECS * ld;             // [GS_WARPS][GS_VECS][ld]
    float *bs = ws + (D + GS_WARPS * GS_VECS) * ld;            // [D]
    if (gdt == WA_F32 && D == GS_MAXD && (reinterpret_cast<uintptr_t>(gw) & 15) == 0) {
        // sixteen 16-byte loads per thread, all on their way at once
        float4 w[GS_MAXD * GS_MAXD / 4 / (GS_WARPS * 32)];
#pragma unroll
        for (int i = 0; i < GS_MAXD * GS_MAXD / 4 / (GS_WARPS * 32); ++i)
            w[i] = __ldg(reinterpret_cast<const float4 *>(gw) + i * GS_WARPS * 32 + threadIdx.x);
#pragma unroll
        for (int i = 0; i < GS_MAXD * GS_MAXD / 4 / (GS_WARPS * 32); ++i)
            *reinterpret_cast<float4 *>(ws + (i * GS_WARPS + warp) * ld + lane * 4) = w[i];
    } else {
        for (int r = warp; r < D; r += GS_WARPS)
            for (int d = lane; d < ld; d += 32) ws[r * ld + d] = d < D ? load_elem(gw, gdt, (long long)r * D + d) : 0.f;
    }
    for (int e = threadIdx.x; e < D; e += GS_WARPS * 32) bs[e] = gb ? load_elem(gb, gdt, e) : 0.f;
    for (int e = lane; e < GS_VECS * ld; e += 32) qv[e] = 0.f;
    __syncthreads();
    const long long stride = (long long)gridDim.x * GS_WARPS * GS_VECS;
    for (long long v0 = ((long long)blockIdx.x * GS_WARPS + warp) * GS_VECS; v0 < n_vec; v0 += stride) {
        const int n = (int)min((long long)GS_VECS, n_vec - v0);
        // lane i places vector i; the others ask it
        const long long vec = min(v0 + (lane & (GS_VECS - 1)), n_vec - 1), row = vec / H;
        const int h_of = (int)(vec - row * H), b_of = (int)(row / L), l_of = (int)(row - (long long)b_of * L);
        auto place = [&](int i, int &b, int &l, int &h) {
            b = __shfl_sync(0xffffffffu, b_of, i);
            l = __shfl_sync(0xffffffffu, l_of, i);
            h = __shfl_sync(0xffffffffu, h_of, i);
        };
        __syncwarp();
        float x0[GS_VECS][GS_MAXD / 32];
#pragma unroll
        for (int i = 0; i < GS_VECS; ++i) {
            int b, l, h;
            place(i, b, l, h);
            const long long qoff = (long long)b * q.sb + (long long)l * q.sl + (long long)h * q.sh;
#pragma unroll
            for (int c = 0; c < GS_MAXD / 32; ++c) x0[i][c] = lane + 32 * c < D ? load_elem(q.ptr, q.dtype, qoff + lane + 32 * c) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < GS_VECS; ++i)
#pragma unroll
            for (int c = 0; c < GS_MAXD / 32; ++c)
                if (lane + 32 * c < D) qv[i * ld + lane + 32 * c] = x0[i][c];
        __syncwarp();
        float z[GS_MAXD / 32][GS_VECS];
#pragma unroll
        for (int c = 0; c < GS_MAXD / 32; ++c)
#pragma unroll
            for (int i = 0; i < GS_VECS; ++i) z[c][i] = lane + 32 * c < D ? bs[lane + 32 * c] : 0.f;
        for (int d = 0; d < D; d += 4) {
            float4 w[GS_MAXD / 32];
#pragma unroll
            for (int c = 0; c < GS_MAXD / 32; ++c)
                w[c] = lane + 32 * c < D ? *reinterpret_cast<const float4 *>(ws + (lane + 32 * c) * ld + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < GS_VECS; ++i) {
                const float4 x = *reinterpret_cast<const float4 *>(qv + i * ld + d);
#pragma unroll
                for (int c = 0; c < GS_MAXD / 32; ++c)
                    z[c][i] = fmaf(x.w, w[c].w, fmaf(x.z, w[c].z, fmaf(x.y, w[c].y, fmaf(x.x, w[c].x, z[c][i]))));
            }
        }
        float branch[2][GS_VECS][GS_MAXD / 32];
#pragma unroll
        for (int i = 0; i < GS_VECS; ++i) {
            int b, l, h;
            place(i, b, l, h);
            const long long soff = (long long)b * sp.sb + (long long)l * sp.sl + (long long)h * sp.sh;
            const long long loff = (long long)b * li.sb + (long long)l * li.sl + (long long)h * li.sh;
#pragma unroll
            for (int c = 0; c < GS_MAXD / 32; ++c) {
                const int e = lane + 32 * c;
                branch[0][i][c] = e < D ? load_elem(sp.ptr, sp.dtype, soff + e) : 0.f;
                branch[1][i][c] = e < D ? load_elem(li.ptr, li.dtype, loff + e) : 0.f;
            }
        }
#pragma unroll
        for (int i = 0; i < GS_VECS; ++i) {
            int b, l, h;
            place(i, b, l, h);
            const long long ooff = (long long)b * osb + (long long)l * osl + (long long)h * osh;
#pragma unroll
            for (int c = 0; c < GS_MAXD / 32; ++c) {
                const int e = lane + 32 * c;
                float gate = 1.0f / (1.0f + expf(-z[c][i]));
                if (round_gate) gate = bf16_round_f(gate);
                if (e < D && i < n) store_elem(out, out_dtype, ooff + e, fmaf(branch[1][i][c], gate, branch[0][i][c]));
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Merge shard partials of one softmax branch.
// ------------------------------------------------------------------------------------------------
__global__ void merge_partials_kernel(const float *__restrict__ outs, const float *__restrict__ lses, int G,
                                      long long rows, int D, float *__restrict__ out, float *__restrict__ lse) {
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    float m = -INFINITY;
    for (int g = 0; g < G; ++g) m = fmaxf(m, lses[(long long)g * rows + row]);
    const float m_safe = m == -INFINITY ? 0.f : m;
    float total = 0.f;
    for (int g = 0; g < G; ++g) total += expf(lses[(long long)g * rows + row] - m_safe);
    const float inv = total > 0.f ? 1.0f / total : 0.f;
    for (int d = lane; d < D; d += 32) {
        float acc = 0.f;
        for (int g = 0; g < G; ++g) {
            const float w = expf(lses[(long long)g * rows + row] - m_safe) * inv;
            acc = fmaf(w, outs[((long long)g * rows + row) * D + d], acc);
        }
        out[row * D + d] = acc;
    }
    if (lse && lane == 0) lse[row] = total > 0.f ? m_safe + logf(total) : -INFINITY;
}

// Merge of packed shard partials.  A record is [sparse (D) | linear (D) | lse_sparse, lse_linear, pad, pad] floats; `recv`
// holds G x vectors of them (shard-major).  One warp per (token, head) vector: per branch out = sum_g e^(lse_g - LSE) O_g,
// the sparse branch rounded to bf16 (the reference stores it so), the linear one kept in float32.
__global__ void __launch_bounds__(256)
merge_packed_kernel(const float *__restrict__ recv, int G, long long vectors, int D, int record,
                    __nv_bfloat16 *__restrict__ sparse_out, float *__restrict__ linear_out) {
    const long long vec = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (vec >= vectors) return;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int branch = 0; branch < 2; ++branch) {
        float m = -INFINITY;
        for (int g = 0; g < G; ++g) m = fmaxf(m, __ldg(recv + ((long long)g * vectors + vec) * record + 2 * D + branch));
        const float m_safe = m == -INFINITY ? 0.f : m;
        float total = 0.f;
        for (int g = 0; g < G; ++g) total += expf(__ldg(recv + ((long long)g * vectors + vec) * record + 2 * D + branch) - m_safe);
        const float inv = total > 0.f ? 1.0f / total : 0.f;
        for (int d = lane * 4; d < D; d += 128) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int g = 0; g < G; ++g) {
                const float *rec = recv + ((long long)g * vectors + vec) * record;
                const float w = expf(__ldg(rec + 2 * D + branch) - m_safe) * inv;
                const float4 o = __ldg(reinterpret_cast<const float4 *>(rec + branch * D + d));
                acc.x = fmaf(w, o.x, acc.x); acc.y = fmaf(w, o.y, acc.y); acc.z = fmaf(w, o.z, acc.z); acc.w = fmaf(w, o.w, acc.w);
            }
            if (branch == 0) {
                __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
                uint2 packed = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
                *reinterpret_cast<uint2 *>(sparse_out + vec * D + d) = packed;
            } else {
                *reinterpret_cast<float4 *>(linear_out + vec * D + d) = acc;
            }
        }
    }
}

static int check_view(const wa_tensor4 *t, const char *what, const char *name) {
    WA_REQUIRE(t && t->ptr, WA_ERR_ARG, "%s: %s is null", what, name);
    WA_REQUIRE(valid_dtype(t->dtype), WA_ERR_ARG, "%s: %s has bad dtype %d", what, name, t->dtype);
    return 0;
}

}  // namespace wa

using namespace wa;

namespace wa {
int block_sparse_run(const wa_tensor4 *q, const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *out, int B, int H, int Lq, int Lkv, int D,
                     int block_size, const int32_t *index, const int32_t *num, int index_stride, const int32_t *block_sizes, int round_inputs_bf16,
                     int round_output_bf16, float *lse, const int32_t *order, bool ahead, cudaStream_t stream) {
    const char *what = "wa_block_sparse_forward";
    int rc;
    if ((rc = check_view(q, what, "q")) || (rc = check_view(k, what, "k")) || (rc = check_view(v, what, "v")) ||
        (rc = check_view(out, what, "out")))
        return rc;
    WA_REQUIRE(index && num, WA_ERR_ARG, "%s: index / num is null", what);
    WA_REQUIRE(B > 0 && H > 0 && Lq > 0 && Lkv > 0 && D > 0 && block_size > 0 && index_stride > 0, WA_ERR_ARG,
               "%s: sizes must be positive", what);
    GenericAttnParams p{};
    p.q = make_view(q); p.k = make_view(k); p.v = make_view(v);
    p.out = out->ptr; p.out_dtype = out->dtype; p.osb = out->stride_b; p.osl = out->stride_l; p.osh = out->stride_h;
    p.H = H; p.Lq = Lq; p.Lkv = Lkv; p.D = D;
    p.q_block = block_size; p.kv_block = block_size; p.n_kv_blocks = ceil_div(Lkv, block_size);
    p.dense = 0; p.index = index; p.num = num; p.index_stride = index_stride; p.block_sizes = block_sizes;
    p.round_in = round_inputs_bf16; p.round_out = round_output_bf16;
    p.scale = (float)(1.0 / sqrt((double)D));
    p.lse = lse;
    p.order = order; p.ahead = ahead;
    return launch_generic_attention(p, B, ceil_div(Lq, block_size), stream, what);
}

int linear_run(const wa_tensor4 *q, const wa_tensor4 *k_coarse, const wa_tensor4 *v_coarse, const wa_tensor4 *out, int B, int H, int Lq, int Lc,
               int D, int round_output_bf16, float *lse, bool beside, cudaStream_t stream) {
    const char *what = "wa_linear_branch";
    int rc;
    if ((rc = check_view(q, what, "q")) || (rc = check_view(k_coarse, what, "k_coarse")) ||
        (rc = check_view(v_coarse, what, "v_coarse")) || (rc = check_view(out, what, "out")))
        return rc;
    WA_REQUIRE(B > 0 && H > 0 && Lq > 0 && Lc > 0 && D > 0, WA_ERR_ARG, "%s: sizes must be positive", what);
    GenericAttnParams p{};
    p.q = make_view(q); p.k = make_view(k_coarse); p.v = make_view(v_coarse);
    p.out = out->ptr; p.out_dtype = out->dtype; p.osb = out->stride_b; p.osl = out->stride_l; p.osh = out->stride_h;
    p.H = H; p.Lq = Lq; p.Lkv = Lc; p.D = D;
    p.q_block = GA_QT; p.kv_block = GA_TK; p.n_kv_blocks = ceil_div(Lc, GA_TK);
    p.dense = 1; p.index = nullptr; p.num = nullptr; p.index_stride = 1; p.block_sizes = nullptr;
    p.round_in = 0; p.round_out = round_output_bf16;
    p.scale = (float)pow((double)D, -0.5);
    p.lse = lse;
    p.beside = beside;
    return launch_generic_attention(p, B, ceil_div(Lq, GA_QT), stream, what);
}
}  // namespace wa

extern "C" int wa_block_sparse_forward(const wa_tensor4 *q, const wa_tensor4 *k, const wa_tensor4 *v,
                                       const wa_tensor4 *out, int B, int H, int Lq, int Lkv, int D,
                                       int block_size, const int32_t *index, const int32_t *num,
                                       int index_stride, const int32_t *block_sizes, int round_inputs_bf16,
                                       int round_output_bf16, float *lse, void *stream) {
    return block_sparse_run(q, k, v, out, B, H, Lq, Lkv, D, block_size, index, num, index_stride, block_sizes, round_inputs_bf16,
                            round_output_bf16, lse, nullptr, false, (cudaStream_t)stream);
}

extern "C" int wa_linear_branch(const wa_tensor4 *q, const wa_tensor4 *k_coarse, const wa_tensor4 *v_coarse,
                                const wa_tensor4 *out, int B, int H, int Lq, int Lc, int D,
                                int round_output_bf16, float *lse, void *stream) {
    return linear_run(q, k_coarse, v_coarse, out, B, H, Lq, Lc, D, round_output_bf16, lse, false, (cudaStream_t)stream);
}

extern "C" int wa_gate_combine(const wa_tensor4 *q, const wa_tensor4 *sparse, const wa_tensor4 *linear,
                               const wa_tensor4 *out, int B, int L, int H, int D, const void *gate_w,
                               const void *gate_b, int gate_dtype, int round_gate_bf16, void *stream) {
    const char *what = "wa_gate_combine";
    int rc;
    if ((rc = check_view(q, what, "q")) || (rc = check_view(sparse, what, "sparse")) ||
        (rc = check_view(linear, what, "linear")) || (rc = check_view(out, what, "out")))
        return rc;
    WA_REQUIRE(B > 0 && L > 0 && H > 0 && D > 0, WA_ERR_ARG, "%s: sizes must be positive", what);
    WA_REQUIRE(!gate_w || valid_dtype(gate_dtype), WA_ERR_ARG, "%s: bad gate dtype", what);
    const long long n_vec = (long long)B * L * H;
    const long long blocks = (n_vec + GC_WARPS - 1) / GC_WARPS;
    WA_REQUIRE(blocks < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many tokens", what);
    if (gate_w && D <= GS_MAXD) {
        static PerDeviceOnce attr_set;
        if (gs_smem(D) > 48 * 1024 && !attr_set.done()) {
            cudaError_t e = cudaFuncSetAttribute(gate_combine_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gs_smem(GS_MAXD));
            if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
            attr_set.mark();
        }
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const long long want = (n_vec + GS_WARPS * GS_VECS - 1) / (GS_WARPS * GS_VECS);
        const unsigned grid = (unsigned)(want < 2ll * sms ? want : 2ll * sms);
        gate_combine_smem_kernel<<<grid, GS_WARPS * 32, gs_smem(D), (cudaStream_t)stream>>>(
            make_view(q), make_view(sparse), make_view(linear), out->ptr, out->dtype, out->stride_b, out->stride_l,
            out->stride_h, n_vec, L, H, D, gs_ld(D), gate_w, gate_b, gate_dtype, round_gate_bf16);
        return check_launch(what);
    }
    const size_t smem = (size_t)GC_WARPS * D * sizeof(float);
    WA_REQUIRE(smem <= 48 * 1024, WA_ERR_UNSUPPORTED, "%s: head_dim %d too large", what, D);
    gate_combine_kernel<<<(unsigned)blocks, GC_WARPS * 32, smem, (cudaStream_t)stream>>>(
        make_view(q), make_view(sparse), make_view(linear), out->ptr, out->dtype, out->stride_b, out->stride_l,
        out->stride_h, n_vec, L, H, D, gate_w, gate_b, gate_dtype, round_gate_bf16);
    return check_launch(what);
}

extern "C" int wa_merge_partials(const float *outs, const float *lses, int G, int64_t rows, int D, float *out,
                                 float *lse, void *stream) {
    WA_REQUIRE(outs && lses && out, WA_ERR_ARG, "wa_merge_partials: null pointer");
    WA_REQUIRE(G > 0 && rows > 0 && D > 0, WA_ERR_ARG, "wa_merge_partials: sizes must be positive");
    const int warps = 8;
    const long long blocks = (rows + warps - 1) / warps;
    WA_REQUIRE(blocks < (1ll << 31), WA_ERR_UNSUPPORTED, "wa_merge_partials: too many rows");
    merge_partials_kernel<<<(unsigned)blocks, warps * 32, 0, (cudaStream_t)stream>>>(outs, lses, G, rows, D, out,
                                                                                     lse);
    return check_launch("wa_merge_partials");
}

extern "C" int wa_merge_packed(const float *recv, int G, int64_t vectors, int D, int record, void *sparse_out, float *linear_out,
                               void *stream) {
    const char *what = "wa_merge_packed";
    WA_REQUIRE(recv && sparse_out && linear_out, WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(G > 0 && vectors > 0 && D > 0, WA_ERR_ARG, "%s: sizes must be positive", what);
    WA_REQUIRE(D % 4 == 0 && record % 4 == 0 && record >= 2 * D + 2, WA_ERR_ARG,
               "%s: D and the record length must be multiples of 4 and a record must hold two vectors and two normalisers", what);
    WA_REQUIRE(((uintptr_t)recv | (uintptr_t)linear_out) % 16 == 0 && (uintptr_t)sparse_out % 8 == 0, WA_ERR_ALIGN,
               "%s: buffers must be 16-byte aligned", what);
    const int warps = 8;
    const long long blocks = (vectors + warps - 1) / warps;
    WA_REQUIRE(blocks < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many vectors", what);
    merge_packed_kernel<<<(unsigned)blocks, warps * 32, 0, (cudaStream_t)stream>>>(recv, G, vectors, D, record,
                                                                                   (__nv_bfloat16 *)sparse_out, linear_out);
    return check_launch(what);
}
