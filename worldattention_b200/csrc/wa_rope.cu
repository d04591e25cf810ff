// q/k RMSNorm + causal rotary embedding in one pass over the projected tokens.
//
// Stands in for WanRMSNorm (wan/modules/model.py:70-86) followed by causal_rope_apply
// (wan/modules/causal_model.py:34-62), which the reference runs as separate tensor operations with a Python
// loop over samples and a float64 complex copy of q and of k.  Bandwidth-bound: one warp per token reads the
// H*D values (twice; the second read hits L1/L2), writes them once.  Rounding points follow the reference:
// the normalised value and its product with the weight are each stored in the input dtype, the rotation is a
// float64 complex product stored once in the input dtype.
#include <type_traits>

#include "wa_common.cuh"

namespace wa {

constexpr int RN_WARPS = 8;

template <typename T> __device__ __forceinline__ float2 load_pair(const T *p);
template <> __device__ __forceinline__ float2 load_pair<float>(const float *p) { return *reinterpret_cast<const float2 *>(p); }
template <> __device__ __forceinline__ float2 load_pair<__nv_bfloat16>(const __nv_bfloat16 *p) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p));
}
template <typename T> __device__ __forceinline__ float round_to(float x);
template <> __device__ __forceinline__ float round_to<float>(float x) { return x; }
template <> __device__ __forceinline__ float round_to<__nv_bfloat16>(float x) { return bf16_round_f(x); }
template <typename T> __device__ __forceinline__ void store_pair(T *p, double re, double im);
template <> __device__ __forceinline__ void store_pair<float>(float *p, double re, double im) {
    *reinterpret_cast<float2 *>(p) = make_float2((float)re, (float)im);
}
template <> __device__ __forceinline__ void store_pair<__nv_bfloat16>(__nv_bfloat16 *p, double re, double im) {
    __nv_bfloat162 v;
    v.x = __double2bfloat16(re);
    v.y = __double2bfloat16(im);
    *reinterpret_cast<__nv_bfloat162 *>(p) = v;
}

template <typename T>
__global__ void __launch_bounds__(RN_WARPS * 32)
qk_norm_rope_kernel(const T *__restrict__ x, long long xsb, long long xsl, long long xsh, T *__restrict__ out, long long osb,
                    long long osl, long long osh, long long tokens, int L, int H, int D, const void *__restrict__ weight, int wdt,
                    float eps, const double2 *__restrict__ freqs, int freq_rows, int start_frame, const int *__restrict__ start_frame_dev,
                    int grid_h, int grid_w) {
    if (start_frame_dev) start_frame = max(*start_frame_dev, 0);   // the position lives on the device (replayed launches)
    const long long tok = (long long)blockIdx.x * RN_WARPS + (threadIdx.x >> 5);
    if (tok >= tokens) return;
    const int lane = threadIdx.x & 31;
    const int b = (int)(tok / L), t = (int)(tok % L);
    const T *src = x + (long long)b * xsb + (long long)t * xsl;
    T *dst = out + (long long)b * osb + (long long)t * osl;
    const int c = D >> 1, pairs = H * c;

    float scale = 1.0f;
    if (weight) {
        double acc = 0.0;
        for (int p = lane; p < pairs; p += 32) {
            const float2 v = load_pair<T>(src + (long long)(p / c) * xsh + 2 * (p % c));
            acc += (double)v.x * (double)v.x + (double)v.y * (double)v.y;
        }
        acc = warp_sum_d(acc);
        const float mean_sq = (float)(acc / (double)(H * D));
        scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, eps)));
    }
    // position of the token in the (frame, row, column) grid; the three bands of a head's pairs take one each
    const int per_frame = grid_h * grid_w;
    const int frame = min(max(start_frame + t / per_frame, 0), freq_rows - 1);
    const int row = min((t / grid_w) % grid_h, freq_rows - 1), col = min(t % grid_w, freq_rows - 1);
    const int ct = c - 2 * (c / 3), ch = c / 3;
    for (int p = lane; p < pairs; p += 32) {
        const int h = p / c, j = p % c;
        float2 v = load_pair<T>(src + (long long)h * xsh + 2 * j);
        if (weight) {
            const float w0 = load_elem(weight, wdt, (long long)h * D + 2 * j), w1 = load_elem(weight, wdt, (long long)h * D + 2 * j + 1);
            v.x = round_to<T>(__fmul_rn(round_to<T>(__fmul_rn(v.x, scale)), w0));
            v.y = round_to<T>(__fmul_rn(round_to<T>(__fmul_rn(v.y, scale)), w1));
        }
        double re = (double)v.x, im = (double)v.y;
        if (freqs) {
            const int pos = j < ct ? frame : (j < ct + ch ? row : col);
            const double2 f = freqs[(long long)pos * c + j];
            const double a = re, bb = im;
            re = a * f.x - bb * f.y;
            im = a * f.y + bb * f.x;
        }
        store_pair<T>(dst + (long long)h * osh + 2 * j, re, im);
    }
}

// bf16 tokens whose heads lie side by side (stride D): the token's H*D values are read ONCE as 16-byte vectors and
// kept in registers (up to 8 vectors per lane: H*D <= 2048).  Same arithmetic per value as the kernel above.
constexpr int RN_MAX_VEC = 8;

__global__ void __launch_bounds__(RN_WARPS * 32)
qk_norm_rope_rows_kernel(const __nv_bfloat16 *__restrict__ x, long long xsb, long long xsl, __nv_bfloat16 *__restrict__ out,
                         long long osb, long long osl, long long tokens, int L, int H, int D, const void *__restrict__ weight, int wdt,
                         float eps, const double2 *__restrict__ freqs, int freq_rows, int start_frame,
                         const int *__restrict__ start_frame_dev, int grid_h, int grid_w) {
    if (start_frame_dev) start_frame = max(*start_frame_dev, 0);
    const long long tok = (long long)blockIdx.x * RN_WARPS + (threadIdx.x >> 5);
    if (tok >= tokens) return;
    const int lane = threadIdx.x & 31;
    const int b = (int)(tok / L), t = (int)(tok % L);
    const uint4 *src = reinterpret_cast<const uint4 *>(x + (long long)b * xsb + (long long)t * xsl);
    uint4 *dst = reinterpret_cast<uint4 *>(out + (long long)b * osb + (long long)t * osl);
    const int nvec = (H * D) >> 3, c = D >> 1;

    uint4 v[RN_MAX_VEC];
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < RN_MAX_VEC; ++i) {
        const int j = i * 32 + lane;
        if (j < nvec) {
            v[i] = src[j];
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double lo = (double)__uint_as_float(w[e] << 16), hi = (double)__uint_as_float(w[e] & 0xffff0000u);
                acc += lo * lo + hi * hi;
            }
        }
    }
    float scale = 1.0f;
    if (weight) {
        acc = warp_sum_d(acc);
        const float mean_sq = (float)(acc / (double)(H * D));
        scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, eps)));
    }
    const int per_frame = grid_h * grid_w;
    const int frame = min(max(start_frame + t / per_frame, 0), freq_rows - 1);
    const int row = min((t / grid_w) % grid_h, freq_rows - 1), col = min(t % grid_w, freq_rows - 1);
    const int ct = c - 2 * (c / 3), ch = c / 3;
#pragma unroll
    for (int i = 0; i < RN_MAX_VEC; ++i) {
        const int j = i * 32 + lane;
        if (j < nvec) {
            const int elem = j << 3, h = elem / D, pair0 = (elem - h * D) >> 1;      // four pairs of one head
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int jp = pair0 + e;
                float vx = __uint_as_float(w[e] << 16), vy = __uint_as_float(w[e] & 0xffff0000u);
                if (weight) {
                    const float w0 = load_elem(weight, wdt, (long long)h * D + 2 * jp), w1 = load_elem(weight, wdt, (long long)h * D + 2 * jp + 1);
                    vx = bf16_round_f(__fmul_rn(bf16_round_f(__fmul_rn(vx, scale)), w0));
                    vy = bf16_round_f(__fmul_rn(bf16_round_f(__fmul_rn(vy, scale)), w1));
                }
                double re = (double)vx, im = (double)vy;
                if (freqs) {
                    const int pos = jp < ct ? frame : (jp < ct + ch ? row : col);
                    const double2 f = freqs[(long long)pos * c + jp];
                    const double a = re, bb = im;
                    re = a * f.x - bb * f.y;
                    im = a * f.y + bb * f.x;
                }
                __nv_bfloat162 r;
                r.x = __double2bfloat16(re);
                r.y = __double2bfloat16(im);
                o[e] = *reinterpret_cast<const uint32_t *>(&r);
            }
            dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// The same where a lane's vectors lie at the same pairs of every head they belong to (D a power of two up to 256), with bf16
// weights or none.  The general kernel is bound by its instructions, not by memory: a float64 conversion is a quarter of a
// product's rate, and each value has four of them.  Here
//   * the squares are summed in float64 as before, but a bf16 magnitude becomes a float64 by shifting its bits (exponents rebiased;
//     a zero or subnormal comes out as about 2^-127, an infinity or NaN as 2^128 or more, so a sum outside [2^-190, 2^250] is
//     taken again with true conversions);
//   * the product with the weight is one bf16x2 instruction (the exact product rounded once);
//   * the rotation is computed in float32 with the bound 2^-22 (|r| + |p|) on its distance from the float64 one (r the result, p
//     the product subtracted or added; the factors', the product's and the sum's roundings are 2^-24 of these each): where both
//     ends of that interval round to the same bf16, that is the result; the other pairs (about one in 3000), those near zero and
//     those with a factor below float32's normal range (whose rounding the bound does not cover) are rotated in float64 as in the
//     kernel above.  The results are therefore the same bits;
//   * four CTAs per SM: the 4680 tokens of a chunk are resident at once.
// 12 heads of 128, 4680 tokens: 18.3 us with the general form, 10.1 here (2.8 TB/s; a chunk of q and k prepared and appended: 54.5 -> 39.0).
template <int NV, bool WEIGHT, bool ROTATE>
__global__ void __launch_bounds__(RN_WARPS * 32, NV > 6 ? 3 : 4)
qk_norm_rope_bits_kernel(const __nv_bfloat16 *__restrict__ x, long long xsb, long long xsl, __nv_bfloat16 *__restrict__ out,
                         long long osb, long long osl, long long tokens, int L, int H, int D, const __nv_bfloat16 *__restrict__ weight,
                         float eps, const double2 *__restrict__ freqs, int freq_rows, int start_frame,
                         const int *__restrict__ start_frame_dev, int grid_h, int grid_w) {
    pdl_wait();
    const long long tok = (long long)blockIdx.x * RN_WARPS + (threadIdx.x >> 5);
    if (tok >= tokens) return;
    const int lane = threadIdx.x & 31;
    const int b = (int)(tok / L), t = (int)(tok - (long long)b * L);
    const uint4 *src = reinterpret_cast<const uint4 *>(x + (long long)b * xsb + (long long)t * xsl);
    uint4 *dst = reinterpret_cast<uint4 *>(out + (long long)b * osb + (long long)t * osl);
    const int nvec = (H * D) >> 3, c = D >> 1;

    uint4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = i * 32 + lane < nvec ? src[i * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);

    const int pair0 = ((lane << 3) & (D - 1)) >> 1;      // first of the lane's four pairs, in the head of each of its vectors
    const double2 *factors[3];                           // table rows of the three bands, at this lane's pairs
    const int ct = c - 2 * (c / 3), ch = c / 3;
    float fx[4], fy[4];
    uint32_t smallest = 0xffffffffu;                     // exponent of the smallest factor that is not zero
    if constexpr (ROTATE) {
        if (start_frame_dev) start_frame = max(*start_frame_dev, 0);
        const int line = t / grid_w, fr = line / grid_h;
        const int frame = min(max(start_frame + fr, 0), freq_rows - 1);
        const int row = min(line - fr * grid_h, freq_rows - 1), col = min(t - line * grid_w, freq_rows - 1);
        factors[0] = freqs + (long long)frame * c + pair0;
        factors[1] = freqs + (long long)row * c + pair0;
        factors[2] = freqs + (long long)col * c + pair0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int jp = pair0 + e;
            const double2 f = __ldg((jp < ct ? factors[0] : (jp < ct + ch ? factors[1] : factors[2])) + e);
            fx[e] = (float)f.x;
            fy[e] = (float)f.y;
            smallest = min(smallest, min(2u * (uint32_t)__double2hiint(f.x) - 1u, 2u * (uint32_t)__double2hiint(f.y) - 1u));
        }
    }

    float scale = 1.0f;
    if constexpr (WEIGHT) {
        double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const double lo = __hiloint2double((int)(((w[e] << 13) & 0x0fffe000u) + 0x38000000u), 0);
                const double hi = __hiloint2double((int)(((w[e] >> 3) & 0x0fffe000u) + 0x38000000u), 0);
                part[e] = fma(lo, lo, part[e]);
                part[e] = fma(hi, hi, part[e]);
            }
        }
        double acc = warp_sum_d((part[0] + part[1]) + (part[2] + part[3]));
        if (!(acc > 0x1p-190 && acc < 0x1p250)) {
            acc = 0.0;
#pragma unroll 1
            for (int j = lane; j < nvec; j += 32) {
                const uint4 again = src[j];
                const uint32_t w[4] = {again.x, again.y, again.z, again.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const double lo = (double)__uint_as_float(w[e] << 16), hi = (double)__uint_as_float(w[e] & 0xffff0000u);
                    acc += lo * lo + hi * hi;
                }
            }
            acc = warp_sum_d(acc);
        }
        const float mean_sq = (float)(acc / (double)(H * D));
        scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, eps)));
    }

    // one pair of values after norm and weight, packed
    auto normed = [&](uint32_t w, uint32_t wt) {
        if constexpr (!WEIGHT) return w;
        const __nv_bfloat162 r = __floats2bfloat162_rn(__fmul_rn(__uint_as_float(w << 16), scale), __fmul_rn(__uint_as_float(w & 0xffff0000u), scale));
        const __nv_bfloat162 p = __hmul2_rn(r, *reinterpret_cast<const __nv_bfloat162 *>(&wt));
        return *reinterpret_cast<const uint32_t *>(&p);
    };
    const uint4 *wv = reinterpret_cast<const uint4 *>(weight);
    uint32_t open = 0u;                                   // pairs whose bf16 the float32 rotation does not settle
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int j = i * 32 + lane;
        if (j < nvec) {
            uint4 wt = make_uint4(0u, 0u, 0u, 0u);
            if constexpr (WEIGHT) wt = __ldg(wv + j);
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w}, ww[4] = {wt.x, wt.y, wt.z, wt.w};
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[e] = normed(w[e], ww[e]);
                if constexpr (ROTATE) {
                    const float a = __uint_as_float(o[e] << 16), bb = __uint_as_float(o[e] & 0xffff0000u);
                    const float p = __fmul_rn(bb, fy[e]), q = __fmul_rn(bb, fx[e]);
                    const float re = __fmaf_rn(a, fx[e], -p), im = __fmaf_rn(a, fy[e], q);
                    const float tr = fabsf(re) + fabsf(p), ti = fabsf(im) + fabsf(q);
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(__fmaf_rn(tr, -0x1p-22f, re), __fmaf_rn(ti, -0x1p-22f, im));
                    const __nv_bfloat162 hi = __floats2bfloat162_rn(__fmaf_rn(tr, 0x1p-22f, re), __fmaf_rn(ti, 0x1p-22f, im));
                    o[e] = *reinterpret_cast<const uint32_t *>(&lo);
                    if (o[e] != *reinterpret_cast<const uint32_t *>(&hi) || !(tr > 0x1p-100f) || !(ti > 0x1p-100f)) open |= 1u << (i * 4 + e);
                }
            }
            dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
    if constexpr (ROTATE) {
        if (smallest < 2u * 0x38100000u - 1u) {          // a factor below 2^-126
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (i * 32 + lane < nvec) open |= 15u << (4 * i);
        }
#pragma unroll 1
        while (open) {
            const int k = __ffs((int)open) - 1;
            open &= open - 1u;
            uint32_t w = 0u;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                if (k == 4 * i) w = v[i].x;
                if (k == 4 * i + 1) w = v[i].y;
                if (k == 4 * i + 2) w = v[i].z;
                if (k == 4 * i + 3) w = v[i].w;
            }
            const int j = (k >> 2) * 32 + lane, e = k & 3, jp = pair0 + e;
            const uint32_t n = normed(w, WEIGHT ? __ldg(reinterpret_cast<const uint32_t *>(weight) + j * 4 + e) : 0u);
            const double2 f = __ldg((jp < ct ? factors[0] : (jp < ct + ch ? factors[1] : factors[2])) + e);
            const double a = (double)__uint_as_float(n << 16), bb = (double)__uint_as_float(n & 0xffff0000u);
            store_pair<__nv_bfloat16>(reinterpret_cast<__nv_bfloat16 *>(dst + j) + 2 * e, a * f.x - bb * f.y, a * f.y + bb * f.x);
        }
    }
}

}  // namespace wa

using namespace wa;

static int qk_norm_rope_launch(const wa_tensor4 *x, const wa_tensor4 *out, int B, int L, int H, int D, const void *norm_weight,
                               int weight_dtype, float eps, const double *freqs, int freq_rows, int start_frame,
                               const int *start_frame_dev, int grid_h, int grid_w, void *stream) {
    const char *what = "wa_qk_norm_rope";
    WA_REQUIRE(x && out && x->ptr && out->ptr, WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(valid_dtype(x->dtype) && x->dtype == out->dtype, WA_ERR_ARG, "%s: x and out must share a dtype", what);
    WA_REQUIRE(B > 0 && L > 0 && H > 0 && D > 0 && D % 2 == 0, WA_ERR_ARG, "%s: sizes must be positive and head_dim even", what);
    WA_REQUIRE(!norm_weight || valid_dtype(weight_dtype), WA_ERR_ARG, "%s: bad weight dtype", what);
    WA_REQUIRE(!freqs || (freq_rows > 0 && grid_h > 0 && grid_w > 0 && start_frame >= 0), WA_ERR_ARG,
               "%s: a rotation needs a table and a positive grid", what);
    const int align = x->dtype == WA_BF16 ? 4 : 8;
    WA_REQUIRE((uintptr_t)x->ptr % align == 0 && (uintptr_t)out->ptr % align == 0 && x->stride_h % 2 == 0 && x->stride_l % 2 == 0 &&
                   x->stride_b % 2 == 0 && out->stride_h % 2 == 0 && out->stride_l % 2 == 0 && out->stride_b % 2 == 0,
               WA_ERR_ALIGN, "%s: pairs must be naturally aligned (even strides)", what);
    const long long tokens = (long long)B * L;
    const long long blocks = (tokens + RN_WARPS - 1) / RN_WARPS;
    WA_REQUIRE(blocks < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many tokens", what);
    if (!freqs) grid_h = grid_w = 1;
    const bool rows_in_registers = x->dtype == WA_BF16 && x->stride_h == D && out->stride_h == D && D % 8 == 0 &&
                                   (long long)H * D <= 32 * RN_MAX_VEC * 8 && (uintptr_t)x->ptr % 16 == 0 && (uintptr_t)out->ptr % 16 == 0 &&
                                   x->stride_l % 8 == 0 && x->stride_b % 8 == 0 && out->stride_l % 8 == 0 && out->stride_b % 8 == 0;
    // D a power of two: the lanes' vectors lie alike in every head; float32 weights and a plain copy stay with the general form
    const bool by_bits = rows_in_registers && D <= 256 && (D & (D - 1)) == 0 && (norm_weight ? weight_dtype == WA_BF16 && (uintptr_t)norm_weight % 16 == 0 : freqs != nullptr);
    if (by_bits) {
        cudaError_t le = cudaSuccess;
        const auto launch = [&](auto kernel) {
            le = launch_dependent(kernel, dim3((unsigned)blocks), dim3(RN_WARPS * 32), 0, (cudaStream_t)stream,
                (const __nv_bfloat16 *)x->ptr, x->stride_b, x->stride_l, (__nv_bfloat16 *)out->ptr, out->stride_b, out->stride_l, tokens, L, H,
                D, (const __nv_bfloat16 *)norm_weight, eps, (const double2 *)freqs, freq_rows, start_frame, start_frame_dev, grid_h, grid_w);
        };
        const auto pick = [&](auto nv) {
            constexpr int NV = decltype(nv)::value;
            if (!norm_weight) launch(qk_norm_rope_bits_kernel<NV, false, true>);
            else if (freqs) launch(qk_norm_rope_bits_kernel<NV, true, true>);
            else launch(qk_norm_rope_bits_kernel<NV, true, false>);
        };
        const int vectors = (H * D / 8 + 31) / 32;
        if (vectors <= 4) pick(std::integral_constant<int, 4>());
        else if (vectors <= 6) pick(std::integral_constant<int, 6>());
        else pick(std::integral_constant<int, 8>());
        if (le != cudaSuccess) return fail((int)le, "%s: %s", what, cudaGetErrorString(le));
    } else if (rows_in_registers)
        qk_norm_rope_rows_kernel<<<(unsigned)blocks, RN_WARPS * 32, 0, (cudaStream_t)stream>>>(
            (const __nv_bfloat16 *)x->ptr, x->stride_b, x->stride_l, (__nv_bfloat16 *)out->ptr, out->stride_b, out->stride_l, tokens, L, H,
            D, norm_weight, weight_dtype, eps, (const double2 *)freqs, freq_rows, start_frame, start_frame_dev, grid_h, grid_w);
    else if (x->dtype == WA_BF16)
        qk_norm_rope_kernel<__nv_bfloat16><<<(unsigned)blocks, RN_WARPS * 32, 0, (cudaStream_t)stream>>>(
            (const __nv_bfloat16 *)x->ptr, x->stride_b, x->stride_l, x->stride_h, (__nv_bfloat16 *)out->ptr, out->stride_b,
            out->stride_l, out->stride_h, tokens, L, H, D, norm_weight, weight_dtype, eps, (const double2 *)freqs, freq_rows,
            start_frame, start_frame_dev, grid_h, grid_w);
    else
        qk_norm_rope_kernel<float><<<(unsigned)blocks, RN_WARPS * 32, 0, (cudaStream_t)stream>>>(
            (const float *)x->ptr, x->stride_b, x->stride_l, x->stride_h, (float *)out->ptr, out->stride_b, out->stride_l,
            out->stride_h, tokens, L, H, D, norm_weight, weight_dtype, eps, (const double2 *)freqs, freq_rows, start_frame,
            start_frame_dev, grid_h, grid_w);
    return check_launch(what);
}

extern "C" int wa_qk_norm_rope(const wa_tensor4 *x, const wa_tensor4 *out, int B, int L, int H, int D, const void *norm_weight,
                               int weight_dtype, float eps, const double *freqs, int freq_rows, int start_frame, int grid_h,
                               int grid_w, void *stream) {
    return qk_norm_rope_launch(x, out, B, L, H, D, norm_weight, weight_dtype, eps, freqs, freq_rows, start_frame, nullptr, grid_h,
                               grid_w, stream);
}

extern "C" int wa_qk_norm_rope_at(const wa_tensor4 *x, const wa_tensor4 *out, int B, int L, int H, int D, const void *norm_weight,
                                  int weight_dtype, float eps, const double *freqs, int freq_rows, const int32_t *start_frame_device,
                                  int grid_h, int grid_w, void *stream) {
    WA_REQUIRE(start_frame_device, WA_ERR_ARG, "wa_qk_norm_rope_at: null position pointer");
    return qk_norm_rope_launch(x, out, B, L, H, D, norm_weight, weight_dtype, eps, freqs, freq_rows, 0, start_frame_device, grid_h,
                               grid_w, stream);
}
