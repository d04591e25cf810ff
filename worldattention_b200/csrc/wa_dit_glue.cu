// The element-wise steps around the attention layer in a DiT block, one pass each (bf16 rows).
//
// WanAttentionBlock.forward (wan/modules/causal_model.py:586-659) wraps its three sub-layers in
//     norm(x).unflatten(frames, tokens) * (1 + e_scale) + e_shift          and          x + y.unflatten(...) * e_gate
// where WanLayerNorm (wan/modules/model.py:89-103) computes in float32 and casts back.  Written with tensor
// expressions that is about twelve passes over the activations per sub-layer (casts, broadcasts, temporaries); here it is
// one read and one write.  The reference's rounding points are kept: the normalised value is rounded to bf16, so are
// 1 + e_scale, the product and the sum, and y * e_gate before the residual addition.
#include <type_traits>

#include "wa_common.cuh"

namespace wa {

constexpr int GLUE_WARPS = 8;
constexpr int GLUE_MAX_VEC = 16;   // 16-byte vectors per lane: rows of up to 32 * 16 * 8 = 4096 bf16

__device__ __forceinline__ __nv_bfloat162 as_pair(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162 *>(&w); }
__device__ __forceinline__ uint32_t as_word(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ float low(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float high(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// A row of C bf16 by one warp, NV vectors of eight per lane, all of them in flight at once: the smallest NV that holds the row
// is taken, since the registers of the widest row cost the narrower ones their warps.  4680 rows of 1536: norm and modulation
// 16.2 -> 7.9 us (3.6 TB/s), residual 7.3 -> 7.2 (6.0 TB/s).
//
// The bf16x2 instructions used below round the exact product or sum once.  The product of two bf16 is exact in float32, and so is a
// sum whose terms lie within 16 binary orders (beyond that it rounds to the larger term either way), so they give the bits of
// the float32 operation followed by a rounding to bf16, at a third of the instructions.

// out = bf16(bf16(bf16(LN(x) [* w + b]) * bf16(1 + scale[f])) + shift[f]); scale / shift are per (batch, frame) vectors
// `[.., C]` with a row stride of `mod_stride` elements, or null.
template <int NV>
__global__ void __launch_bounds__(GLUE_WARPS * 32, NV > 8 ? 1 : (NV > 6 ? 3 : 4))
ln_modulate_kernel(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ out, long long rows, int C, float eps,
                   const __nv_bfloat16 *__restrict__ weight, const __nv_bfloat16 *__restrict__ bias,
                   const __nv_bfloat16 *__restrict__ scale, const __nv_bfloat16 *__restrict__ shift, long long mod_stride,
                   int tokens_per_frame) {
    pdl_wait();
    const long long row = (long long)blockIdx.x * GLUE_WARPS + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31, nvec = C >> 3;
    const uint4 *src = reinterpret_cast<const uint4 *>(x + row * C);
    uint4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = i * 32 + lane < nvec ? src[i * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) sum += low(w[e]), sum += high(w[e]);
    }
    sum = warp_sum(sum);
    const float mean = sum / (float)C;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        if (i * 32 + lane < nvec) {
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float a = low(w[e]) - mean, b = high(w[e]) - mean;
                sq += a * a;
                sq += b * b;
            }
        }
    }
    sq = warp_sum(sq);
    const float rstd = rsqrtf(sq / (float)C + eps);
    const long long frame = row / tokens_per_frame;
    const uint4 *wv = reinterpret_cast<const uint4 *>(weight), *bv = reinterpret_cast<const uint4 *>(bias);
    const uint4 *sc = scale ? reinterpret_cast<const uint4 *>(scale + frame * mod_stride) : nullptr;
    const uint4 *sh = shift ? reinterpret_cast<const uint4 *>(shift + frame * mod_stride) : nullptr;
    uint4 *dst = reinterpret_cast<uint4 *>(out + row * C);
    const __nv_bfloat162 one = __floats2bfloat162_rn(1.f, 1.f);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int j = i * 32 + lane;
        if (j < nvec) {
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            float f[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                f[2 * e] = (low(w[e]) - mean) * rstd;
                f[2 * e + 1] = (high(w[e]) - mean) * rstd;
            }
            if (wv) {
                const uint4 t = __ldg(wv + j);
                const uint32_t a[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) f[2 * e] *= low(a[e]), f[2 * e + 1] *= high(a[e]);
            }
            if (bv) {
                const uint4 t = __ldg(bv + j);
                const uint32_t a[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) f[2 * e] += low(a[e]), f[2 * e + 1] += high(a[e]);
            }
            __nv_bfloat162 r[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) r[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
            if (sc) {
                const uint4 t = __ldg(sc + j);
                const uint32_t a[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) r[e] = __hmul2_rn(r[e], __hadd2_rn(one, as_pair(a[e])));
            }
            if (sh) {
                const uint4 t = __ldg(sh + j);
                const uint32_t a[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) r[e] = __hadd2_rn(r[e], as_pair(a[e]));
            }
            dst[j] = make_uint4(as_word(r[0]), as_word(r[1]), as_word(r[2]), as_word(r[3]));
        }
    }
}

// out = bf16(x + bf16(y * gate[f])) (gate null: out = bf16(x + y)).  One warp per row.
template <int NV>
__global__ void __launch_bounds__(GLUE_WARPS * 32, NV > 6 ? 3 : 4)
gated_residual_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ y, __nv_bfloat16 *__restrict__ out,
                      long long rows, int C, const __nv_bfloat16 *__restrict__ gate, long long mod_stride, int tokens_per_frame) {
    pdl_wait();
    const long long row = (long long)blockIdx.x * GLUE_WARPS + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31, nvec = C >> 3;
    const uint4 *xv = reinterpret_cast<const uint4 *>(x + row * C), *yv = reinterpret_cast<const uint4 *>(y + row * C);
    const uint4 *gv = gate ? reinterpret_cast<const uint4 *>(gate + row / tokens_per_frame * mod_stride) : nullptr;
    uint4 *dst = reinterpret_cast<uint4 *>(out + row * C);
    for (int j0 = lane; j0 < nvec; j0 += 32 * NV) {
        uint4 a[NV], b[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (j0 + 32 * i < nvec) {
                a[i] = xv[j0 + 32 * i];
                b[i] = yv[j0 + 32 * i];
            }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int j = j0 + 32 * i;
            if (j < nvec) {
                const uint32_t xw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, yw[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
                uint32_t o[4];
                if (gv) {
                    const uint4 t = __ldg(gv + j);
                    const uint32_t g[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[e] = as_word(__hadd2_rn(as_pair(xw[e]), __hmul2_rn(as_pair(yw[e]), as_pair(g[e]))));
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[e] = as_word(__hadd2_rn(as_pair(xw[e]), as_pair(yw[e])));
                }
                dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

// calls f with the smallest of the kernels' widths that holds rows of C elements (the widest for longer ones)
template <typename F>
static void with_width(int C, const F &f) {
    const int vectors = (C / 8 + 31) / 32;
    if (vectors <= 2) f(std::integral_constant<int, 2>());
    else if (vectors <= 4) f(std::integral_constant<int, 4>());
    else if (vectors <= 6) f(std::integral_constant<int, 6>());
    else if (vectors <= 8) f(std::integral_constant<int, 8>());
    else f(std::integral_constant<int, GLUE_MAX_VEC>());
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace wa

using namespace wa;

extern "C" int wa_ln_modulate(const void *x, void *out, long long rows, int C, float eps, const void *weight, const void *bias,
                              const void *scale, const void *shift, long long mod_stride, int tokens_per_frame, void *stream) {
    const char *what = "wa_ln_modulate";
    WA_REQUIRE(x && out, WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(rows >= 0 && C > 0 && tokens_per_frame > 0, WA_ERR_ARG, "%s: sizes must be positive", what);
    WA_REQUIRE(C % 8 == 0 && C <= 32 * GLUE_MAX_VEC * 8, WA_ERR_UNSUPPORTED, "%s: row length must be a multiple of 8 and at most %d, got %d",
               what, 32 * GLUE_MAX_VEC * 8, C);
    WA_REQUIRE(aligned16(x) && aligned16(out) && aligned16(weight) && aligned16(bias) && aligned16(scale) && aligned16(shift) &&
                   mod_stride % 8 == 0,
               WA_ERR_ALIGN, "%s: pointers must be 16-byte aligned and the modulation stride a multiple of 8 elements", what);
    if (rows == 0) return 0;
    const long long ctas = (rows + GLUE_WARPS - 1) / GLUE_WARPS;
    WA_REQUIRE(ctas < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many rows", what);
    cudaError_t le = cudaSuccess;
    with_width(C, [&](auto nv) {
        le = launch_dependent(ln_modulate_kernel<decltype(nv)::value>, dim3((unsigned)ctas), dim3(GLUE_WARPS * 32), 0, (cudaStream_t)stream,
            (const __nv_bfloat16 *)x, (__nv_bfloat16 *)out, rows, C, eps, (const __nv_bfloat16 *)weight, (const __nv_bfloat16 *)bias,
            (const __nv_bfloat16 *)scale, (const __nv_bfloat16 *)shift, mod_stride, tokens_per_frame);
    });
    if (le != cudaSuccess) return fail((int)le, "%s: %s", what, cudaGetErrorString(le));
    return check_launch(what);
}

extern "C" int wa_gated_residual(const void *x, const void *y, void *out, long long rows, int C, const void *gate,
                                 long long mod_stride, int tokens_per_frame, void *stream) {
    const char *what = "wa_gated_residual";
    WA_REQUIRE(x && y && out, WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(rows >= 0 && C > 0 && tokens_per_frame > 0, WA_ERR_ARG, "%s: sizes must be positive", what);
    WA_REQUIRE(C % 8 == 0, WA_ERR_UNSUPPORTED, "%s: row length must be a multiple of 8, got %d", what, C);
    WA_REQUIRE(aligned16(x) && aligned16(y) && aligned16(out) && aligned16(gate) && mod_stride % 8 == 0, WA_ERR_ALIGN,
               "%s: pointers must be 16-byte aligned and the modulation stride a multiple of 8 elements", what);
    if (rows == 0) return 0;
    const long long ctas = (rows + GLUE_WARPS - 1) / GLUE_WARPS;
    WA_REQUIRE(ctas < (1ll << 31), WA_ERR_UNSUPPORTED, "%s: too many rows", what);
    cudaError_t le = cudaSuccess;
    with_width(C, [&](auto nv) {
        constexpr int NV = decltype(nv)::value < 8 ? decltype(nv)::value : 8;
        le = launch_dependent(gated_residual_kernel<NV>, dim3((unsigned)ctas), dim3(GLUE_WARPS * 32), 0, (cudaStream_t)stream,
            (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)y, (__nv_bfloat16 *)out, rows, C, (const __nv_bfloat16 *)gate, mod_stride,
            tokens_per_frame);
    });
    if (le != cudaSuccess) return fail((int)le, "%s: %s", what, cudaGetErrorString(le));
    return check_launch(what);
}
