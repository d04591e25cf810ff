// Internal (non-ABI) declarations shared between translation units.
#pragma once
#include "wa_common.cuh"

namespace wa {

// Launch preparation of the tcgen05 kernel that can ride on another kernel: the heaviest-first work
// order over all (batch, head, query block) items, the reset of the work counter and failure flag,
// and the bf16 copy of the gate weight.  `order == nullptr` means "nothing to prepare".
struct SchedJob {
    int32_t *order;
    int *work_counter;
    int *error_flag;
    const void *gate_w, *gate_b;
    int gate_dt;
    __nv_bfloat16 *w_out;   // [128 x 128] bf16
    float *b_out;           // [128] float32
    bool paired;            // a work item is two neighbouring query blocks (rows of `num`) of one head: pair_lists_kernel makes the order
    bool by_head;           // paired: work order head by head (see sort_items_by_head)
    bool by_counts;         // paired: the routing makes the work order, by the larger count of a pair, not pair_lists_kernel by the tiles
    int *pairs_done;        // paired: CTAs of pair_lists_kernel that are done; zero before it runs
    bool release_at_start;  // the next launch does not wait for the routing (it compresses K and V meanwhile)
    int beside_sms;         // ... and takes up so many SMs, where that is known (0: it is not)
    bool one_part;          // ... and is done sooner beside one routing CTA per head than beside two (see route_short_parts)
    int release_dependents_after_rows;   // timing experiment (WA_B200_PDL=2), see route_row
};

constexpr int SCHED_BINS = 4096;
constexpr int SCHED_HEADS = 256;

// Counting sort of the items by weight, heaviest first.  The last CTA of the routing runs it alone and the attention waits:
// what is not needed for single rows (the pairs' look-ups, the order by heads) has code of its own, because instructions that
// are fetched for the first time cost as much here as the sort (with one code for all, 16.5 -> 18.7 us of routing on
// changing inputs).
template <typename Count>
__device__ __forceinline__ void sort_items(Count count_of, int n_items, int Nkv, int *hist, int *warp_tot, int32_t *__restrict__ order,
                                           int *work_counter, int *error_flag) {
    const int T = blockDim.x, tid = threadIdx.x;
    // bins 0..top hold counts top..0 (bin 0 = heaviest); `per` bins per thread, a power of two >= 1
    const int top = min(Nkv, SCHED_BINS - 1);
    int per = 1;
    while (per * T < top + 1) per <<= 1;
    for (int i = tid; i < per * T; i += T) hist[i] = 0;
    if (tid == 0) {
        *work_counter = 0;
        *error_flag = 0;
    }
    __syncthreads();
    // the counts are read only once when they fit in registers
    constexpr int KEEP = 4;
    int bin_of[KEEP];
#pragma unroll
    for (int u = 0; u < KEEP; ++u) {
        const int i = tid + u * T;
        bin_of[u] = i < n_items ? top - max(0, min(count_of(i), top)) : -1;
    }
#pragma unroll
    for (int u = 0; u < KEEP; ++u)
        if (bin_of[u] >= 0) atomicAdd(&hist[bin_of[u]], 1);
    for (int i = tid + KEEP * T; i < n_items; i += T) atomicAdd(&hist[top - max(0, min(count_of(i), top))], 1);
    __syncthreads();
    // exclusive prefix over the bins: a contiguous run of bins per thread, then a block scan of the run totals
    const int b0 = tid * per;
    int mine = 0;
    for (int i = 0; i < per; ++i) mine += hist[b0 + i];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += v;
    }
    if ((tid & 31) == 31) warp_tot[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32) {
        int w = tid < (T >> 5) ? warp_tot[tid] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, w, o);
            if (tid >= o) w += v;
        }
        warp_tot[tid] = w;
    }
    __syncthreads();
    int base = incl - mine + ((tid >> 5) ? warp_tot[(tid >> 5) - 1] : 0);
    for (int i = 0; i < per; ++i) {
        const int c = hist[b0 + i];
        hist[b0 + i] = base;
        base += c;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < KEEP; ++u)
        if (bin_of[u] >= 0) order[atomicAdd(&hist[bin_of[u]], 1)] = tid + u * T;
    for (int i = tid + KEEP * T; i < n_items; i += T) order[atomicAdd(&hist[top - max(0, min(count_of(i), top))], 1)] = i;
}

// Head by head, the head with the most work first and a head's items heaviest first, so that the CTAs at work at a time read
// the keys of a few heads (counts from the mass over a window of 21 frames: 797 against 716 us a call).  The last heads, as many as
// the CTAs work on at a time, are taken together, heaviest item first: the keys are no more than before, and the items that come last
// are then the lightest of all these and not the lightest of one head behind heavier ones (with weights that are tiles, see
// pair_lists_kernel, 496 -> 465 us).  Taken
// back: only the heavier 60 % of a head's items by head and the rest by weight over all heads, which mixes the heads again (764 us).
template <typename Count>
__device__ __forceinline__ void sort_items_by_head(Count count_of, int n_items, int each, int Nkv, int ctas, int *hist, int32_t *__restrict__ order,
                                                   int *work_counter, int *error_flag) {
    const int T = blockDim.x, tid = threadIdx.x, heads = n_items / each;
    int *head_sum = hist + SCHED_BINS - 2 * SCHED_HEADS, *head_rank = head_sum + SCHED_HEADS;   // behind the items' weights
    for (int i = tid; i < heads; i += T) head_sum[i] = 0;
    if (tid == 0) {
        *work_counter = 0;
        *error_flag = 0;
    }
    __syncthreads();
    for (int i = tid; i < n_items; i += T) {
        const int w = max(0, min(count_of(i), Nkv));
        hist[i] = (w << 12) | (SCHED_BINS - 1 - i);      // all different: an item's rank is the number of larger ones
        atomicAdd(&head_sum[i / each], w);
    }
    __syncthreads();
    for (int i = tid; i < heads; i += T) {
        int rank = 0;
        for (int j = 0; j < heads; ++j) rank += head_sum[j] > head_sum[i] || (head_sum[j] == head_sum[i] && j < i);
        head_rank[i] = rank;
    }
    __syncthreads();
    const int alone = max(0, heads - (ctas + each - 1) / each);      // heads that keep to themselves
    for (int i = tid; i < n_items; i += T) {
        const int head = i / each, mine = hist[i], by_itself = head_rank[head] < alone;
        int rank = 0;
        for (int other = by_itself ? head : 0; other < (by_itself ? head + 1 : heads); ++other) {
            if (!by_itself && head_rank[other] < alone) continue;
#pragma unroll 8
            for (int j = 0; j < each; ++j) rank += hist[other * each + j] > mine;
        }
        order[(by_itself ? head_rank[head] : alone) * each + rank] = i;
    }
}

// Work order of single rows, heaviest first.  Called by every thread of ONE CTA whose size is a power of two between 32 and 1024.
// `count_of(row)` is a row's number of selected blocks.
template <typename Count>
__device__ __forceinline__ void schedule_rows(Count count_of, int rows, int Nkv, const SchedJob &job) {
    __shared__ int hist[SCHED_BINS];
    __shared__ int warp_tot[32];
    sort_items(count_of, rows, Nkv, hist, warp_tot, job.order, job.work_counter, job.error_flag);
}

// The same after a routing kernel, whose counts were written by other CTAs of this launch: they are read past L1.
__device__ inline void schedule_items(const int32_t *num, int rows, int Nq, int Nkv, const SchedJob &job) {
    __shared__ int hist[SCHED_BINS];
    __shared__ int warp_tot[32];
    if (!job.paired) {
        sort_items([&](int row) { return __ldcg(num + row); }, rows, Nkv, hist, warp_tot, job.order, job.work_counter, job.error_flag);
    } else if (job.by_counts) {
        const int each = (Nq + 1) >> 1;
        auto count_of = [&](int i) {      // no branches: a thread's look-ups are all on their way at once
            const int head = i / each, q = 2 * (i - head * each);
            const int32_t *at = num + (long long)head * Nq + q;
            return max(__ldcg(at), __ldcg(at + (q + 1 < Nq ? 1 : 0)));
        };
        sort_items(count_of, rows / Nq * each, Nkv, hist, warp_tot, job.order, job.work_counter, job.error_flag);
    }
}

// Elements [first, first + count) of the gate weight -> bf16 (it is an MMA operand) and of the bias -> float32.
__device__ inline void convert_gate_slice(const SchedJob &job, int first, int count) {
    if (first == 0 && threadIdx.x == 0 && job.pairs_done) *job.pairs_done = 0;
    if (!job.gate_w) return;
    if (job.gate_dt == WA_F32 && ((uintptr_t)job.gate_w & 15) == 0 && first % 4 == 0 && count % 4 == 0) {      // four at a time
        for (int i = first + 4 * threadIdx.x; i < first + count && i < 128 * 128; i += 4 * blockDim.x) {
            const float4 w = __ldg(reinterpret_cast<const float4 *>((const float *)job.gate_w + i));
            const __nv_bfloat162 lo = __floats2bfloat162_rn(w.x, w.y), hi = __floats2bfloat162_rn(w.z, w.w);
            *reinterpret_cast<uint2 *>(job.w_out + i) = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
            if (i < 128)
                *reinterpret_cast<float4 *>(job.b_out + i) =
                    job.gate_b ? make_float4(load_elem(job.gate_b, WA_F32, i), load_elem(job.gate_b, WA_F32, i + 1), load_elem(job.gate_b, WA_F32, i + 2),
                                             load_elem(job.gate_b, WA_F32, i + 3))
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        return;
    }
    for (int i = first + threadIdx.x; i < first + count && i < 128 * 128; i += blockDim.x) {
        job.w_out[i] = __float2bfloat16_rn(load_elem(job.gate_w, job.gate_dt, i));
        if (i < 128) job.b_out[i] = job.gate_b ? load_elem(job.gate_b, job.gate_dt, i) : 0.f;
    }
}

// routing (wa_routing.cu): pools x and optionally y in one launch; zeroes `n_zero` ints at `zero` on the way.
// `y_first_block`: the first blocks of y are already pooled in py (rows [0, y_first_block) per batch and head).
int pool_launch(const wa_tensor4 *x, int Lx, float *px, const wa_tensor4 *y, int Ly, float *py, int B, int H, int D,
                int block_size, cudaStream_t stream, int *zero = nullptr, int n_zero = 0, int y_first_block = 0,
                int *status_mirror = nullptr);   // host-visible word that receives a non-zero code if a bounded wait of the TMA kernel runs out

// routing (wa_routing.cu): scores, sort, Gini thresholds and counts, in one launch or, with many logits, two (plus `job` when its order is set).
// `sorted` ([rows, Nkv] float32) and `gini` ([rows]) are scratch; `counters` are H + 1 ints that are zero on entry.
int route_fused_launch(const float *q_pooled, const float *k_pooled, int B, int H, int Nq, int Nkv, int D, double tau_min,
                       double tau_max, const int32_t *fixed_num_per_head, float *sorted, int32_t *index, int32_t *num,
                       float *thresholds, float *gini, int *counters, const SchedJob &job, cudaStream_t stream,
                       bool whole_order = true);   // false: only the first num[row] ids of a row are needed (fixed counts)

// optional CUDA-event bracket around the attention kernel (wa_api.cu)
void profile_mark(bool begin, cudaStream_t stream);
void profile_pause(bool on);   // nested launches that must not move the bracket

// tcgen05 fused HSA kernel (wa_hsa_sm100.cu)
size_t hsa_sm100_workspace_bytes(const wa_hsa_params *p);
size_t hsa_sm100_status_offset(const wa_hsa_params *p);   // int32 flag inside the tuned workspace
bool hsa_sm100_supported(const wa_hsa_params *p, int Lc, const wa_tensor4 *kc, const wa_tensor4 *vc);
SchedJob hsa_sm100_sched_job(const wa_hsa_params *p, void *workspace);
// `prepared`: the SchedJob of this call has already run on the stream (as part of the routing kernel)
int hsa_sm100_launch(const wa_hsa_params *p, int Lc, const wa_tensor4 *kc, const wa_tensor4 *vc,
                     const int32_t *index, const int32_t *num, int Nq, int Nkv, void *workspace,
                     bool prepared, int32_t *lists, int32_t *both, cudaStream_t stream);   // scratch: as large as index, as num

// the linear branch alone on the tcgen05 kernel (bf16, head_dim 128; any routing block size): float32 [B, Lq, H, 128]
bool hsa_sm100_linear_supported(const wa_hsa_params *p, int Lc, const wa_tensor4 *kc, const wa_tensor4 *vc);
int hsa_sm100_launch_linear(const wa_hsa_params *p, int Lc, const wa_tensor4 *kc, const wa_tensor4 *vc, float *linear_out,
                            void *workspace, cudaStream_t stream);

// block-mean pooling as a TMA stream (wa_pool_sm100.cu); y may be null; out_blocks_y = rows per (batch, head) of py
bool pool_sm100_supported(const wa_tensor4 *x, const wa_tensor4 *y, int H, int D, int block_size);
int pool_sm100_launch(const wa_tensor4 *x, int Lx, float *px, const wa_tensor4 *y, int Ly, float *py, int out_blocks_y, int B, int H,
                      int D, int block_size, cudaStream_t stream, int *zero, int n_zero, int *status_mirror);

// compress_kv / KV-cache append as a TMA + tcgen05 stream (wa_compress_sm100.cu)
bool compress_sm100_supported(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *ok, const wa_tensor4 *ov,
                              const wa_tensor4 *dst_k, const wa_tensor4 *dst_v, int H, int D, int proj_dtype, int proj_cols,
                              int rank_full, const void *k_proj, const void *v_proj);
int compress_sm100_launch(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *ok, const wa_tensor4 *ov,
                          const wa_tensor4 *dst_k, const wa_tensor4 *dst_v, int dst_row0, int B, int L, int H, int D,
                          int segment_len, int block_size, const void *k_proj, const void *v_proj, int proj_rank, int proj_cols,
                          int slot0, int slot_stride, cudaStream_t stream, bool beside_routing = false);

// wa_block_sparse_forward and wa_linear_branch for wa_hsa_forward.  `order`: routing rows in the order in which they are taken (heaviest
// first), or null.  `ahead`: the launch after this one may start while it runs; `beside`: this launch reads nothing that the one before it
// writes and starts on what that leaves free, but completes only after it (head_dim 128; otherwise one after the other).
int block_sparse_run(const wa_tensor4 *q, const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *out, int B, int H, int Lq, int Lkv, int D,
                     int block_size, const int32_t *index, const int32_t *num, int index_stride, const int32_t *block_sizes, int round_inputs_bf16,
                     int round_output_bf16, float *lse, const int32_t *order, bool ahead, cudaStream_t stream);
int linear_run(const wa_tensor4 *q, const wa_tensor4 *k_coarse, const wa_tensor4 *v_coarse, const wa_tensor4 *out, int B, int H, int Lq, int Lc,
               int D, int round_output_bf16, float *lse, bool beside, cudaStream_t stream);

// float32 keys and values rounded to bf16, both contiguous `[B, L, H, D]` at dst, for the sparse branch (wa_attention_generic.cu)
bool round_kv_supported(const wa_tensor4 *k, const wa_tensor4 *v, int D);
// `beside`: it starts on what the launch before it leaves free, and completes only after that one.
int round_kv_launch(const wa_tensor4 *k, const wa_tensor4 *v, int B, int L, int H, int D, void *dst, bool beside, cudaStream_t stream);

// CTAs per head of the routing of short rows (route_head_kernel), 0 where another kernel routes
int route_short_parts(int B, int Nq, int Nkv, int D, bool beside);

// SMs that compress_kv_launch takes up if compress_cluster_kernel covers the call, otherwise 0.
int compress_cluster_sms(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *out_k, const wa_tensor4 *out_v, int B, int L, int H,
                         int D, int segment_len, int block_size, const void *k_proj, const void *v_proj, int proj_dtype, int proj_rank,
                         int proj_cols, int others);

// compress_kv by whichever kernel covers the call (wa_compress.cu).  `beside_routing`: the launch before this one on the
// stream is a routing kernel that released its dependents at its start (SchedJob::release_at_start).  The two share nothing, so
// the compression runs on what the routing leaves free of the chip; it completes only after the routing has, so that
// whatever waits for it may read both.  (One latent frame of 390 tokens over three: the call 49.5 -> 43.1 us.)  `ahead`: the launch
// after this one reads nothing of it and may start while it runs (where the kernel that covers the call does so).  `others`: SMs that the launch before it
// keeps busy.
int compress_kv_launch(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *out_k, const wa_tensor4 *out_v, int B, int L, int H, int D,
                       int segment_len, int block_size, const void *k_proj, const void *v_proj, int proj_dtype, int proj_rank, int proj_cols,
                       bool beside_routing, cudaStream_t stream, bool ahead = false, int others = 0);

}  // namespace wa
