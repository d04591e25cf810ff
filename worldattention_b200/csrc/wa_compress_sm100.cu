// compress_kv -- and the KV-cache append fused with it -- as a TMA-fed tcgen05 stream for sm_100a.
//
// compress_kv (wan/modules/hsa/attention.py:64-110) is, per segment, the product of the [rank x tokens]
// projection with the [tokens x H*D] token rows: 13..25 output rows for 1560 x 1536 inputs, so the
// kernel's job is to read K and V once at HBM speed; the contraction itself rides along on the tensor
// cores.  Work item = (128 or 64 columns, segment, K|V, batch).  A persistent CTA of four warps streams the
// item's tokens in 128-token tiles through a five-stage shared-memory ring:
//   warp 1  TMA loads: the token tile [128 tokens x columns] and the matching [32 rows x 128 tokens] tile of the
//           projection (rows past the rank and tokens past the segment come back as zeros).  The copy engine works by
//           128-byte row pieces, so only the rows that a rank can have are loaded: the product has M = 128 rows, and
//           what lies in shared memory behind the 32 enters accumulator lanes that nobody reads;
//   warp 2  tcgen05.mma, D[rank rows x 128 columns] (+)= E_tile . X_tile, float32 in tensor memory,
//           two accumulators so that the next item starts while the last one is read out;
//   warp 3  (append only) TMA store of the same shared-memory tile into the KV cache -- the rows are
//           read from HBM once and leave twice;
//   warp 0  reads the accumulator's first `rank` lanes and writes the bf16 slots.
// 64 columns per item where items of 128 would leave SMs without one (a chunk of a few segments).
// 12 heads of 128, segments of 1560 tokens: twelve segments 32.7 -> 23 us (115 MB: 5.0 TB/s), three appended ones 17.4 -> 13.3 us
// against three stages and projection tiles of 128 rows.
// Every mbarrier wait is bounded; a wait that runs out raises a flag that wa_compress_status reads.
#include <cstring>

#include "wa_internal.cuh"
#include "wa_sm100_ptx.cuh"

namespace wa {
namespace sm100 {
namespace compress {

constexpr int THREADS = 128;
constexpr int STAGES = 5;
constexpr int E_ROWS = 32, E_HALF_BYTES = E_ROWS * 128;    // projection tile: two halves of 64 tokens, 32 rows of 128 bytes each
constexpr int STAGE_BYTES = TILE_BYTES + 2 * E_HALF_BYTES; // token tile + projection tile
// the A operand of the last stage's products reaches 128 rows past the start of its second half
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES - E_HALF_BYTES + HALF_BYTES + 1024;
constexpr int TMEM_COLS = 256;                             // two [128 x 128] float32 accumulators

struct Barriers {
    uint64_t full[STAGES], empty[STAGES];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(STAGES * STAGE_BYTES + sizeof(Barriers) <= SMEM_BYTES && SMEM_BYTES <= 227 * 1024, "shared memory budget");

struct Job {
    int n_seg, tiles_cols, B;          // items = B * 2 * n_seg * tiles_cols
    int cols;                          // columns of an item: 128 or 64
    int L, segment_len, block_size, proj_rank;
    int slot0, slot_stride;            // first compressed slot of segment 0; slots between consecutive segments
    int beside;                        // runs beside the launch before it, whose results it neither reads nor overwrites
    int copy;                          // also store the token tiles through the destination maps
    __nv_bfloat16 *out_k, *out_v;
    long long osb, osl;
    int *status;
};

__device__ int g_status;               // 0, or the site code of a wait that ran out

// Accumulator row `lane` (rank <= 32 is a condition of these kernels) as bf16 to `out`, 32 columns at a time; by a whole warp.
__device__ __forceinline__ void write_slots(__nv_bfloat16 *out, uint32_t acc, int cols, bool real) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (c * 32 >= cols) break;
        uint32_t v[32];
        TMEM_LD32(acc + c * 32, v);
        tmem_wait_ld();
        if (real) {
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                packed[j] = *reinterpret_cast<uint32_t *>(&h);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<uint4 *>(out + c * 32 + j * 8) = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
        }
    }
}

__global__ void __launch_bounds__(THREADS, 1)
compress_stream_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const __grid_constant__ CUtensorMap tm_ek, const __grid_constant__ CUtensorMap tm_ev,
                       const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv, const Job job) {
    extern __shared__ __align__(1024) uint8_t smem[];
    Barriers *bar = reinterpret_cast<Barriers *>(smem + STAGES * STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort_flag = &bar->abort_flag;
    const FailSink sink{job.status, nullptr};

    if (threadIdx.x == 0) {
        bar->abort_flag = (smem_u32(smem) & 1023u) ? 1 : 0;
        if (bar->abort_flag) report_failure(sink, 99);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&bar->full[i], 1);
            mbar_init(&bar->empty[i], job.copy ? 2 : 1);   // the products that read the stage have landed (+ the store warp is done with it)
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar->acc_full[i], 1);
            mbar_init(&bar->acc_empty[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bar->tmem_base)),
                     "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (!job.beside) pdl_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bar->tmem_base;
    const int n_items = job.B * 2 * job.n_seg * job.tiles_cols;

    // item -> (column tile fastest, then segment, K|V, batch): neighbouring CTAs read neighbouring columns of the same rows
    auto decode = [&](int item, int &ct, int &seg, int &which, int &b) {
        ct = item % job.tiles_cols;
        seg = (item / job.tiles_cols) % job.n_seg;
        which = (item / (job.tiles_cols * job.n_seg)) & 1;
        b = item / (job.tiles_cols * job.n_seg * 2);
    };
    auto seg_tiles = [&](int seg) {
        const int n_tok = min(job.segment_len, job.L - seg * job.segment_len);
        return (n_tok + TILE - 1) / TILE;
    };

    if (warp == 1) {
        // ================= producer =================
        if (lane == 0) {
            uint32_t count = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                int ct, seg, which, b;
                decode(item, ct, seg, which, b);
                const CUtensorMap *tx = which ? &tm_v : &tm_k, *te = which ? &tm_ev : &tm_ek;
                const int tok0 = seg * job.segment_len, n_tiles = seg_tiles(seg);
                for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                    const uint32_t s = count % STAGES;
                    ok = mbar_wait(&bar->empty[s], ((count / STAGES) & 1u) ^ 1u, abort_flag, sink, 1);
                    if (!ok) break;
                    uint8_t *xs = smem + s * STAGE_BYTES, *es = xs + TILE_BYTES;
                    mbar_expect_tx(&bar->full[s], (job.cols == TILE ? TILE_BYTES : HALF_BYTES) + 2 * E_HALF_BYTES);
                    tma_load_3d(xs, tx, &bar->full[s], ct * job.cols, tok0 + t * TILE, b);
                    if (job.cols == TILE) tma_load_3d(xs + HALF_BYTES, tx, &bar->full[s], ct * job.cols + 64, tok0 + t * TILE, b);
                    tma_load_2d(es, te, &bar->full[s], t * TILE, 0);
                    tma_load_2d(es + E_HALF_BYTES, te, &bar->full[s], t * TILE + 64, 0);
                }
            }
        }
    } else if (warp == 2) {
        // ================= issuer =================
        const bool leader = elect_one();
        const uint32_t idesc = job.cols == TILE ? instr_desc(true, TILE) : instr_desc(true, 64);   // A = projection tile (K-major), B = token tile (columns contiguous)
        uint32_t count = 0, n_done = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++n_done) {
            int ct, seg, which, b;
            decode(item, ct, seg, which, b);
            const uint32_t buf = n_done & 1u;
            // the accumulator was read out two items ago
            ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_empty[buf], ((n_done >> 1) & 1u) ^ 1u, abort_flag, sink, 2));
            if (!ok) break;
            const int n_tiles = seg_tiles(seg);
            for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                const uint32_t s = count % STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(&bar->full[s], (count / STAGES) & 1u, abort_flag, sink, 3));
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t xs = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t bd = smem_desc(xs, HALF_BYTES, 1024), ad = smem_desc(xs + TILE_BYTES, 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        mma_ss(tmem + buf * TILE, ad + (uint64_t)(((kk >> 2) * E_HALF_BYTES + (kk & 3) * 32) >> 4),
                               bd + (uint64_t)((kk * 2048) >> 4), idesc, !(t == 0 && kk == 0));
                    tc_commit(&bar->empty[s]);
                    if (t == n_tiles - 1) tc_commit(&bar->acc_full[buf]);
                }
                __syncwarp();
            }
        }
    } else if (warp == 3) {
        // ================= store warp: the token tile also goes to the cache (append), or straight back to the producer ===
        if (lane == 0 && job.copy) {
            uint32_t count = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                int ct, seg, which, b;
                decode(item, ct, seg, which, b);
                const CUtensorMap *td = which ? &tm_dv : &tm_dk;
                const int tok0 = seg * job.segment_len, n_tiles = seg_tiles(seg);
                for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                    const uint32_t s = count % STAGES;
                    ok = mbar_wait(&bar->full[s], (count / STAGES) & 1u, abort_flag, sink, 4);
                    if (!ok) break;
                    uint8_t *xs = smem + s * STAGE_BYTES;
                    // rows past the appended range are clipped by the destination map
                    tma_store_3d(td, xs, ct * job.cols, tok0 + t * TILE, b);
                    if (job.cols == TILE) tma_store_3d(td, xs + HALF_BYTES, ct * job.cols + 64, tok0 + t * TILE, b);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    mbar_arrive(&bar->empty[s]);
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else {
        // ================= epilogue: accumulator rows (= ranks) of lanes 0..31, 32 columns at a time =================
        uint32_t n_done = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++n_done) {
            int ct, seg, which, b;
            decode(item, ct, seg, which, b);
            const uint32_t buf = n_done & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_full[buf], (n_done >> 1) & 1u, abort_flag, sink, 5));
            if (!ok) break;
            tc_fence_after();
            const int n_tok = min(job.segment_len, job.L - seg * job.segment_len);
            const int rank = min(job.proj_rank, (n_tok + job.block_size - 1) / job.block_size);
            __nv_bfloat16 *out = (which ? job.out_v : job.out_k) + (long long)b * job.osb +
                                 (long long)(job.slot0 + seg * job.slot_stride + lane) * job.osl + ct * job.cols;
            write_slots(out, tmem + buf * TILE, job.cols, lane < rank);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->acc_empty[buf]);
        }
    }

    pdl_wait();       // beside the routing (see compress_kv_launch): done only when that is
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// Install of retrieved pages into the online caches of all layers, fused with the compression of what is installed: the copy
// loop of HKVCache.apply (pipeline/hkv/cache.py:229-254) and compress_kv of every layer in ONE launch.  As two steps the pages are
// read and written once and read once more (30 blocks, twelve frames of 1560 x 1536: 1.23 ms and 30 x 23 us); here the token tile
// that the product needs is the one that is stored: 1.20 ms (6.9 GB: 5.8 TB/s, bound by HBM), the whole retrieval and install 3.55 -> 2.70 ms.
//
// Work item = (128 columns, frame, layer and K|V, batch item), the stream above with four more warps between the load and its two
// consumers: they turn the keys' temporal pairs by the page's rotation, in place, with the page-copy kernel's arithmetic.
// Token tiles come from a 4-D map (column, token of the frame, frame, batch), so that rows behind a frame's end arrive
// as zeros and are not stored, whatever lies there.  The maps of all pages, layers and projections lie in a table in global
// memory that the caller fills on the host (wa_hkv_install_table).  Same tiles and order of products as compress_stream_kernel:
// the slots are the same bits.
// ------------------------------------------------------------------------------------------------
namespace install {

constexpr int TURN_WARPS = 4, WARPS = 4 + TURN_WARPS;

struct Slots {                 // compressed slots of one (layer, K|V)
    __nv_bfloat16 *base;
    long long batch, row;      // strides in elements
};
struct Segment {               // one installed frame
    int page, frame, rot, pad; // row of the plan, frame inside it, row of the rotation table or -1
};
struct Table {                 // offsets in bytes
    size_t dst, proj, slots, segments, total;
};
__host__ __device__ inline Table table_plan(int pages, int tensors, int segments) {
    Table t;
    t.dst = (size_t)pages * tensors * sizeof(CUtensorMap);
    t.proj = t.dst + (size_t)tensors * sizeof(CUtensorMap);
    t.slots = t.proj + (size_t)tensors * sizeof(CUtensorMap);
    t.segments = t.slots + (size_t)tensors * sizeof(Slots);
    t.total = t.segments + (size_t)segments * sizeof(Segment);
    return t;
}
struct Job {
    const unsigned char *table;
    Table at;
    const float2 *rotations;
    int tensors, n_seg, tiles_cols, B, D, frame, rank, nt;
    int *status, *status_mirror;
};

struct Barriers {
    uint64_t full[STAGES], ready[STAGES], empty[STAGES];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(STAGES * STAGE_BYTES + sizeof(Barriers) <= SMEM_BYTES, "shared memory budget");

// a tensor map in global memory that the host wrote
__device__ __forceinline__ const CUtensorMap *acquire_map(const unsigned char *at) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(at) : "memory");
    return reinterpret_cast<const CUtensorMap *>(at);
}

__global__ void __launch_bounds__(WARPS * 32, 1)
install_stream_kernel(const Job job) {
    extern __shared__ __align__(1024) uint8_t smem[];
    Barriers *bar = reinterpret_cast<Barriers *>(smem + STAGES * STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int *abort_flag = &bar->abort_flag;
    const FailSink sink{job.status, job.status_mirror};      // sites 301 to 309
    const Segment *segments = reinterpret_cast<const Segment *>(job.table + job.at.segments);

    if (threadIdx.x == 0) {
        bar->abort_flag = (smem_u32(smem) & 1023u) ? 1 : 0;
        if (bar->abort_flag) report_failure(sink, 309);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&bar->full[i], 1);
            mbar_init(&bar->ready[i], TURN_WARPS);
            mbar_init(&bar->empty[i], 2);      // the products and the store have read the stage
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar->acc_full[i], 1);
            mbar_init(&bar->acc_empty[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bar->tmem_base)),
                     "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bar->tmem_base;
    const int n_tiles = (job.frame + TILE - 1) / TILE;
    const int n_items = job.B * job.tensors * job.n_seg * job.tiles_cols;
    // item -> (column tile fastest, then frame, layer and K|V, batch)
    auto decode = [&](int item, int &ct, int &seg, int &tensor, int &b) {
        ct = item % job.tiles_cols;
        seg = (item / job.tiles_cols) % job.n_seg;
        tensor = (item / (job.tiles_cols * job.n_seg)) % job.tensors;
        b = item / (job.tiles_cols * job.n_seg * job.tensors);
    };

    if (warp == 1) {
        // ================= producer =================
        if (lane == 0) {
            uint32_t count = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                int ct, seg, tensor, b;
                decode(item, ct, seg, tensor, b);
                const Segment sg = segments[seg];
                const CUtensorMap *tx = acquire_map(job.table + ((size_t)sg.page * job.tensors + tensor) * sizeof(CUtensorMap));
                const CUtensorMap *te = acquire_map(job.table + job.at.proj + (size_t)tensor * sizeof(CUtensorMap));
                for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                    const uint32_t s = count % STAGES;
                    ok = mbar_wait(&bar->empty[s], ((count / STAGES) & 1u) ^ 1u, abort_flag, sink, 301);
                    if (!ok) break;
                    uint8_t *xs = smem + s * STAGE_BYTES, *es = xs + TILE_BYTES;
                    mbar_expect_tx(&bar->full[s], TILE_BYTES + 2 * E_HALF_BYTES);
                    tma_load_4d(xs, tx, &bar->full[s], ct * TILE, t * TILE, sg.frame, b);
                    tma_load_4d(xs + HALF_BYTES, tx, &bar->full[s], ct * TILE + 64, t * TILE, sg.frame, b);
                    tma_load_2d(es, te, &bar->full[s], t * TILE, 0);
                    tma_load_2d(es + E_HALF_BYTES, te, &bar->full[s], t * TILE + 64, 0);
                }
            }
        }
    } else if (warp == 2) {
        // ================= issuer =================
        const bool leader = elect_one();
        constexpr uint32_t idesc = instr_desc(true, TILE);
        uint32_t count = 0, n_done = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++n_done) {
            const uint32_t buf = n_done & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_empty[buf], ((n_done >> 1) & 1u) ^ 1u, abort_flag, sink, 302));
            if (!ok) break;
            for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                const uint32_t s = count % STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(&bar->full[s], (count / STAGES) & 1u, abort_flag, sink, 303) &&
                                                 mbar_wait(&bar->ready[s], (count / STAGES) & 1u, abort_flag, sink, 304));
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t xs = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t bd = smem_desc(xs, HALF_BYTES, 1024), ad = smem_desc(xs + TILE_BYTES, 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        mma_ss(tmem + buf * TILE, ad + (uint64_t)(((kk >> 2) * E_HALF_BYTES + (kk & 3) * 32) >> 4),
                               bd + (uint64_t)((kk * 2048) >> 4), idesc, !(t == 0 && kk == 0));
                    tc_commit(&bar->empty[s]);
                    if (t == n_tiles - 1) tc_commit(&bar->acc_full[buf]);
                }
                __syncwarp();
            }
        }
    } else if (warp == 3) {
        // ================= store =================
        if (lane == 0) {
            uint32_t count = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                int ct, seg, tensor, b;
                decode(item, ct, seg, tensor, b);
                const CUtensorMap *td = acquire_map(job.table + job.at.dst + (size_t)tensor * sizeof(CUtensorMap));
                for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                    const uint32_t s = count % STAGES;
                    ok = mbar_wait(&bar->full[s], (count / STAGES) & 1u, abort_flag, sink, 305) &&
                         mbar_wait(&bar->ready[s], (count / STAGES) & 1u, abort_flag, sink, 306);
                    if (!ok) break;
                    const uint8_t *xs = smem + s * STAGE_BYTES;
                    tma_store_4d(td, xs, ct * TILE, t * TILE, seg, b);
                    tma_store_4d(td, xs + HALF_BYTES, ct * TILE + 64, t * TILE, seg, b);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    mbar_arrive(&bar->empty[s]);
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else if (warp >= 4) {
        // ================= turn: a thread per token row, 16-byte pieces of four pairs =================
        const int row = threadIdx.x - 128;
        uint32_t count = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            int ct, seg, tensor, b;
            decode(item, ct, seg, tensor, b);
            const int rot = (tensor & 1) || !job.rotations ? -1 : segments[seg].rot;
            const float2 *turn = job.rotations + (long long)max(rot, 0) * job.nt;
            for (int t = 0; t < n_tiles && ok; ++t, ++count) {
                const uint32_t s = count % STAGES;
                ok = __all_sync(0xffffffffu, mbar_wait(&bar->full[s], (count / STAGES) & 1u, abort_flag, sink, 307));
                if (!ok) break;
                if (rot >= 0) {
                    uint8_t *line = smem + s * STAGE_BYTES + row * 128;
#pragma unroll 1
                    for (int piece = 0; piece < 16; ++piece) {
                        const int pair0 = ((ct * TILE + piece * 8) % job.D) >> 1;     // of the head that the piece belongs to
                        if (pair0 >= job.nt) continue;
                        uint4 *at = reinterpret_cast<uint4 *>(line + (piece >> 3) * HALF_BYTES + (((piece & 7) ^ (row & 7)) << 4));
                        const uint4 v = *at;
                        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (pair0 + e < job.nt) {
                                const float2 f = __ldg(turn + pair0 + e);
                                const float a = __uint_as_float(w[e] << 16), c = __uint_as_float(w[e] & 0xffff0000u);
                                const __nv_bfloat162 o = __floats2bfloat162_rn(__fsub_rn(__fmul_rn(a, f.x), __fmul_rn(c, f.y)),
                                                                               __fadd_rn(__fmul_rn(a, f.y), __fmul_rn(c, f.x)));
                                w[e] = *reinterpret_cast<const uint32_t *>(&o);
                            }
                        *at = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the products and the store read it by the other proxy
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar->ready[s]);
            }
        }
    } else {
        // ================= epilogue: accumulator rows (= ranks) of lanes 0..31 =================
        uint32_t n_done = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++n_done) {
            int ct, seg, tensor, b;
            decode(item, ct, seg, tensor, b);
            const uint32_t buf = n_done & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(&bar->acc_full[buf], (n_done >> 1) & 1u, abort_flag, sink, 308));
            if (!ok) break;
            tc_fence_after();
            const Slots sl = reinterpret_cast<const Slots *>(job.table + job.at.slots)[tensor];
            write_slots(sl.base + (long long)b * sl.batch + (long long)(seg * job.rank + lane) * sl.row + ct * TILE, tmem + buf * TILE, TILE,
                        lane < job.rank);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->acc_empty[buf]);
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace install

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// `[B, rows, H*D]` bf16 rows with contiguous heads -> 3-D map (column, row, batch), box 64 x 128 x 1, 128-byte swizzle.
static bool map_rows(CUtensorMap *map, void *base, int cols, int rows, int B, long long stride_row, long long stride_b) {
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)B};
    cuuint64_t strides[2] = {(cuuint64_t)stride_row * 2, (cuuint64_t)(B == 1 ? stride_row * rows : stride_b) * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)TILE, 1}, elem[3] = {1, 1, 1};
    return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// projection `[rank, proj_cols]` bf16 -> 2-D map (token, rank) restricted to the first `tokens` columns, box 64 x 32
static bool map_projection(CUtensorMap *map, const void *base, int tokens, int rank, int proj_cols) {
    cuuint64_t dims[2] = {(cuuint64_t)tokens, (cuuint64_t)rank};
    cuuint64_t strides[1] = {(cuuint64_t)proj_cols * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)E_ROWS}, elem[2] = {1, 1};
    return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, elem,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// whole frames of `[B, rows, H*D]` bf16 rows (contiguous) -> 4-D map (column, token, frame, batch), box 64 x 128 x 1 x 1
static bool map_frames(CUtensorMap *map, unsigned long long base, int cols, int frame, int frames, int B, long long stride_b) {
    const cuuint64_t row = (cuuint64_t)cols * 2;
    cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)frame, (cuuint64_t)frames, (cuuint64_t)B};
    cuuint64_t strides[3] = {row, row * frame, B == 1 ? row * frame * frames : (cuuint64_t)stride_b * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)TILE, 1, 1}, elem[4] = {1, 1, 1, 1};
    return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, reinterpret_cast<void *>(base), dims, strides, box, elem,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int *status_address() {   // of the current device; looked up once per device
    static int *status_of[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!status_of[dev] && cudaGetSymbolAddress((void **)&status_of[dev], g_status) != cudaSuccess) status_of[dev] = nullptr;
    return status_of[dev];
}

}  // namespace compress
}  // namespace sm100

// Whether the tcgen05 stream covers this call (bf16 everything, contiguous heads, 16-byte aligned rows, rank <= 32,
// an sm_100 device); `dst_*` are null for a plain compress_kv.
bool compress_sm100_supported(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *ok, const wa_tensor4 *ov,
                              const wa_tensor4 *dst_k, const wa_tensor4 *dst_v, int H, int D, int proj_dtype, int proj_cols,
                              int rank_full, const void *k_proj, const void *v_proj) {
    using namespace sm100::compress;
    const wa_tensor4 *views[6] = {k, v, ok, ov, dst_k, dst_v};
    for (const wa_tensor4 *t : views) {
        if (!t) continue;
        if (t->dtype != WA_BF16 || t->stride_h != D || (uintptr_t)t->ptr % 16 || t->stride_l % 8 || t->stride_b % 8 || t->stride_l < (long long)H * D)
            return false;
    }
    if (proj_dtype != WA_BF16 || (H * D) % sm100::TILE || rank_full > 32 || proj_cols % 8 || (uintptr_t)k_proj % 16 || (uintptr_t)v_proj % 16)
        return false;
    int dev = 0, major = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        major != 10)
        return false;
    return encode_fn() != nullptr;
}

// Compress the L tokens of `k` / `v` (segments of segment_len from token 0) into slots slot0 + seg * slot_stride + r of
// out_k / out_v; with dst_k / dst_v also copy the rows to rows [dst_row0, dst_row0 + L) of those tensors.
int compress_sm100_launch(const wa_tensor4 *k, const wa_tensor4 *v, const wa_tensor4 *ok, const wa_tensor4 *ov,
                          const wa_tensor4 *dst_k, const wa_tensor4 *dst_v, int dst_row0, int B, int L, int H, int D,
                          int segment_len, int block_size, const void *k_proj, const void *v_proj, int proj_rank, int proj_cols,
                          int slot0, int slot_stride, cudaStream_t stream, bool beside_routing) {
    using namespace sm100::compress;
    const char *what = "wa_compress_kv(tcgen05)";
    const int cols = H * D;
    CUtensorMap tk, tv, tek, tev, tdk, tdv;
    bool good = map_rows(&tk, k->ptr, cols, L, B, k->stride_l, k->stride_b) && map_rows(&tv, v->ptr, cols, L, B, v->stride_l, v->stride_b);
    const int e_tokens = proj_cols < segment_len ? proj_cols : segment_len;
    good = good && map_projection(&tek, k_proj, e_tokens, proj_rank, proj_cols) && map_projection(&tev, v_proj, e_tokens, proj_rank, proj_cols);
    const bool copy = dst_k != nullptr;
    if (copy) {
        char *bk = (char *)dst_k->ptr + (size_t)dst_row0 * dst_k->stride_l * 2, *bv = (char *)dst_v->ptr + (size_t)dst_row0 * dst_v->stride_l * 2;
        good = good && map_rows(&tdk, bk, cols, L, B, dst_k->stride_l, dst_k->stride_b) &&
               map_rows(&tdv, bv, cols, L, B, dst_v->stride_l, dst_v->stride_b);
    } else {
        tdk = tk;
        tdv = tv;
    }
    WA_REQUIRE(good, WA_ERR_ALIGN, "%s: a tensor map was rejected", what);
    static PerDeviceOnce attr_set;
    if (!attr_set.done()) {
        cudaError_t e = cudaFuncSetAttribute(compress_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
        attr_set.mark();
    }
    int *status = status_address();
    if (!status) return fail(WA_ERR_DEVICE, "%s: no usable current device", what);
    Job job{};
    job.n_seg = ceil_div(L, segment_len);
    job.B = B;
    job.L = L; job.segment_len = segment_len; job.block_size = block_size; job.proj_rank = proj_rank;
    job.slot0 = slot0; job.slot_stride = slot_stride;
    job.copy = copy ? 1 : 0;
    job.out_k = (__nv_bfloat16 *)ok->ptr; job.out_v = (__nv_bfloat16 *)ov->ptr;
    job.osb = ok->stride_b; job.osl = ok->stride_l;
    job.status = status;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    job.cols = (long long)B * 2 * job.n_seg * (cols / sm100::TILE) < sms ? 64 : sm100::TILE;
    job.tiles_cols = cols / job.cols;
    const long long items = (long long)B * 2 * job.n_seg * job.tiles_cols;
    WA_REQUIRE(items < (1ll << 30), WA_ERR_UNSUPPORTED, "%s: too many work items", what);
    const int grid = items < sms ? (int)items : sms;
    job.beside = beside_routing ? 1 : 0;
    const cudaError_t e = launch_dependent(compress_stream_kernel, dim3(grid), dim3(THREADS), SMEM_BYTES, stream, tk, tv, tek, tev, tdk, tdv, job);
    if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
    return check_launch(what);
}

}  // namespace wa

extern "C" int wa_compress_status(int *status) {
    using namespace wa;
    WA_REQUIRE(status, WA_ERR_ARG, "wa_compress_status: null pointer");
    cudaError_t e = cudaMemcpyFromSymbol(status, sm100::compress::g_status, sizeof(int));
    if (e != cudaSuccess) return fail((int)e, "wa_compress_status: %s", cudaGetErrorString(e));
    return 0;
}

extern "C" size_t wa_hkv_install_table_bytes(int pages, int tensors, int segments) {
    if (pages <= 0 || tensors <= 0 || segments <= 0) return 0;
    return wa::sm100::compress::install::table_plan(pages, tensors, segments).total;
}

static int install_check(const wa_hkv_install *p, const char *what) {
    using namespace wa;
    WA_REQUIRE(p && p->page_frames && p->page_rot && p->src && p->src_batch && p->dst && p->dst_batch && p->coarse && p->coarse_batch &&
                   p->coarse_row && p->proj,
               WA_ERR_ARG, "%s: null pointer", what);
    WA_REQUIRE(p->pages > 0 && p->tensors > 0 && p->tensors % 2 == 0 && p->B > 0 && p->H > 0 && p->D > 0 && p->frame > 0 && p->segments > 0 &&
                   p->block_size > 0 && p->proj_rank > 0 && p->proj_cols >= p->frame && p->n_temporal >= 0 && 2 * p->n_temporal <= p->D,
               WA_ERR_ARG, "%s: bad sizes", what);
    return 0;
}

static int install_rank(const wa_hkv_install *p) {
    const int blocks = wa::ceil_div(p->frame, p->block_size);
    return p->proj_rank < blocks ? p->proj_rank : blocks;
}

extern "C" int wa_hkv_install_table(const wa_hkv_install *p, void *table, size_t bytes) {
    using namespace wa;
    using namespace wa::sm100::compress;
    const char *what = "wa_hkv_install_table";
    if (const int rc = install_check(p, what)) return rc;
    const install::Table at = install::table_plan(p->pages, p->tensors, p->segments);
    WA_REQUIRE(table && bytes >= at.total, WA_ERR_ARG, "%s: a table of %zu bytes is needed", what, at.total);
    const int cols = p->H * p->D;
    int total = 0;
    for (int i = 0; i < p->pages; ++i) {
        WA_REQUIRE(p->page_frames[i] > 0, WA_ERR_ARG, "%s: page %d holds no frame", what, i);
        total += p->page_frames[i];
    }
    WA_REQUIRE(total == p->segments, WA_ERR_ARG, "%s: the pages hold %d frames, not %d", what, total, p->segments);
    int dev = 0, major = 0;
    bool good = cudaGetDevice(&dev) == cudaSuccess &&
                cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) == cudaSuccess && major == 10;
    good = good && cols % wa::sm100::TILE == 0 && p->D % 8 == 0 && p->proj_cols % 8 == 0 && install_rank(p) <= 32 &&
           (long long)p->B * p->tensors * p->segments * (cols / wa::sm100::TILE) < (1ll << 30);
    for (int t = 0; t < p->tensors && good; ++t) {
        good = p->dst[t] % 16 == 0 && p->coarse[t] % 16 == 0 && p->proj[t] % 16 == 0 && p->coarse_row[t] % 8 == 0 && p->coarse_batch[t] % 8 == 0 &&
               (p->B == 1 || p->dst_batch[t] % 8 == 0);
        for (int i = 0; i < p->pages && good; ++i)
            good = p->src[(size_t)i * p->tensors + t] % 16 == 0 && (p->B == 1 || p->src_batch[(size_t)i * p->tensors + t] % 8 == 0);
    }
    WA_REQUIRE(good && encode_fn(), WA_ERR_UNSUPPORTED, "%s: not covered (rows of a multiple of 128 values, 16-byte aligned, rank <= 32)", what);
    unsigned char *base = reinterpret_cast<unsigned char *>(table);
    alignas(64) CUtensorMap map;      // the table itself need not be aligned on the host
    const auto put = [&](size_t offset) { memcpy(base + offset, &map, sizeof map); };
    for (int t = 0; t < p->tensors && good; ++t) {
        for (int i = 0; i < p->pages && good; ++i) {
            const size_t e = (size_t)i * p->tensors + t;
            good = map_frames(&map, p->src[e], cols, p->frame, p->page_frames[i], p->B, p->src_batch[e]);
            put(e * sizeof map);
        }
        good = good && map_frames(&map, p->dst[t], cols, p->frame, p->segments, p->B, p->dst_batch[t]);
        put(at.dst + t * sizeof map);
        good = good && map_projection(&map, reinterpret_cast<const void *>(p->proj[t]), p->frame, p->proj_rank, p->proj_cols);
        put(at.proj + t * sizeof map);
        const install::Slots sl{reinterpret_cast<__nv_bfloat16 *>(p->coarse[t]), (long long)p->coarse_batch[t], (long long)p->coarse_row[t]};
        memcpy(base + at.slots + t * sizeof sl, &sl, sizeof sl);
    }
    WA_REQUIRE(good, WA_ERR_UNSUPPORTED, "%s: a tensor map was rejected", what);
    int n = 0;
    for (int i = 0; i < p->pages; ++i)
        for (int f = 0; f < p->page_frames[i]; ++f, ++n) {
            const install::Segment sg{i, f, p->page_rot[i], 0};
            memcpy(base + at.segments + n * sizeof sg, &sg, sizeof sg);
        }
    return 0;
}

extern "C" int wa_hkv_install_pages(const wa_hkv_install *p, const void *device_table, const float *rotations, void *stream) {
    return wa_hkv_install_pages_mirrored(p, device_table, rotations, nullptr, stream);
}

extern "C" int wa_hkv_install_pages_mirrored(const wa_hkv_install *p, const void *device_table, const float *rotations, int32_t *status_mirror,
                                             void *stream) {
    using namespace wa;
    using namespace wa::sm100::compress;
    const char *what = "wa_hkv_install_pages";
    if (const int rc = install_check(p, what)) return rc;
    WA_REQUIRE(device_table && (uintptr_t)device_table % 64 == 0, WA_ERR_ALIGN, "%s: the table must be 64-byte aligned", what);
    static PerDeviceOnce attr_set;
    if (!attr_set.done()) {
        const cudaError_t e = cudaFuncSetAttribute(install::install_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return fail((int)e, "%s: %s", what, cudaGetErrorString(e));
        attr_set.mark();
    }
    install::Job job{};
    job.table = (const unsigned char *)device_table;
    job.at = install::table_plan(p->pages, p->tensors, p->segments);
    job.rotations = reinterpret_cast<const float2 *>(rotations);
    job.tensors = p->tensors; job.n_seg = p->segments; job.B = p->B; job.D = p->D; job.frame = p->frame; job.nt = p->n_temporal;
    job.tiles_cols = p->H * p->D / wa::sm100::TILE;
    job.rank = install_rank(p);
    job.status = status_address();
    job.status_mirror = status_mirror;
    if (!job.status) return fail(WA_ERR_DEVICE, "%s: no usable current device", what);
    const long long items = (long long)p->B * p->tensors * p->segments * job.tiles_cols;
    const int sms = sm_count();
    install::install_stream_kernel<<<(unsigned)(items < sms ? items : sms), install::WARPS * 32, SMEM_BYTES, (cudaStream_t)stream>>>(job);
    return check_launch(what);
}
