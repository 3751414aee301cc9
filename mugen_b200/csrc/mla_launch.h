// Host-callable launchers of the MLA kernels (internal to the library; the public surface is
// include/mugen_mla.h).
#pragma once

#include <cuda.h>

#include "mla_common.cuh"

namespace mla {

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time libcuda); nullptr where the driver has none
using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encoder()
{
    static const TensorMapEncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(p);
    }();
    return fn;
}

// rows x cols matrix of 16-bit values (0: half, 1: bfloat16), row after row: boxes of 64 values x box_rows rows, 128-byte swizzle
inline bool make_matrix_map(CUtensorMap* map, int dtype, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows)
{
    const TensorMapEncodeFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows}, estr[2] = {1, 1};
    return enc(map, dtype == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int launch_append(int dtype, const void* kv_a, void* layer_pool, uint64_t pool_slots,
                   const void* norm_w, const float* cos_sin, uint32_t cs_rows, float eps,
                   const StepMeta& m, uint32_t* status, const LaunchStream& st);

// Page-locked host memory -> device memory in pieces of 16 bytes, both 16-byte aligned.  A kernel behind it that is not launched plain
// (LaunchStream) starts before the copy is done.
int launch_fetch(const void* host, void* device, uint32_t pieces, cudaStream_t st);

void launch_write_rows(const void* src, void* layer_pool, uint64_t pool_slots, const uint32_t* table,
                       uint32_t row_begin, uint32_t n, uint32_t* status, cudaStream_t st);

// Split-KV attention, legacy tensor path (mma.sync m16n8k16): grid (segments, ceil(H/16)).
// Returns a cudaError_t-compatible code from the launch configuration.
int launch_decode_mma(int dtype, const void* q_abs, const void* layer_pool, uint32_t n_pages,
                      const StepMeta& m, float* recs, uint32_t H, uint32_t* status, cudaStream_t st);
int decode_mma_configure();   // the *_configure() functions set kernel attributes on the CURRENT device: once per device

// Split-KV attention on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM, cache tiles staged by TMA), tokens as M
// rows, `columns` (16, 32, 48 or 64) head rows as columns: grid (persistent blocks, groups of head rows).  tmaps points at the
// context's host CUtensorMap array (kMap* below), pool at the whole cache pool; uses kMapPoolV, kMapPoolSub and query_map(columns).
int launch_decode_tc5(int dtype, uint32_t columns, const void* tmaps, const void* pool, uint32_t layer0, uint32_t n_pages, const StepMeta& m,
                      float* recs, uint32_t H, uint32_t* status, cudaStream_t st);
int decode_tc5_configure(int dtype);   // sets the kernels' attributes on the current device
// columns for a launch whose largest query group has `heads` head rows
inline uint32_t decode_tc5_columns(uint32_t heads) { return heads <= 32 ? 32 : heads <= 48 ? 48 : 64; }

// Tensor maps a context builds once (mla_api.cu, make_tensor_maps), by index into its array.
enum : int {
    kMapPoolSub = 0,      // cache pool [layers][slots][576]: box 64 values x 64 tokens (one K sub-tile)
    kMapPoolV = 1,        // cache pool, whole-row view (64 values, slots, 9 chunks, layers): box 64 tokens x 2 chunks
    kMapQueries = 2,      // absorbed queries, whole-row view: box 64 head rows x 9 chunks
    kMapQueries16 = 3,    // the same with 16, 32 and 48 head rows
    kMapQueries32 = 4,
    kMapQueries48 = 5,
    kMapCount = 6
};
constexpr int query_map(uint32_t head_rows)
{
    return head_rows == 16 ? kMapQueries16 : head_rows == 32 ? kMapQueries32 : head_rows == 48 ? kMapQueries48 : kMapQueries;
}

// Split-KV attention on a pair of SMs (cluster of 2, tcgen05.mma.cta_group::2), 128-token tiles (two pages per score
// MMA series): grid (2 x persistent pairs, ceil(H/128)).  Uses kMapPoolSub, kMapPoolV, kMapQueries and the
// whole pool.
int launch_decode_tc5_pair128(int dtype, const void* tmaps, const void* pool, uint32_t layer0, uint32_t n_pages,
                              const StepMeta& m, float* recs, uint32_t H, uint32_t prefetch_tiles, const void* next_weights,
                              uint32_t next_weights_bytes, uint32_t* status, cudaStream_t st);
int decode_tc5_pair128_configure();

// Merge of the partial states + W_UV on the warp-level tensor path (the no-allocation entry point), and the merged,
// un-normalised state of every row written out (the per-GPU partial of a KV-range-sharded sequence).
void launch_merge(int dtype, const float* recs, const StepMeta& m, const void* w_uv, void* out, uint32_t H, cudaStream_t st);
int launch_export_partial(const float* recs, const StepMeta& m, float* exported, uint32_t H, cudaStream_t st);
int merge_mma_configure();

// Absorb on tcgen05; w_map: host CUtensorMap over W_UK^T of all layers,
// [layers*H*512 d][128 i], box 64 i x 128 d, 128-byte swizzle.  With kv_a != nullptr the same launch appends the step's
// new rows (launch_append's arguments) in extra blocks.  rotate_q: q arrives before its RoPE; the kernel rotates
// the last 64 dims of every head with the row's position (m.row_pos) and the cos/sin table.  append_waits: kv_a may
// have been written by the kernel launched just before this one (the append blocks then wait for it before reading).
// behind_upload: that kernel is the upload (launch_fetch) of m, and st is not plain: the weights are loaded while it runs, everything else,
// and the start of the kernels behind, waits for it.
int launch_absorb_tc5(int dtype, const void* q, const void* w_map, void* q_abs, uint32_t H, uint32_t layer0, const void* kv_a,
                      void* layer_pool, uint64_t pool_slots, const void* norm_w, const float* cos_sin, uint32_t cs_rows,
                      float eps, const StepMeta& m, bool rotate_q, bool append_waits, bool behind_upload, uint32_t sm_count, uint32_t* status, const LaunchStream& st);
int absorb_tc5_configure();

// The same merge + projection on tcgen05; w_map: host CUtensorMap over W_UV of
// all layers, [layers*H*128 outputs][512 dims], box 64 dims x 128 outputs, 128-byte swizzle.
int launch_merge_tc5(int dtype, const float* recs, const StepMeta& m, uint32_t n_parts, const void* w_map, void* out, uint32_t H,
                     uint32_t layer0, uint32_t sm_count, uint32_t* status, const LaunchStream& st);
int merge_tc5_configure();

// Dense projections C = A . W^T on tcgen05 (mla_gemm_tc5.cu), up to two weights over the same activations in one launch.
struct alignas(64) GemmWeightMaps {
    CUtensorMap box128, box64;     // W [rows][K] (or its packed form) in boxes of 64 values x 128 / 64 rows
};
struct GemmWeight {
    const CUtensorMap *map, *map64;
    uint32_t row0, N;          // first row of the weight inside the map, outputs (a multiple of 8)
    void* out;                 // DEVICE [M][N] in the storage type
};
struct GemmCall {
    const void* A = nullptr;                   // DEVICE [M][K], 16-byte aligned, or:
    const CUtensorMap* paged_map = nullptr;    // the cache pool (kMapPoolSub): A = the first M rows of a sequence, K <= 576
    const uint32_t* table = nullptr;           //   its block table (DEVICE)
    uint32_t layer = 0, n_pages = 0;
    uint32_t M = 0, K = 0;
    int n_weights = 0;
    GemmWeight w[2];
    bool packed = false;                       // weights in the layout of launch_gemm_pack (row0 = 0)
    bool residual = false;                     // out = T(float(out) + float(T(x)))
    const void* norm_w = nullptr;              // not null: A's rows go through the RMSNorm with this weight first, ...
    float eps = 0.0f;
    void* norm_out = nullptr;                  // ... rounded to the storage type here [M][K] where the kernel does not do it itself
    bool exchange_near = false;                // the projection just before this one was one that gemm_few_tc5_exchanges
};
struct GemmWorkspace {
    float* partial;            // gemm_tc5_partial_bytes(blocks)
    uint32_t* counters;        // [max_tiles], zero before the first launch
    uint32_t blocks, max_tiles;
    uint32_t clusters[4];      // gemm_few_tc5_clusters
};
// launched: kernels launched are added to it.  exchanged: whether blocks traded sums of squares (gemm_few_tc5_exchanges)
int launch_gemm_tc5(int dtype, const GemmCall& g, const GemmWorkspace& ws, uint32_t* status, const LaunchStream& st, uint64_t& launched,
                    bool* exchanged = nullptr);
// The same for few rows and weights that fit the SMs in one go, the norm included (mla_gemm_few_tc5.cu); launch_gemm_tc5 picks.
uint32_t gemm_few_tc5_cluster(const GemmCall& g, const uint32_t (&resident)[4]);
bool gemm_few_tc5_exchanges(const GemmCall& g);
int launch_gemm_few_tc5(int dtype, const GemmCall& g, uint32_t cs, uint32_t* status, const LaunchStream& st);
int gemm_few_tc5_clusters(int dtype, uint32_t (&n)[4]);
int gemm_few_tc5_configure(int dtype);
size_t gemm_tc5_partial_bytes(uint32_t blocks);
// Projection weights repacked into tiles (see the kernel file): values of the packed form, the packing itself, its maps.
size_t gemm_tc5_packed_values(uint64_t N, uint64_t K);
int launch_gemm_pack(const void* src, void* dst, uint32_t N, uint32_t K, cudaStream_t st);
bool gemm_tc5_packed_maps(GemmWeightMaps* maps, int dtype, const void* packed, uint64_t N, uint64_t K);
bool gemm_tc5_weight_maps(GemmWeightMaps* maps, int dtype, const void* W, uint64_t rows, uint64_t K);
int launch_rmsnorm_rows(int dtype, const void* x, const void* w, void* y, uint32_t rows, uint32_t N, float eps, const LaunchStream& st);
int gemm_tc5_configure(int dtype);

// Chunked prefill (mla_prefill_tc5.cu): causal flash attention of the new tokens of several sequences over expanded keys /
// values (see the file's header).
struct alignas(16) PrefillTile {       // 128 query tokens of one chunk
    uint32_t q_row;            // first row of the tile in the caller's q / out
    uint32_t n_q;              // live query tokens (1..128)
    uint32_t pos;              // cache row of the tile's first query token in its sequence (causal limit)
    uint32_t total;            // cache rows of the sequence, the chunk included
    uint32_t row0;             // first row of the sequence in the expanded keys / values (a multiple of 128)
    uint32_t rope_pos;         // global position of the first query token
    uint32_t pad[2];
};
struct PrefillCall {
    const void *q = nullptr, *kx = nullptr, *vx = nullptr;      // q [..][H][192]; kx / vx [rows][H][128]
    void* out = nullptr;                                        // [..][H][128]
    const CUtensorMap* pool_map = nullptr;                      // kMapPoolSub: the shared rope keys come from the cache pages
    const uint32_t* pages = nullptr;                            // page of every 64 expanded rows (DEVICE)
    const PrefillTile* tiles = nullptr;                         // (DEVICE)
    uint32_t n_tiles = 0, rows = 0, H = 0, layer = 0, n_pages = 0;
    const float* cos_sin = nullptr;                             // not null: q arrives before its RoPE
    uint32_t cs_rows = 0;
};
int launch_prefill_tc5(int dtype, const PrefillCall& p, uint32_t* status, cudaStream_t st);
int prefill_tc5_configure();

// One block that waits `limit_cycles` on a barrier nothing completes, raises ST_WAIT_TIMEOUT in *status, frees its
// tensor memory and returns; report[0] = 0 when the wait gave up, report[1] = cycles waited.
// stored[rank] = 1 where a block of two took the sum for complete although the other one's share never came
void launch_lost_share_selftest(long long limit_cycles, uint32_t* status, uint32_t* stored, cudaStream_t st);
void launch_wait_timeout_selftest(long long limit_cycles, uint32_t* status, uint32_t* report, cudaStream_t st);

}  // namespace mla
