// Shared definitions of the sm_100a MLA decode kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mla {

constexpr int kRank  = 512;   // kv_lora_rank: width of c_kv
constexpr int kRope  = 64;    // qk_rope_head_dim
constexpr int kNope  = 128;   // qk_nope_head_dim
constexpr int kVDim  = 128;   // v_head_dim
constexpr int kRow   = kRank + kRope;   // 576 values per latent cache row
constexpr int kQDim  = kNope + kRope;   // 192 values per head of q
constexpr int kPage  = 64;    // tokens per page
constexpr int kPart  = kRank + 2;       // floats per head of an exported partial (m, l, acc)

// Bits of the device status word (kernels set these instead of trapping).
enum : uint32_t {
    ST_BAD_SLOT      = 1u << 0,   // append: destination slot outside the pool
    ST_BAD_PAGE      = 1u << 1,   // attend: block-table entry outside the pool
    ST_WAIT_TIMEOUT  = 1u << 2,   // a bounded mbarrier wait gave up
    ST_BAD_SEGMENT   = 1u << 3,   // segment descriptor inconsistent
    ST_BAD_ALIGNMENT = 1u << 4,   // dynamic shared memory did not start on the 1 KB boundary a kernel relies on
};

// Programmatic dependent launch: a kernel launched with launch_pdl() may become resident while the
// previous kernel of the stream is still draining.  It must call grid_dependency_wait() before its
// first access to memory that any earlier kernel of the stream reads or writes (the wait returns
// once the previous grid has completed and flushed; completion is transitive because every kernel
// of the chain waits before it completes).  grid_launch_dependents() lets the next kernel's blocks
// start as soon as this kernel's blocks have all called it.  Both are no-ops in a plain launch.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Step metadata is read ahead of the wait by most kernels, so none of those may start before the upload is done and flushed.  The first
// kernel behind an upload sees to that, in one of two ways: it is launched plain, and so starts when the upload is over; or it
// reads no metadata ahead of its wait and calls grid_launch_dependents() only behind it (AbsorbArgs::behind_upload).  Either
// way every kernel further on starts with the metadata in place.
struct LaunchStream {
    cudaStream_t st;
    bool plain;
    LaunchStream(cudaStream_t s, bool is_plain = false) : st(s), plain(is_plain) {}
};
template <typename K, typename... Args>
inline cudaError_t launch_pdl(K kernel, dim3 grid, dim3 block, size_t smem, const LaunchStream& st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st.st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = st.plain ? 0 : 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename T> struct Elem;
template <> struct Elem<__half> {
    using pair = __half2;
    static __device__ __forceinline__ float to_f32(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half from_f32(float v) { return __float2half_rn(v); }
    static __device__ __forceinline__ uint32_t pack2(float a, float b) {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
};
template <> struct Elem<__nv_bfloat16> {
    using pair = __nv_bfloat162;
    static __device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 from_f32(float v) { return __float2bfloat16_rn(v); }
    static __device__ __forceinline__ uint32_t pack2(float a, float b) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
};

// One KV segment of a plan: a run of whole pages of one sequence in one layer, attended by one query group.  A query
// group is a run of consecutive step rows of the same sequence whose attend lengths grow by one per row (the new tokens
// of a sequence in a step); its rows' heads lie side by side in the absorbed queries, so the attention kernels see
// `heads` = rows x n_heads head rows over ONE stream of the pages.  32 bytes, read as two 16-byte loads.
struct alignas(16) SegDesc {
    uint32_t q_row;        // first row of the group among the plan's query rows (layer * rows + row)
    uint32_t tbl;          // index in `tables` of the segment's first page
    uint32_t n_tok;        // tokens of the segment that the group's LAST row may see (0: an empty segment)
    uint32_t layer;        // relative to the first layer of the launch
    int32_t  lim0;         // tokens of the segment that the group's first row may see (may be <= 0); row i: lim0 + i
    uint32_t heads;        // live head rows of the group
    uint32_t pad[2];
};
static_assert(sizeof(SegDesc) == 32, "read as two 16-byte loads");

__device__ __forceinline__ SegDesc load_seg_desc(const SegDesc* seg) {
    SegDesc s;
    const uint4* p = reinterpret_cast<const uint4*>(seg);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    s.q_row = a.x; s.tbl = a.y; s.n_tok = a.z; s.layer = a.w;
    s.lim0 = int32_t(b.x); s.heads = b.y;
    return s;
}
// tokens of the segment that head row vh of its group may see
__device__ __forceinline__ int seg_visible(const SegDesc& s, uint32_t vh, uint32_t H) {
    return min(int(s.n_tok), s.lim0 + int(vh / H));
}

// Where a query row's partial states are: records (seg * rec_stride + rec_off + head) for seg in [begin, end).
struct alignas(16) RowParts {
    uint32_t begin, end, rec_off, pad;
};

// Metadata of one launch series resident on the device: `layers` consecutive layers of a step, `rows` query rows in each.
struct StepMeta {
    const SegDesc* seg;             // [segs]
    const uint32_t* tables;         // physical page ids, sequence after sequence
    const uint32_t* cta_seg_begin;  // [ctas+1]  a persistent block's segments are contiguous
    const RowParts* parts;          // [layers * rows]
    const uint32_t* row_pos;        // [rows]  global position of the query row (RoPE)
    uint32_t rows, layers, segs, ctas;
    uint32_t rec_stride;            // partial-state records per segment (rows of the largest query group x n_heads)
    // The step's new tokens, in the caller's row order (kv_a rows): what the append writes.  Usually the same rows as
    // the query rows above; a step that routes long chunks to the prefill path keeps them here but not among the
    // query rows, which then carry the index of their row in the caller's q / out tensors.
    uint32_t app_rows;
    const uint32_t* app_pos;        // [app_rows]  global position (RoPE)
    const uint64_t* app_slot;       // [app_rows]  destination token slot (all ones: nothing to append)
    const uint32_t* att_row;        // [rows]  query row -> row of the caller's q / out (nullptr: the same index)
};

}  // namespace mla
