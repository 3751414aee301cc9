// C ABI of the B200 MLA decode path (see include/mugen_mla.h): context, paged latent cache,
// per-step scheduling metadata, kernel dispatch.  Host logic only; kernels live beside it.
#include "../../include/mugen_mla.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <memory>
#include <string>
#include <vector>

#include "../host/page_table.hpp"
#include "../host/rope_table.hpp"
#include "../host/upload_order.hpp"
#include "mla_launch.h"

using mugen::mla::PageTable;
using mugen::mla::Segment;

namespace {

thread_local std::string g_create_error;

constexpr int kMetaRing = 8;

// a step row: one new token (or the query-only row of a sequence that takes none)
struct RowSpec {
    uint32_t seq_index;   // index into the step's sequence list
    uint32_t attend_len;  // rows attended (0 allowed)
    uint32_t pos;         // global position of the appended token
    uint64_t slot;        // destination slot (all ones: nothing to append)
};

// Device metadata and kernel choice for a series of launches (see build_plan).
struct Plan {
    mla::StepMeta m{};
    uint32_t kernel = 0;
    uint32_t min_pages = 0, max_pages = 0;     // of any persistent worker
    bool ready = false;
};
// the plans of a step live side by side in the device metadata buffer
enum { kPlanStep = 0, kPlanRest, kPlanStack, kPlanStackTail, kPlanRegions };

// projection weights of one layer's attention block (mla_set_block_weights), all in the storage type on the device
struct BlockW {
    uint32_t embed = 0, q_lora = 0;
    void *attn_norm = nullptr, *q_a = nullptr, *q_a_norm = nullptr, *q_b = nullptr, *q = nullptr, *kv_a = nullptr, *wo = nullptr;
    mla::GemmWeightMaps q_a_map, q_b_map, q_map, kv_a_map, wo_map;
    bool set = false;
};

struct MetaBuf {
    char* host = nullptr;       // pinned
    cudaEvent_t done = nullptr;
    bool in_flight = false;
};

}  // namespace

struct mla_ctx {
    mla_config cfg{};
    int sm_count = 0;
    uint32_t kernel = MLA_KERNEL_MMA;
    std::unique_ptr<PageTable> pt;
    std::string err;
    uint64_t launches = 0;

    char* pool = nullptr;           // [layers][n_pages*64][576] elements
    uint64_t pool_slots = 0;        // token slots per layer
    // weights of all layers side by side, so that one tensor map (and one launch) reaches any run of layers
    char* w_uk = nullptr;            // [layers][H][512][128]: W_UK transposed per head
    char* w_uk_rows = nullptr;       // [layers][H*128][512]: as registered, the prefill path expands keys with it
    char* w_uv = nullptr;            // [layers][H*128][512]
    char* norm = nullptr;            // [layers][512]
    std::vector<char> layer_set;     // weights registered
    alignas(64) CUtensorMap w_uk_map, w_uv_map;
    mla::GemmWeightMaps w_uk_rows_maps, w_uv_maps;       // the same weights for the prefill expansion
    std::vector<BlockW> blocks;
    // workspaces of the block projections, grown on demand: normalised hidden state, q_a,
    // and the block's q, kv_a and attention output when the library owns them (mla_step_block: one allocation)
    void *blk_hidden2 = nullptr, *blk_qa = nullptr, *blk_rows = nullptr;
    size_t blk_hidden2_cap = 0, blk_qa_cap = 0, blk_rows_cap = 0;
    mla::GemmWorkspace gemm_ws{};    // partial tiles and counters of the projections
    float* cos_sin = nullptr;       // device [max positions][64]
    uint32_t cs_rows = 0;           // positions filled so far
    uint32_t cs_cap = 0;

    void* q_abs = nullptr;          // [ws_rows][H][576]
    float* recs = nullptr;          // [rec_cap][514]
    uint32_t ws_rows = 0;           // query rows a launch series may hold: max_rows, or a group of layers of fewer rows
    size_t rec_cap = 0;
    uint32_t* status_dev = nullptr;
    // tensor maps of the tcgen05 attention kernels (make_tensor_maps; indices mla::kMap*)
    alignas(64) CUtensorMap tmaps[mla::kMapCount];

    // metadata upload ring
    MetaBuf ring[kMetaRing];
    int ring_next = 0;
    size_t meta_cap = 0;
    char* meta_dev = nullptr;       // [kPlanRegions][meta_cap]
    char* meta_host = nullptr;      // [kMetaRing][meta_cap], page-locked
    mugen::mla::UploadOrder<kPlanRegions> uploads;       // those that no kernel has followed yet (launch_stream)
    // Plans of the open step.  `plan`: every new token is a decode-style query row, one layer at a time.  A step that holds
    // prefill chunks (sequences taking >= kPrefillMin new tokens) also has `plan_rest`: its query rows are the step's OTHER
    // rows, the chunks go through the expanded-form prefill kernels (run_layer); the explicit per-layer calls
    // (mla_step_append / _attend / _attend_partial) keep using the first.  mla_step_begin makes and uploads these two on its
    // own stream, so that the calls behind it only launch: on any stream ordered behind it, and under capture.
    // `stack` / `stack_tail`: groups of layers of one mla_step_layers call, made and uploaded by the call that needs them.
    Plan plan, plan_rest, stack, stack_tail;
    bool has_chunks = false;
    std::vector<RowSpec> rows;       // of the open step
    struct Chunk { uint32_t seq_index, q_row0, n_new, start, base_pos; };
    std::vector<Chunk> chunks;
    // Chunks whose expanded keys and values share the workspace and the launches: `rows` expanded rows (every sequence padded
    // to 128), their pages and query tiles in the upload of plan_rest
    struct ChunkGroup { uint32_t rows, n_tiles; const uint32_t* pages; const mla::PrefillTile* tiles; };
    std::vector<ChunkGroup> chunk_groups;
    uint32_t step_rows = 0;          // rows of the step in the caller's q / kv_a / out tensors
    // prefill workspace, grown on demand: expanded keys, then values
    void* pf_kv = nullptr;
    size_t pf_kv_cap = 0;

    // pages of the last planned step per persistent worker (mla_step_balance)
    uint32_t plan_workers = 0, plan_min_pages = 0, plan_max_pages = 0;
    uint32_t step_new_rows = 0;     // rows the open step appends (a KV-range shard that does not own the tail has none)

    // step state
    bool in_step = false;
    std::vector<uint32_t> step_seqs, step_nnew;

    // optional per-launch timing of the attention kernel
    bool q_rope_in_kernel = false;  // queries arrive before their RoPE (mla_set_q_rope)
    bool profiling = false;
    uint32_t prof_stride = 1, prof_seq = 0;     // every prof_stride-th attention launch is timed
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> prof_events;
    size_t prof_used = 0;

    // host-buffer entry point staging
    void *h_in = nullptr, *h_out = nullptr, *d_kv = nullptr, *d_q = nullptr, *d_out = nullptr;
    // page-locked callers: copies run on two streams of their own so that layer L+1's inputs and layer L-1's
    // outputs move while layer L computes; one event triple per layer orders copy-in -> compute -> copy-out
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    struct HostEv { cudaEvent_t in = nullptr, compute = nullptr, out = nullptr; bool used = false, pending = false; };
    std::vector<HostEv> host_ev;
};

namespace {

int fail(mla_ctx* c, int code, std::string msg)
{
    if (c) c->err = std::move(msg);
    else g_create_error = std::move(msg);
    return code;
}

#define CU_TRY(c, expr)                                                                           \
    do {                                                                                          \
        cudaError_t e__ = (expr);                                                                 \
        if (e__ != cudaSuccess)                                                                   \
            return fail((c), MLA_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e__)); \
    } while (0)

// Every entry point that launches or copies makes the context's device current first: a host thread that
// drives several contexts (one per GPU) would otherwise launch on whichever device it used last.
#define USE_DEVICE(c) CU_TRY((c), cudaSetDevice((c)->cfg.device))

int pt_code(mla_ctx* c, int e)
{
    if (e == mugen::mla::PT_OK) return MLA_OK;
    c->err = c->pt->error();
    return e;   // PT_* values equal the MLA_ERR_* values they stand for
}

// Names a stream whatever handle it goes by: the default stream has two handles, the per-thread one is another stream in every
// thread.  (cudaStreamGetId would tell them apart too, but a call of it ends a capture.)
uint64_t stream_key(cudaStream_t st)
{
    static thread_local char this_thread;
    if (st == cudaStreamPerThread) return uint64_t(reinterpret_cast<uintptr_t>(&this_thread));
    return st == cudaStreamLegacy ? 0 : uint64_t(reinterpret_cast<uintptr_t>(st));
}

bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// Sequences that take at least this many new tokens in a step go through the prefill kernels.
constexpr uint32_t kPrefillMin = 64;
// Most query rows and bytes of absorbed queries of a group of layers (mla_step_layers).  Queries and partial states of a group this
// large do not stay in L2 between its launches, and that costs less than the start, the drain and the uneven last segments of more
// launches: 1024 rows and 48 MB against these, 27 layers of 16 heads, 16 sequences x 5 rows 321 -> 305 us, 64 x 8 rows 1312 -> 969,
// 40 single rows 201 -> 176, 128 of 2000 tokens 1470 -> 1415; 6 layers of 64 heads x 120 ragged sequences 334 -> 287; 3 layers of 128
// heads x 128 837 -> 830; slower in one of 27 shapes (4 layers of 128 heads, 30 sequences x 4 rows: 466 -> 468).  160 MB give no more.
constexpr uint64_t kGroupRows = 4096, kGroupBytes = 96ull << 20;
// The smaller ones where pool and weights leave less than kRoomForGroups of the device: what the caller allocates beside them has the
// room that it had.  Which ones a context has goes by its configuration, so that a program cuts KV ranges alike, and gives the same
// bits, whatever else is on the device; but where the larger workspace would leave less than kLeftByGroups, and a later step could fail
// for want of it, the smaller one is taken.
constexpr uint64_t kSmallGroupRows = 1024, kSmallGroupBytes = 48ull << 20;
constexpr size_t kRoomForGroups = 16ull << 30, kLeftByGroups = 1ull << 30;
// Expanded keys and values of the chunks that share a launch (a chunk that needs more has one of its own).
constexpr uint64_t kExpandBytes = 256ull << 20;

inline float half_bits_to_f32(uint16_t h) { return __half2float(__ushort_as_half(h)); }
inline uint16_t f32_to_half_bits(float f) { return __half_as_ushort(__float2half_rn(f)); }
inline uint16_t f32_to_bf16_bits(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }

// Decodes (n_rows x 512) weights of GGML type `w_type` into the context storage dtype.
int decode_weights(mla_ctx* c, const void* w, uint32_t w_type, size_t n_rows, std::vector<uint16_t>& out)
{
    const size_t n = n_rows * mla::kRank;
    out.resize(n);
    const bool to_half = c->cfg.dtype == MLA_DTYPE_F16;
    auto put = [&](size_t i, float v) { out[i] = to_half ? f32_to_half_bits(v) : f32_to_bf16_bits(v); };
    if (w_type == MLA_W_F16) {
        const auto* s = static_cast<const uint16_t*>(w);
        if (to_half) std::memcpy(out.data(), s, n * 2);
        else for (size_t i = 0; i < n; i++) put(i, half_bits_to_f32(s[i]));
    } else if (w_type == MLA_W_BF16) {
        const auto* s = static_cast<const uint16_t*>(w);
        if (!to_half) std::memcpy(out.data(), s, n * 2);
        else for (size_t i = 0; i < n; i++) {
            const uint32_t u = uint32_t(s[i]) << 16;
            float f;
            std::memcpy(&f, &u, 4);
            put(i, f);
        }
    } else if (w_type == MLA_W_Q8_0) {
        const auto* s = static_cast<const uint8_t*>(w);
        const size_t nb = n / 32;
        for (size_t b = 0; b < nb; b++) {
            const uint8_t* blk = s + b * 34;
            uint16_t d;
            std::memcpy(&d, blk, 2);
            const float sc = half_bits_to_f32(d);
            for (int j = 0; j < 32; j++) put(b * 32 + j, sc * float(int8_t(blk[2 + j])));
        }
    } else if (w_type == MLA_W_Q4_0) {
        const auto* s = static_cast<const uint8_t*>(w);
        const size_t nb = n / 32;
        for (size_t b = 0; b < nb; b++) {
            const uint8_t* blk = s + b * 18;
            uint16_t d;
            std::memcpy(&d, blk, 2);
            const float sc = half_bits_to_f32(d);
            for (int j = 0; j < 16; j++) {
                put(b * 32 + j, float(int(blk[2 + j] & 0x0F) - 8) * sc);
                put(b * 32 + j + 16, float(int(blk[2 + j] >> 4) - 8) * sc);
            }
        }
    } else {
        return fail(c, MLA_ERR_UNSUPPORTED, "weight type " + std::to_string(w_type) +
                                                " is not one of F16, BF16, Q8_0, Q4_0");
    }
    return MLA_OK;
}

int ensure_rope_rows(mla_ctx* c, uint32_t upto, cudaStream_t st)
{
    if (upto <= c->cs_rows) return MLA_OK;
    if (upto > c->cs_cap)
        return fail(c, MLA_ERR_CAPACITY, "position " + std::to_string(upto - 1) +
                                             " beyond the rotary table capacity " + std::to_string(c->cs_cap));
    // grow in chunks so that a decode loop does not upload one row per step
    uint32_t target = std::min<uint32_t>(c->cs_cap, std::max<uint32_t>(upto, c->cs_rows + 4096));
    std::vector<float> rows(size_t(target - c->cs_rows) * mla::kRope);
    mugen::mla::fill_rope_rows(rows.data(), c->cs_rows, target, c->cfg.rope_scaling_factor,
                               c->cfg.rope_original_ctx, c->cfg.rope_theta);
    CU_TRY(c, cudaMemcpyAsync(c->cos_sin + size_t(c->cs_rows) * mla::kRope, rows.data(),
                              rows.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    CU_TRY(c, cudaStreamSynchronize(st));   // `rows` is pageable and about to go away
    c->cs_rows = target;
    return MLA_OK;
}

uint32_t workers_of(const mla_ctx* c, uint32_t kernel, uint32_t heads)
{
    if (kernel == MLA_KERNEL_TCGEN05_PAIR128) return std::max<uint32_t>(1, (c->sm_count / 2) / ((heads + 127) / 128));
    if (kernel == MLA_KERNEL_TCGEN05) return std::max<uint32_t>(1, c->sm_count / ((heads + 63) / 64));
    if (kernel == MLA_KERNEL_TCGEN05_T16) return std::max<uint32_t>(1, c->sm_count / ((heads + 15) / 16));
    return std::max<uint32_t>(1, c->sm_count * 2 / ((heads + 15) / 16));
}

// The attention kernel for `heads` head rows over one stream of the cache.  More than 64 rows go to the SM-pair kernel,
// which streams the cache once for 128 of them at the same rate whether all are live or not (a second pass of the 64-column
// kernel costs more than the padding); up to 64 take the transposed form with 16 columns (T16) or as many as the rows need.
uint32_t kernel_for(const mla_ctx* c, uint32_t heads)
{
    if (c->cfg.kernel != MLA_KERNEL_AUTO) return c->cfg.kernel;
    return (heads > 64 && c->sm_count % 2 == 0) ? uint32_t(MLA_KERNEL_TCGEN05_PAIR128)
         : heads > 16 ? uint32_t(MLA_KERNEL_TCGEN05) : uint32_t(MLA_KERNEL_TCGEN05_T16);
}

// Head rows that one stream of the cache can serve: what a query group may fill.
uint32_t group_heads(const mla_ctx* c)
{
    switch (c->cfg.kernel) {
    case MLA_KERNEL_AUTO: return c->sm_count % 2 == 0 ? 128 : 64;
    case MLA_KERNEL_TCGEN05_PAIR128: return 128;
    case MLA_KERNEL_TCGEN05: return 64;
    case MLA_KERNEL_TCGEN05_T16: return 16;
    default: return 1;
    }
}

size_t meta_capacity(const mla_ctx* c)
{
    const size_t R = c->cfg.max_rows, V = c->ws_rows, W = size_t(c->sm_count) * 2;
    const size_t max_pages_per_seq = (size_t(c->cfg.max_seq_len) + mla::kPage - 1) / mla::kPage;
    const size_t tbl_entries = std::min<size_t>(size_t(c->cfg.max_seqs) * max_pages_per_seq, c->cfg.n_pages) + 4;
    return align16(R * 8) + 3 * align16(R * 4) + align16(tbl_entries * 4) + align16((W + V) * sizeof(mla::SegDesc)) +
           align16(V * sizeof(mla::RowParts)) + align16((W + 1) * 4) +
           align16((tbl_entries + 2 * size_t(c->cfg.max_seqs)) * 4) +                                        // chunks: pages padded to 128 rows,
           align16((R / 128 + c->cfg.max_seqs + 1) * sizeof(mla::PrefillTile)) + 256;                        // and query tiles
}

// what the prefill kernels of a step read (rest_plan)
struct ChunkMeta {
    std::vector<uint32_t> pages;             // page of every 64 expanded rows
    std::vector<mla::PrefillTile> tiles;
    struct Group { uint32_t rows, page0, tile0, n_tiles; };
    std::vector<Group> groups;
};

// Plans `layers` identical layers of query rows over the persistent attention workers, packs the metadata of the launch
// series (new rows to append, query rows, block tables, segments) and uploads it through the page-locked ring into region
// `region` of the device buffer, behind earlier work of `st`.
//   app      the step's new rows, in the caller's row order (what the append writes)
//   query    the query rows; nullptr: app.  att_row: their rows in the caller's tensors (with query only)
//   layers   0: no attention (append or row copy only)
int build_plan(mla_ctx* c, Plan& plan, int region, const std::vector<uint32_t>& seq_ids, const std::vector<RowSpec>& app,
               const std::vector<RowSpec>* query, const std::vector<uint32_t>* att_row, uint32_t layers, cudaStream_t st,
               const ChunkMeta* chunks = nullptr)
{
    const std::vector<RowSpec>& rows = query ? *query : app;
    const uint32_t A = uint32_t(app.size()), R = layers ? uint32_t(rows.size()) : 0, S = uint32_t(seq_ids.size()), H = c->cfg.n_heads;
    plan = Plan{};
    if (uint64_t(R) * layers > c->ws_rows)
        return fail(c, MLA_ERR_CAPACITY, "step needs " + std::to_string(uint64_t(R) * layers) + " query rows, the workspace holds " +
                                             std::to_string(c->ws_rows));
    // block tables, sequence after sequence
    size_t tbl_total = 0;
    std::vector<uint32_t> tbl_off(S);
    for (uint32_t i = 0; i < S; i++) {
        tbl_off[i] = uint32_t(tbl_total);
        tbl_total += c->pt->seq(seq_ids[i])->pages.size();
    }
    std::vector<Segment> segs;
    std::vector<uint32_t> grp_seg_begin{0}, cta_seg_begin{0};
    // Query groups: the new tokens of a sequence are consecutive rows whose attend lengths grow by one, and with few heads
    // several of them fit the head rows of one stream of the cache (5 rows of 16 heads: one pass instead of five).
    struct Group { uint32_t row, n; };
    std::vector<Group> groups;
    uint32_t k = 1;                  // rows of the largest group
    auto follows = [&](uint32_t r) {
        return rows[r].seq_index == rows[r - 1].seq_index && rows[r].attend_len == rows[r - 1].attend_len + 1 && rows[r - 1].attend_len > 0;
    };
    if (R) {
        uint32_t longest = 1;
        for (uint32_t r = 1, run = 1; r < R; r++) {
            run = follows(r) ? run + 1 : 1;
            longest = std::max(longest, run);
        }
        for (uint32_t cap = std::max(1u, std::min(group_heads(c) / H, longest));; cap = cap / 2) {
            const uint32_t n_groups = (longest + cap - 1) / cap;
            k = (longest + n_groups - 1) / n_groups;
            groups.clear();
            for (uint32_t r = 0; r < R; r++) {
                if (r && follows(r) && groups.back().n < k) groups.back().n++;
                else groups.push_back({r, 1});
            }
            const uint32_t NG = uint32_t(groups.size());
            plan.kernel = kernel_for(c, k * H);
            const uint32_t workers = workers_of(c, plan.kernel, k * H);
            if ((size_t(workers) + size_t(NG) * layers) * k * H > c->rec_cap && k > 1) continue;     // many single rows beside a long run
            std::vector<uint32_t> lens(size_t(NG) * layers);
            for (uint32_t g = 0; g < NG; g++) lens[g] = rows[groups[g].row + groups[g].n - 1].attend_len;
            for (uint32_t l = 1; l < layers; l++) std::copy(lens.begin(), lens.begin() + NG, lens.begin() + size_t(l) * NG);
            if (plan.kernel == MLA_KERNEL_TCGEN05_PAIR128)
                // a worker pays a few tiles' time per segment it starts (queries, pipeline fill, state drain)
                mugen::mla::plan_min_makespan(lens, mla::kPage, workers, segs, grp_seg_begin, cta_seg_begin, 2u, 3u);
            else       // in pages; three where 32 to 64 columns of queries and states come and go (8 layers of 64 heads x 8 sequences of up to 3000
                       // tokens 55.7 -> 54.5 us, host entry 16 sequences 313.9 -> 305.2, others 0.5 to 1 %; four: 53.9, 308.7)
                mugen::mla::plan_min_makespan(lens, mla::kPage, workers, segs, grp_seg_begin, cta_seg_begin, 1u,
                                              plan.kernel == MLA_KERNEL_TCGEN05 ? 3u : 2u);
            break;
        }
        if (segs.size() * k * H > c->rec_cap)
            return fail(c, MLA_ERR_CAPACITY, "step needs " + std::to_string(segs.size()) + " KV segments, more than the workspace holds");
    }
    const uint32_t NG = uint32_t(groups.size());
    const uint32_t G = uint32_t(segs.size()), W = uint32_t(cta_seg_begin.size()) - 1;
    if (layers) {
        plan.min_pages = R && W ? ~0u : 0u;
        for (uint32_t w = 0; w < W; w++) {
            uint32_t pages = 0;
            for (uint32_t g = cta_seg_begin[w]; g < cta_seg_begin[w + 1]; g++) pages += segs[g].page_end - segs[g].page_begin;
            plan.min_pages = std::min(plan.min_pages, pages);
            plan.max_pages = std::max(plan.max_pages, pages);
        }
        if (region == kPlanStep || region == kPlanRest) {      // what mla_step_balance reports: one layer of the step
            c->plan_workers = std::max(W, 1u);
            c->plan_min_pages = plan.min_pages;
            c->plan_max_pages = plan.max_pages;
        }
    }
    // layout
    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align16(off + bytes); return o; };
    const size_t o_slot = take(size_t(A) * 8), o_apos = take(size_t(A) * 4), o_tbl = take(tbl_total * 4),
                 o_pos = query ? take(size_t(R) * 4) : o_apos, o_att = take(att_row ? size_t(R) * 4 : 0),
                 o_seg = take(size_t(G) * sizeof(mla::SegDesc)), o_parts = take(size_t(R) * layers * sizeof(mla::RowParts)),
                 o_csb = take(size_t(W + 1) * 4), o_cpg = take(chunks ? chunks->pages.size() * 4 : 0),
                 o_ctl = take(chunks ? chunks->tiles.size() * sizeof(mla::PrefillTile) : 0);
    if (off > c->meta_cap)
        return fail(c, MLA_ERR_CAPACITY, "step metadata (" + std::to_string(off) + " B) exceeds the buffer (" +
                                             std::to_string(c->meta_cap) + " B)");
    MetaBuf& mb = c->ring[c->ring_next];
    c->ring_next = (c->ring_next + 1) % kMetaRing;
    if (mb.in_flight) {
        CU_TRY(c, cudaEventSynchronize(mb.done));
        mb.in_flight = false;
    }
    char* h = mb.host;
    auto* p_slot = reinterpret_cast<uint64_t*>(h + o_slot);
    auto* p_apos = reinterpret_cast<uint32_t*>(h + o_apos);
    for (uint32_t r = 0; r < A; r++) { p_slot[r] = app[r].slot; p_apos[r] = app[r].pos; }
    auto* p_tbl = reinterpret_cast<uint32_t*>(h + o_tbl);
    for (uint32_t i = 0; i < S; i++) {
        const auto& pg = c->pt->seq(seq_ids[i])->pages;
        std::memcpy(p_tbl + tbl_off[i], pg.data(), pg.size() * 4);
    }
    if (query) {
        auto* p_pos = reinterpret_cast<uint32_t*>(h + o_pos);
        for (uint32_t r = 0; r < R; r++) p_pos[r] = rows[r].pos;
    }
    if (att_row) std::memcpy(h + o_att, att_row->data(), size_t(R) * 4);
    auto* p_seg = reinterpret_cast<mla::SegDesc*>(h + o_seg);
    for (uint32_t g = 0; g < G; g++) {
        const uint32_t l = segs[g].row / NG;
        const Group& gr = groups[segs[g].row % NG];
        const RowSpec &first = rows[gr.row], &last = rows[gr.row + gr.n - 1];
        const uint32_t tok0 = segs[g].page_begin * mla::kPage, tok1 = std::min(last.attend_len, segs[g].page_end * uint32_t(mla::kPage));
        const uint32_t n_tok = tok1 > tok0 ? tok1 - tok0 : 0;
        p_seg[g] = mla::SegDesc{l * R + gr.row, tbl_off[first.seq_index] + segs[g].page_begin, n_tok, l,
                                int32_t(first.attend_len) - int32_t(tok0), gr.n * H, {0, 0}};
    }
    auto* p_parts = reinterpret_cast<mla::RowParts*>(h + o_parts);
    for (uint32_t l = 0; l < layers; l++)
        for (uint32_t g = 0; g < NG; g++) {
            const uint32_t v = l * NG + g;
            for (uint32_t i = 0; i < groups[g].n; i++) p_parts[l * R + groups[g].row + i] = mla::RowParts{grp_seg_begin[v], grp_seg_begin[v + 1], i * H, 0};
        }
    std::memcpy(h + o_csb, cta_seg_begin.data(), size_t(W + 1) * 4);
    char* d = c->meta_dev + size_t(region) * c->meta_cap;
    if (chunks) {
        std::memcpy(h + o_cpg, chunks->pages.data(), chunks->pages.size() * 4);
        std::memcpy(h + o_ctl, chunks->tiles.data(), chunks->tiles.size() * sizeof(mla::PrefillTile));
        c->chunk_groups.clear();
        for (const auto& g : chunks->groups)
            c->chunk_groups.push_back({g.rows, g.n_tiles, reinterpret_cast<const uint32_t*>(d + o_cpg) + g.page0,
                                       reinterpret_cast<const mla::PrefillTile*>(d + o_ctl) + g.tile0});
    }
    if (capturing(st)) {
        CU_TRY(c, cudaMemcpyAsync(d, h, off, cudaMemcpyHostToDevice, st));       // a graph's kernels follow a copy without further care
    } else {
        CU_TRY(c, cudaError_t(mla::launch_fetch(h, d, uint32_t(off / 16), st)));
        c->uploads.uploaded(size_t(region), stream_key(st));
    }
    CU_TRY(c, cudaEventRecord(mb.done, st));
    mb.in_flight = true;

    mla::StepMeta& m = plan.m;
    m.seg = reinterpret_cast<const mla::SegDesc*>(d + o_seg);
    m.tables = reinterpret_cast<const uint32_t*>(d + o_tbl);
    m.cta_seg_begin = reinterpret_cast<const uint32_t*>(d + o_csb);
    m.parts = reinterpret_cast<const mla::RowParts*>(d + o_parts);
    m.row_pos = reinterpret_cast<const uint32_t*>(d + o_pos);
    m.rows = R;
    m.layers = layers ? layers : 1;
    m.segs = G;
    m.ctas = W;
    m.rec_stride = k * H;
    m.app_rows = A;
    m.app_pos = reinterpret_cast<const uint32_t*>(d + o_apos);
    m.app_slot = reinterpret_cast<const uint64_t*>(d + o_slot);
    m.att_row = att_row ? reinterpret_cast<const uint32_t*>(d + o_att) : nullptr;
    plan.ready = true;
    return MLA_OK;
}

// the plan of a step with prefill chunks: its decode-style rows are the query rows, all its rows are appended
int rest_plan(mla_ctx* c, cudaStream_t st)
{
    std::vector<RowSpec> rest;
    std::vector<uint32_t> att_row;
    uint32_t r = 0;
    for (uint32_t i = 0; i < c->step_nnew.size(); i++) {
        const uint32_t cnt = std::max<uint32_t>(c->step_nnew[i], 1);
        if (c->step_nnew[i] < kPrefillMin)
            for (uint32_t t = 0; t < cnt; t++) { rest.push_back(c->rows[r + t]); att_row.push_back(r + t); }
        r += cnt;
    }
    // the chunks' expanded rows and query tiles, as many chunks per group as the workspace bound allows
    ChunkMeta cm;
    const uint64_t row_bytes = uint64_t(c->cfg.n_heads) * (mla::kNope + mla::kVDim) * 2;
    for (const auto& ch : c->chunks) {
        const uint32_t total = ch.start + ch.n_new, padded = (total + 127) / 128 * 128;
        if (cm.groups.empty() || (cm.groups.back().rows + padded) * row_bytes > kExpandBytes) cm.groups.push_back({0, uint32_t(cm.pages.size()), uint32_t(cm.tiles.size()), 0});
        auto& g = cm.groups.back();
        const auto& pg = c->pt->seq(c->step_seqs[ch.seq_index])->pages;
        const uint32_t n_pages = (total + mla::kPage - 1) / mla::kPage;
        for (uint32_t i = 0; i < padded / mla::kPage; i++) cm.pages.push_back(pg[std::min(i, n_pages - 1)]);   // padding: the last page again
        for (uint32_t t = 0; t < ch.n_new; t += 128)
            cm.tiles.push_back({ch.q_row0 + t, std::min(128u, ch.n_new - t), ch.start + t, total, g.rows, ch.base_pos + ch.start + t, {0, 0}});
        g.rows += padded;
        g.n_tiles = uint32_t(cm.tiles.size()) - g.tile0;
    }
    for (auto& g : cm.groups)           // the tiles that see the most keys first
        std::stable_sort(cm.tiles.begin() + g.tile0, cm.tiles.begin() + g.tile0 + g.n_tiles,
                         [](const mla::PrefillTile& a, const mla::PrefillTile& b) { return a.pos > b.pos; });
    return build_plan(c, c->plan_rest, kPlanRest, c->step_seqs, c->rows, &rest, &att_row, 1, st, &cm);
}

// The stream of a launch that may be the first behind an upload of metadata.  A captured launch keeps its overlap: a graph starts when
// what lies ahead of it in its stream is done, and inside a capture uploads are copies (build_plan).
mla::LaunchStream launch_stream(const mla_ctx* c, cudaStream_t st)
{
    return mla::LaunchStream(st, c->uploads.open(stream_key(st)) && !capturing(st));
}
// ... and once it is in the stream (a captured launch is not)
void launched(mla_ctx* c, cudaStream_t st) { if (c->uploads.open(stream_key(st)) && !capturing(st)) c->uploads.followed(stream_key(st)); }

char* layer_pool(mla_ctx* c, uint32_t layer)
{
    return c->pool + size_t(layer) * c->pool_slots * mla::kRow * 2;
}

int check_layer(mla_ctx* c, uint32_t layer, bool need_weights)
{
    if (layer >= c->cfg.n_layers) return fail(c, MLA_ERR_INVALID, "layer " + std::to_string(layer) + " out of range");
    if (need_weights && !c->layer_set[layer])
        return fail(c, MLA_ERR_STATE, "weights of layer " + std::to_string(layer) + " were never registered");
    return MLA_OK;
}

// one layer's slices of the weights
size_t weight_bytes(const mla_ctx* c) { return size_t(c->cfg.n_heads) * mla::kNope * mla::kRank * 2; }
char* layer_norm(mla_ctx* c, uint32_t layer) { return c->norm + size_t(layer) * mla::kRank * 2; }

int run_append(mla_ctx* c, uint32_t layer, const void* kv_a, const mla::StepMeta& m, cudaStream_t st)
{
    const int e = mla::launch_append(int(c->cfg.dtype), kv_a, layer_pool(c, layer), c->pool_slots, layer_norm(c, layer),
                                     c->cos_sin, c->cs_rows, c->cfg.rms_norm_eps, m, c->status_dev, launch_stream(c, st));
    if (e != 0) return fail(c, MLA_ERR_CUDA, std::string("append launch: ") + cudaGetErrorString(cudaError_t(e)));
    if (m.app_rows) launched(c, st);
    c->launches += m.app_rows ? 1 : 0;
    return MLA_OK;
}

// absorb -> split-KV attention -> merge (+ W_UV, or export of the merged partial state) of the plan's layers from `layer` on
// With fused_kv_a the absorb launch also appends the step's new rows (the caller then skips run_append).
// own_upload: the caller has just uploaded p, and nobody else can have launched anything on st since; the absorb then starts before the
// upload is over, and holds back the kernels behind it until it is.
int run_attend(mla_ctx* c, uint32_t layer, const void* q, void* out, float* exported, const Plan& p, cudaStream_t st,
               const void* fused_kv_a = nullptr, bool kv_a_settled = false, bool own_upload = false)
{
    const mla::StepMeta& m = p.m;
    if (m.rows == 0) return MLA_OK;
    const uint32_t H = c->cfg.n_heads;
    const int dt = int(c->cfg.dtype);
    const int ae = mla::launch_absorb_tc5(dt, q, &c->w_uk_map, c->q_abs, H, layer, fused_kv_a, layer_pool(c, layer), c->pool_slots,
                                          layer_norm(c, layer), c->cos_sin, c->cs_rows, c->cfg.rms_norm_eps, m, c->q_rope_in_kernel,
                                          !kv_a_settled, own_upload, uint32_t(c->sm_count), c->status_dev,
                                          own_upload ? mla::LaunchStream(st) : launch_stream(c, st));
    if (ae != 0) return fail(c, MLA_ERR_CUDA, std::string("absorb launch: ") + cudaGetErrorString(cudaError_t(ae)));
    launched(c, st);
    int e;
    const bool timed = c->profiling && c->prof_used < c->prof_events.size() && (c->prof_seq++ % c->prof_stride) == 0;
    if (timed) CU_TRY(c, cudaEventRecord(c->prof_events[c->prof_used].first, st));
    // the W_UK the stream will want next: the following layer's (the first layer's after the last: the next step)
    const uint32_t nl = (layer + m.layers) % c->cfg.n_layers;
    const void* next_w = c->layer_set[nl] ? c->w_uk + nl * weight_bytes(c) : nullptr;
    if (p.kernel == MLA_KERNEL_TCGEN05_PAIR128)
        // short work lists (few sequences on this GPU) are bound by load latency, not bandwidth: prefetch one tile ahead
        e = mla::launch_decode_tc5_pair128(dt, c->tmaps, c->pool, layer, c->cfg.n_pages, m, c->recs, H, p.max_pages <= 64 ? 1u : 0u,
                                           next_w, next_w ? uint32_t(weight_bytes(c)) : 0u, c->status_dev, st);
    else if (p.kernel == MLA_KERNEL_TCGEN05)
        e = mla::launch_decode_tc5(dt, mla::decode_tc5_columns(m.rec_stride), c->tmaps, c->pool, layer, c->cfg.n_pages, m, c->recs, H, c->status_dev, st);
    else if (p.kernel == MLA_KERNEL_TCGEN05_T16)
        e = mla::launch_decode_tc5(dt, 16, c->tmaps, c->pool, layer, c->cfg.n_pages, m, c->recs, H, c->status_dev, st);
    else
        e = mla::launch_decode_mma(dt, c->q_abs, layer_pool(c, layer), c->cfg.n_pages, m, c->recs, H, c->status_dev, st);
    if (e != 0) return fail(c, MLA_ERR_CUDA, std::string("attention launch: ") + cudaGetErrorString(cudaError_t(e)));
    if (timed) CU_TRY(c, cudaEventRecord(c->prof_events[c->prof_used++].second, st));
    if (exported) {
        e = mla::launch_export_partial(c->recs, m, exported, H, st);
    } else {
        e = mla::launch_merge_tc5(dt, c->recs, m, 0, &c->w_uv_map, out, H, layer, uint32_t(c->sm_count), c->status_dev, st);
    }
    if (e != 0) return fail(c, MLA_ERR_CUDA, std::string("merge launch: ") + cudaGetErrorString(cudaError_t(e)));
    c->launches += 3;
    return MLA_OK;
}

// slack: a quarter more, for a buffer whose need grows from step to step
int grow(mla_ctx* c, void** p, size_t* cap, size_t bytes, bool slack = false)
{
    if (bytes <= *cap) return MLA_OK;
    if (slack) bytes += bytes / 4;
    CU_TRY(c, cudaDeviceSynchronize());          // an earlier launch may still use the smaller buffer
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    CU_TRY(c, cudaMalloc(p, bytes));
    *cap = bytes;
    return MLA_OK;
}

// partial tiles and counters of the projections: contexts that register no block and take no prompt chunk have none
int ensure_gemm_workspace(mla_ctx* c)
{
    mla::GemmWorkspace& w = c->gemm_ws;
    if (w.counters) return MLA_OK;
    w.blocks = uint32_t(c->sm_count);
    w.max_tiles = 16 * w.blocks;
    CU_TRY(c, cudaError_t(mla::gemm_few_tc5_clusters(int(c->cfg.dtype), w.clusters)));
    if (!w.partial) CU_TRY(c, cudaMalloc(&w.partial, mla::gemm_tc5_partial_bytes(w.blocks)));
    uint32_t* counters = nullptr;
    CU_TRY(c, cudaMalloc(&counters, w.max_tiles * 4));
    cudaError_t e = cudaMemset(counters, 0, w.max_tiles * 4);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();       // the launches that count on zeros are on other streams
    if (e != cudaSuccess) cudaFree(counters);
    CU_TRY(c, e);
    w.counters = counters;
    return MLA_OK;
}

mla::GemmWeight gemm_weight(const mla::GemmWeightMaps& maps, uint32_t n_outputs, void* out, uint32_t row0 = 0)
{
    return mla::GemmWeight{&maps.box128, &maps.box64, row0, n_outputs, out};
}

// The chunks of the open step: expand each sequence's latent rows (the chunk's own were appended by the launch before) into
// per-head keys and values with W_UK / W_UV, straight from the cache pages, and run causal flash attention of the chunks'
// queries over them.  Reference semantics: src/core/model/transformer.cpp:1263-1337.
int run_chunks(mla_ctx* c, uint32_t layer, const void* q, void* out, cudaStream_t st)
{
    const uint32_t H = c->cfg.n_heads;
    const int dt = int(c->cfg.dtype);
    if (int e = ensure_gemm_workspace(c)) return e;
    for (const auto& g : c->chunk_groups) {
        const size_t k_bytes = size_t(g.rows) * H * mla::kNope * 2, v_bytes = size_t(g.rows) * H * mla::kVDim * 2;
        if (int e = grow(c, &c->pf_kv, &c->pf_kv_cap, k_bytes + v_bytes, true)) return e;
        void *kx = c->pf_kv, *vx = static_cast<char*>(c->pf_kv) + k_bytes;               // rows of 256 bytes
        mla::GemmCall gc;
        gc.paged_map = &c->tmaps[mla::kMapPoolSub];
        gc.table = g.pages;
        gc.layer = layer;
        gc.n_pages = c->cfg.n_pages;
        gc.M = g.rows;
        gc.K = mla::kRank;
        gc.n_weights = 2;
        gc.w[0] = gemm_weight(c->w_uk_rows_maps, H * mla::kNope, kx, layer * H * mla::kNope);
        gc.w[1] = gemm_weight(c->w_uv_maps, H * mla::kVDim, vx, layer * H * mla::kVDim);
        int rc = mla::launch_gemm_tc5(dt, gc, c->gemm_ws, c->status_dev, st, c->launches);
        if (rc) return fail(c, rc == -1 ? MLA_ERR_INVALID : MLA_ERR_CUDA, "key / value expansion launch failed");
        mla::PrefillCall p;
        p.q = q; p.out = out; p.kx = kx; p.vx = vx;
        p.pool_map = &c->tmaps[mla::kMapPoolSub];
        p.pages = g.pages;
        p.tiles = g.tiles;
        p.n_tiles = g.n_tiles;
        p.rows = g.rows;
        p.H = H;
        p.layer = layer;
        p.n_pages = c->cfg.n_pages;
        p.cos_sin = c->q_rope_in_kernel ? c->cos_sin : nullptr;
        p.cs_rows = c->cs_rows;
        rc = mla::launch_prefill_tc5(dt, p, c->status_dev, st);
        if (rc) return fail(c, rc == -1 ? MLA_ERR_INVALID : MLA_ERR_CUDA, "prefill attention launch failed");
        c->launches++;
    }
    return MLA_OK;
}

// one layer of a step: append + attention, with the append riding in the absorb launch where it can.
// kv_a_settled: kv_a was complete before the kernel launched just ahead of this layer's started (see launch_absorb_tc5).
int run_layer(mla_ctx* c, uint32_t layer, const void* kv_a, const void* q, void* out, cudaStream_t st, bool kv_a_settled = false)
{
    if (c->has_chunks) {
        // decode-style rows through their own plan (their append covers ALL new rows of the step), then the chunks
        if (c->plan_rest.m.rows) {
            if (int e = run_attend(c, layer, q, out, nullptr, c->plan_rest, st, kv_a, kv_a_settled)) return e;
        } else {
            if (int e = run_append(c, layer, kv_a, c->plan_rest.m, st)) return e;
        }
        return run_chunks(c, layer, q, out, st);
    }
    return run_attend(c, layer, q, out, nullptr, c->plan, st, kv_a, kv_a_settled);
}

int make_tensor_maps(mla_ctx* c)
{
    const mla::TensorMapEncodeFn enc = mla::tensor_map_encoder();
    if (!enc) return fail(c, MLA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    const CUtensorMapDataType dt = c->cfg.dtype == MLA_DTYPE_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    auto encode = [&](int slot, const char* what, cuuint32_t rank, void* basep, const cuuint64_t* dims,
                      const cuuint64_t* strides, const cuuint32_t* box) -> int {
        const CUresult r = enc(&c->tmaps[slot], dt, rank, basep, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return fail(c, MLA_ERR_CUDA, std::string("cuTensorMapEncodeTiled(") + what + ") failed with code " + std::to_string(int(r)));
        return MLA_OK;
    };
    {   // W_UV of all layers as [layers*H*128 outputs][512 dims], boxes of 64 dims x 128 outputs (merge), and W_UK^T as
        // [layers*H*512 d][128 i], boxes of 64 i x 128 d (absorb)
        const uint64_t heads = uint64_t(c->cfg.n_layers) * c->cfg.n_heads;
        const int type = int(c->cfg.dtype);
        if (!mla::make_matrix_map(&c->w_uv_map, type, c->w_uv, heads * mla::kVDim, mla::kRank, mla::kVDim) ||
            !mla::make_matrix_map(&c->w_uk_map, type, c->w_uk, heads * mla::kRank, mla::kNope, 128) ||
            !mla::gemm_tc5_weight_maps(&c->w_uk_rows_maps, type, c->w_uk_rows, heads * mla::kNope, mla::kRank) ||
            !mla::gemm_tc5_weight_maps(&c->w_uv_maps, type, c->w_uv, heads * mla::kVDim, mla::kRank))
            return fail(c, MLA_ERR_CUDA, "cuTensorMapEncodeTiled(W_UK, W_UV) failed");
    }
    {   // cache pool: 576 values innermost, then the token slots of a layer, then layers;
        // box = 64 values (128 B, one swizzle row) x 64 tokens (one page)
        const cuuint64_t dims[3] = {cuuint64_t(mla::kRow), c->pool_slots, c->cfg.n_layers};
        const cuuint64_t strides[2] = {cuuint64_t(mla::kRow) * 2, c->pool_slots * mla::kRow * 2};
        const cuuint32_t box[3] = {64, 64, 1};
        if (int e = encode(mla::kMapPoolSub, "cache pool", 3, c->pool, dims, strides, box)) return e;
    }
    // Whole-row views: the 576 values of a row are exposed as (64 values, 9 chunks) with the chunk
    // dimension OUTSIDE the row dimension, so one box {64 values, R rows, C chunks} lands in shared
    // memory as C consecutive swizzled sub-tiles [R rows][128 B] — a whole operand in ONE TMA
    // instruction instead of nine (a TMA issue costs its thread ~100 cycles).
    {
        const cuuint64_t dims[4] = {64, c->pool_slots, 9, c->cfg.n_layers};
        const cuuint64_t strides[3] = {cuuint64_t(mla::kRow) * 2, 128, c->pool_slots * mla::kRow * 2};
        const cuuint32_t box_v[4] = {64, 64, 2, 1};
        if (int e = encode(mla::kMapPoolV, "cache pool, two chunks of a page", 4, c->pool, dims, strides, box_v)) return e;
        // 64 spare rows behind the queries: boxes of up to 64 head rows may start at the last row's heads
        const cuuint64_t qdims[3] = {64, cuuint64_t(c->ws_rows) * c->cfg.n_heads + 64, 9};
        const cuuint64_t qstrides[2] = {cuuint64_t(mla::kRow) * 2, 128};
        for (int head_rows : {16, 32, 48, 64}) {
            const cuuint32_t qbox[3] = {64, cuuint32_t(head_rows), 9};
            if (int e = encode(mla::query_map(head_rows), "absorbed queries", 3, c->q_abs, qdims, qstrides, qbox)) return e;
        }
    }
    return MLA_OK;
}

}  // namespace

extern "C" {

int mla_create(const mla_config* cfg, mla_ctx** out)
{
    if (!cfg || !out) return fail(nullptr, MLA_ERR_INVALID, "null argument");
    *out = nullptr;
    // same wording as KVCache::create's validation (src/core/memory/kv_cache.cpp:146-159)
    if (cfg->n_layers == 0) return fail(nullptr, MLA_ERR_INVALID, "n_layers must be > 0");
    if (cfg->n_heads == 0) return fail(nullptr, MLA_ERR_INVALID, "n_heads must be > 0");
    if (cfg->max_seq_len == 0) return fail(nullptr, MLA_ERR_INVALID, "max_seq_len must be > 0");
    if (cfg->kv_lora_rank != 512 || cfg->qk_nope_head_dim != 128 || cfg->qk_rope_head_dim != 64 ||
        cfg->v_head_dim != 128)
        return fail(nullptr, MLA_ERR_UNSUPPORTED,
                    "only kv_lora_rank 512, qk_nope_head_dim 128, qk_rope_head_dim 64, v_head_dim 128 are built");
    if (cfg->page_tokens != 64) return fail(nullptr, MLA_ERR_UNSUPPORTED, "page_tokens must be 64");
    if (cfg->n_pages == 0 || cfg->max_seqs == 0) return fail(nullptr, MLA_ERR_INVALID, "n_pages and max_seqs must be > 0");
    if (cfg->dtype > MLA_DTYPE_BF16) return fail(nullptr, MLA_ERR_INVALID, "dtype must be MLA_DTYPE_F16 or MLA_DTYPE_BF16");
    if (cfg->kernel > MLA_KERNEL_TCGEN05_T16) return fail(nullptr, MLA_ERR_INVALID, "unknown kernel selector");

    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0)
        return fail(nullptr, MLA_ERR_CUDA, std::string("no CUDA device: ") + cudaGetErrorString(e) +
                                               " (this library has no CPU path)");
    if (cfg->device < 0 || cfg->device >= ndev) return fail(nullptr, MLA_ERR_INVALID, "device ordinal out of range");

    auto c = std::make_unique<mla_ctx>();
    c->cfg = *cfg;
    if (c->cfg.max_rows == 0) c->cfg.max_rows = c->cfg.max_seqs;
    mla_ctx* cp = c.get();
    auto bail = [&](int code) { g_create_error = cp->err; mla_destroy(c.release()); return code; };
#define CR_TRY(expr)                                                                            \
    do {                                                                                        \
        cudaError_t e__ = (expr);                                                               \
        if (e__ != cudaSuccess) {                                                               \
            cp->err = std::string(#expr) + ": " + cudaGetErrorString(e__);                     \
            return bail(MLA_ERR_CUDA);                                                          \
        }                                                                                       \
    } while (0)
    CR_TRY(cudaSetDevice(cfg->device));
    cudaDeviceProp prop{};
    CR_TRY(cudaGetDeviceProperties(&prop, cfg->device));
    c->sm_count = prop.multiProcessorCount;
    if (prop.major != 10)
        { cp->err = "this library is built for sm_100a only; device is sm_" + std::to_string(prop.major * 10 + prop.minor);
          return bail(MLA_ERR_UNSUPPORTED); }
    c->kernel = kernel_for(cp, cfg->n_heads);
    const uint32_t H = cfg->n_heads;

    c->pt = std::make_unique<PageTable>(cfg->page_tokens, cfg->n_pages, cfg->max_seqs, cfg->max_seq_len);
    c->layer_set.resize(cfg->n_layers, 0);
    c->blocks.resize(cfg->n_layers);
    c->pool_slots = uint64_t(cfg->n_pages) * cfg->page_tokens;
    const size_t pool_bytes = size_t(cfg->n_layers) * c->pool_slots * mla::kRow * 2;
    CR_TRY(cudaMalloc(&c->pool, pool_bytes));
    // zero-fill: rows past a sequence's end inside its last page are multiplied by P = 0 and
    // must therefore hold finite values
    CR_TRY(cudaMemset(c->pool, 0, pool_bytes));
    for (char** w : {&c->w_uk, &c->w_uk_rows, &c->w_uv}) CR_TRY(cudaMalloc(w, weight_bytes(cp) * cfg->n_layers));
    CR_TRY(cudaMalloc(&c->norm, size_t(cfg->n_layers) * mla::kRank * 2));
    // rotary table: one row per position a sequence can reach
    c->cs_cap = std::max(cfg->max_seq_len, cfg->max_position);
    CR_TRY(cudaMalloc(&c->cos_sin, size_t(c->cs_cap) * mla::kRope * sizeof(float)));
    // Workspace for the rows of one step, or of a group of layers when a step has few rows (mla_step_layers).
    const uint64_t row_bytes = uint64_t(H) * mla::kRow * 2;
    auto group_rows = [&](uint64_t rows, uint64_t bytes) {
        return std::max<uint32_t>(c->cfg.max_rows, uint32_t(std::min<uint64_t>({uint64_t(c->cfg.max_rows) * cfg->n_layers, rows,
                                                                                std::max<uint64_t>(1, bytes / row_bytes)})));
    };
    const uint32_t small_groups = group_rows(kSmallGroupRows, kSmallGroupBytes);
    const size_t own_bytes = pool_bytes + 3 * weight_bytes(cp) * cfg->n_layers;
    c->ws_rows = prop.totalGlobalMem >= own_bytes + kRoomForGroups ? group_rows(kGroupRows, kGroupBytes) : small_groups;
    CR_TRY(cudaMalloc(&c->status_dev, sizeof(uint32_t)));
    CR_TRY(cudaMemset(c->status_dev, 0, sizeof(uint32_t)));
    c->meta_cap = meta_capacity(cp);
    CR_TRY(cudaMalloc(&c->meta_dev, kPlanRegions * c->meta_cap));
    CR_TRY(cudaMallocHost(&c->meta_host, kMetaRing * c->meta_cap));
    for (int i = 0; i < kMetaRing; i++) {
        MetaBuf& mb = c->ring[i];
        mb.host = c->meta_host + i * c->meta_cap;
        CR_TRY(cudaEventCreateWithFlags(&mb.done, cudaEventDisableTiming));
    }
    if (int ce = mla::decode_mma_configure()) {
        cp->err = std::string("mma attention kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::merge_mma_configure()) {
        cp->err = std::string("mma merge kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::prefill_tc5_configure()) {
        cp->err = std::string("tcgen05 prefill kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::gemm_tc5_configure(int(cfg->dtype))) {
        cp->err = std::string("tcgen05 projection kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::absorb_tc5_configure()) {
        cp->err = std::string("tcgen05 absorb kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::merge_tc5_configure()) {
        cp->err = std::string("tcgen05 merge kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    // The last allocations.  Where the device is too full for groups of layers and of rows, smaller ones or one layer of max_rows rows
    // must do: with the last of them steps go layer by layer, and rows of one sequence share a stream of its pages as far as the
    // records hold them.
    auto workspace = [&](uint32_t rows, bool groups, size_t left) -> cudaError_t {
        c->ws_rows = rows;
        // a plan has at most one segment per query group more than it has workers, each of up to group_heads (or H) records
        c->rec_cap = (size_t(workers_of(cp, c->kernel, H)) + rows) * H;
        if (groups && group_heads(cp) >= 2 * H) c->rec_cap += size_t(c->sm_count) * group_heads(cp) + size_t(rows) * H;
        // 64 spare rows: the tcgen05 kernels fetch queries in boxes of 64 head rows
        const size_t q_bytes = (size_t(rows) * H + 64) * mla::kRow * 2;
        size_t free_bytes = 0, total_bytes = 0;
        cudaError_t e = cudaMalloc(&c->q_abs, q_bytes);
        if (e == cudaSuccess) e = cudaMalloc(&c->recs, c->rec_cap * mla::kPart * sizeof(float));
        if (e == cudaSuccess) e = cudaMemGetInfo(&free_bytes, &total_bytes);
        if (e == cudaSuccess && free_bytes < left) e = cudaErrorMemoryAllocation;
        if (e == cudaSuccess) return cudaMemset(c->q_abs, 0, q_bytes);
        cudaGetLastError();
        cudaFree(c->q_abs);
        cudaFree(c->recs);
        c->q_abs = nullptr;
        c->recs = nullptr;
        return e;
    };
    cudaError_t we = cudaErrorMemoryAllocation;
    if (c->ws_rows > small_groups) we = workspace(c->ws_rows, true, kLeftByGroups);
    if (we == cudaErrorMemoryAllocation) we = workspace(small_groups, true, 0);
    if (we == cudaErrorMemoryAllocation) we = workspace(c->cfg.max_rows, false, 0);
    CR_TRY(we);
    if (int rc = make_tensor_maps(cp)) return bail(rc);
    if (int ce = mla::decode_tc5_pair128_configure()) {
        cp->err = std::string("tcgen05 pair128 kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
    if (int ce = mla::decode_tc5_configure(int(cfg->dtype))) {
        cp->err = std::string("tcgen05 kernel configuration: ") + cudaGetErrorString(cudaError_t(ce));
        return bail(MLA_ERR_CUDA);
    }
#undef CR_TRY
    *out = c.release();
    return MLA_OK;
}

void mla_destroy(mla_ctx* c)
{
    if (!c) return;
    cudaSetDevice(c->cfg.device);
    cudaDeviceSynchronize();
    cudaFree(c->pool);
    cudaFree(c->w_uk); cudaFree(c->w_uk_rows); cudaFree(c->w_uv); cudaFree(c->norm);
    cudaFree(c->pf_kv);
    cudaFree(c->cos_sin);
    cudaFree(c->q_abs);
    cudaFree(c->recs);
    cudaFree(c->status_dev);
    cudaFree(c->meta_dev);
    for (auto& mb : c->ring) {
        if (mb.done) cudaEventDestroy(mb.done);
    }
    if (c->meta_host) cudaFreeHost(c->meta_host);
    for (auto& pe : c->prof_events) { cudaEventDestroy(pe.first); cudaEventDestroy(pe.second); }
    if (c->h_in) cudaFreeHost(c->h_in);
    if (c->h_out) cudaFreeHost(c->h_out);
    cudaFree(c->d_kv); cudaFree(c->d_q); cudaFree(c->d_out);
    for (auto& b : c->blocks) { cudaFree(b.attn_norm); cudaFree(b.q_a); cudaFree(b.q_a_norm); cudaFree(b.q_b); cudaFree(b.q); cudaFree(b.kv_a); cudaFree(b.wo); }
    cudaFree(c->blk_hidden2); cudaFree(c->blk_qa); cudaFree(c->blk_rows); cudaFree(c->gemm_ws.partial); cudaFree(c->gemm_ws.counters);
    for (auto& ev : c->host_ev) { cudaEventDestroy(ev.in); cudaEventDestroy(ev.compute); cudaEventDestroy(ev.out); }
    if (c->copy_in) cudaStreamDestroy(c->copy_in);
    if (c->copy_out) cudaStreamDestroy(c->copy_out);
    delete c;
}

const char* mla_last_error(const mla_ctx* c) { return c ? c->err.c_str() : g_create_error.c_str(); }

int mla_status(mla_ctx* c, void* stream, uint32_t* device_status)
{
    if (!c || !device_status) return MLA_ERR_INVALID;
    USE_DEVICE(c);
    auto st = static_cast<cudaStream_t>(stream);
    uint32_t v = 0;
    CU_TRY(c, cudaMemcpyAsync(&v, c->status_dev, 4, cudaMemcpyDeviceToHost, st));
    CU_TRY(c, cudaStreamSynchronize(st));
    if (v) {
        CU_TRY(c, cudaMemsetAsync(c->status_dev, 0, 4, st));
        // a projection that gave up in the middle may have left tile counters behind
        if (c->gemm_ws.counters) CU_TRY(c, cudaMemsetAsync(c->gemm_ws.counters, 0, c->gemm_ws.max_tiles * 4, st));
    }
    *device_status = v;
    if (v) return fail(c, MLA_ERR_DEVICE, "device status word = " + std::to_string(v));
    return MLA_OK;
}

int mla_set_layer_weights(mla_ctx* c, uint32_t layer, const void* w_uk, const void* w_uv, uint32_t w_type,
                          const void* kv_norm)
{
    if (!c || !w_uk || !w_uv || !kv_norm) return fail(c, MLA_ERR_INVALID, "null argument");
    if (int e = check_layer(c, layer, false)) return e;
    CU_TRY(c, cudaSetDevice(c->cfg.device));
    std::vector<uint16_t> buf;
    const size_t H = c->cfg.n_heads;
    if (int e = decode_weights(c, w_uk, w_type, H * mla::kNope, buf)) return e;
    {   // the absorb kernel reads W_UK transposed per head: [h][d][i] (contraction index contiguous)
        std::vector<uint16_t> tr(buf.size());
        for (size_t h = 0; h < H; h++)
            for (size_t i = 0; i < size_t(mla::kNope); i++)
                for (size_t d = 0; d < size_t(mla::kRank); d++)
                    tr[(h * mla::kRank + d) * mla::kNope + i] = buf[(h * mla::kNope + i) * mla::kRank + d];
        CU_TRY(c, cudaMemcpy(c->w_uk + layer * weight_bytes(c), tr.data(), tr.size() * 2, cudaMemcpyHostToDevice));
        CU_TRY(c, cudaMemcpy(c->w_uk_rows + layer * weight_bytes(c), buf.data(), buf.size() * 2, cudaMemcpyHostToDevice));
    }
    if (int e = decode_weights(c, w_uv, w_type, H * mla::kVDim, buf)) return e;
    CU_TRY(c, cudaMemcpy(c->w_uv + layer * weight_bytes(c), buf.data(), buf.size() * 2, cudaMemcpyHostToDevice));
    CU_TRY(c, cudaMemcpy(layer_norm(c, layer), kv_norm, mla::kRank * 2, cudaMemcpyHostToDevice));
    c->layer_set[layer] = 1;
    return MLA_OK;
}

int mla_seq_create(mla_ctx* c, uint32_t* id)
{
    if (!c || !id) return MLA_ERR_INVALID;
    return pt_code(c, c->pt->seq_create(id));
}
// While a step is open its uploaded block tables name the sequences' pages: giving pages back (or moving a
// counter the step is about to move) in between would let another sequence take pages the kernels still read.
static int refuse_in_step(mla_ctx* c, const char* what)
{
    return fail(c, MLA_ERR_STATE, std::string(what) + " is not allowed while a step is open");
}
int mla_seq_free(mla_ctx* c, uint32_t id)
{
    if (!c) return MLA_ERR_INVALID;
    if (c->in_step) return refuse_in_step(c, "seq_free");
    return pt_code(c, c->pt->seq_free(id));
}
int mla_seq_len(const mla_ctx* c, uint32_t id, uint32_t* len)
{
    if (!c || !len) return MLA_ERR_INVALID;
    return c->pt->seq_len(id, len);
}
int mla_advance(mla_ctx* c, uint32_t id, uint32_t n)
{
    if (!c) return MLA_ERR_INVALID;
    if (c->in_step) return refuse_in_step(c, "advance");
    return pt_code(c, c->pt->advance(id, n));
}
int mla_truncate(mla_ctx* c, uint32_t id, uint32_t n)
{
    if (!c) return MLA_ERR_INVALID;
    if (c->in_step) return refuse_in_step(c, "truncate");
    return pt_code(c, c->pt->truncate(id, n));
}
int mla_rollback(mla_ctx* c, uint32_t n_seq, const uint32_t* seq_ids, const uint32_t* keep_lens)
{
    if (!c || (n_seq && (!seq_ids || !keep_lens))) return fail(c, MLA_ERR_INVALID, "null argument");
    if (c->in_step) return refuse_in_step(c, "rollback");
    for (uint32_t i = 0; i < n_seq; i++)
        if (!c->pt->seq(seq_ids[i])) return fail(c, MLA_ERR_INVALID, "unknown sequence id " + std::to_string(seq_ids[i]));
    for (uint32_t i = 0; i < n_seq; i++)
        if (c->pt->seq(seq_ids[i])->len > keep_lens[i])
            if (int e = pt_code(c, c->pt->truncate(seq_ids[i], keep_lens[i]))) return e;
    return MLA_OK;
}
int mla_clear(mla_ctx* c, uint32_t id)
{
    if (!c) return MLA_ERR_INVALID;
    if (c->in_step) return refuse_in_step(c, "clear");
    return pt_code(c, c->pt->clear(id));
}
int mla_seq_set_base(mla_ctx* c, uint32_t id, uint32_t base) { return c ? pt_code(c, c->pt->set_base(id, base)) : MLA_ERR_INVALID; }
int mla_free_pages(const mla_ctx* c, uint32_t* n)
{
    if (!c || !n) return MLA_ERR_INVALID;
    *n = c->pt->free_pages();
    return MLA_OK;
}
int mla_shuffle_free_pages(mla_ctx* c, uint64_t seed)
{
    if (!c) return MLA_ERR_INVALID;
    c->pt->shuffle_free(seed);
    return MLA_OK;
}
int mla_seq_pages(const mla_ctx* c, uint32_t id, uint32_t* pages, uint32_t cap, uint32_t* n_pages)
{
    if (!c || !n_pages) return MLA_ERR_INVALID;
    const auto* s = c->pt->seq(id);
    if (!s) return MLA_ERR_INVALID;
    *n_pages = uint32_t(s->pages.size());
    if (pages) std::memcpy(pages, s->pages.data(), std::min<size_t>(cap, s->pages.size()) * 4);
    return MLA_OK;
}

int mla_append_rows(mla_ctx* c, uint32_t layer, uint32_t n, const uint32_t* seq_ids, const uint32_t* positions,
                    const void* kv_a, void* stream)
{
    if (!c || (n && (!seq_ids || !positions || !kv_a))) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (int e = check_layer(c, layer, true)) return e;
    if (c->in_step) return fail(c, MLA_ERR_STATE, "explicit-position calls are not allowed while a step is open");
    if (n > c->cfg.max_rows) return fail(c, MLA_ERR_CAPACITY, "more rows than max_rows");
    auto st = static_cast<cudaStream_t>(stream);
    std::vector<uint32_t> seqs;
    std::vector<RowSpec> rows(n);
    uint32_t max_pos = 0;
    for (uint32_t r = 0; r < n; r++) {
        const auto* s = c->pt->seq(seq_ids[r]);
        if (!s) return fail(c, MLA_ERR_INVALID, "unknown sequence id " + std::to_string(seq_ids[r]));
        if (positions[r] < s->base_pos) return fail(c, MLA_ERR_INVALID, "position below the sequence's base position");
        const uint32_t local = positions[r] - s->base_pos;
        if (int e = pt_code(c, c->pt->reserve(seq_ids[r], local + 1))) return e;
        rows[r] = {0, 0, positions[r], c->pt->slot(seq_ids[r], local)};
        max_pos = std::max(max_pos, positions[r]);
    }
    if (n) if (int e = ensure_rope_rows(c, max_pos + 1, st)) return e;
    if (int e = build_plan(c, c->plan, kPlanStep, seqs, rows, nullptr, nullptr, 0, st)) return e;
    return run_append(c, layer, kv_a, c->plan.m, st);
}

int mla_attend_rows(mla_ctx* c, uint32_t layer, uint32_t n, const uint32_t* seq_ids, const uint32_t* attend_lens,
                    const void* q, void* out, void* stream)
{
    if (!c || (n && (!seq_ids || !attend_lens || !q || !out))) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (int e = check_layer(c, layer, true)) return e;
    if (c->in_step) return fail(c, MLA_ERR_STATE, "explicit-position calls are not allowed while a step is open");
    if (n > c->cfg.max_rows) return fail(c, MLA_ERR_CAPACITY, "more rows than max_rows");
    auto st = static_cast<cudaStream_t>(stream);
    std::vector<uint32_t> seqs;
    std::vector<RowSpec> rows(n);
    uint32_t max_pos = 0;
    for (uint32_t r = 0; r < n; r++) {
        const auto* s = c->pt->seq(seq_ids[r]);
        if (!s) return fail(c, MLA_ERR_INVALID, "unknown sequence id " + std::to_string(seq_ids[r]));
        if (uint64_t(attend_lens[r]) > uint64_t(s->pages.size()) * mla::kPage)
            return fail(c, MLA_ERR_INVALID, "attend length " + std::to_string(attend_lens[r]) +
                                                " reaches rows that were never appended");
        uint32_t idx = 0;
        for (; idx < seqs.size(); idx++) if (seqs[idx] == seq_ids[r]) break;
        if (idx == seqs.size()) seqs.push_back(seq_ids[r]);
        // the query stands at the last attended position (matters only when the library rotates q)
        const uint32_t qpos = s->base_pos + (attend_lens[r] ? attend_lens[r] - 1 : 0);
        rows[r] = {idx, attend_lens[r], qpos, 0};
        max_pos = std::max(max_pos, qpos);
    }
    if (n && c->q_rope_in_kernel) if (int e = ensure_rope_rows(c, max_pos + 1, st)) return e;
    if (int e = build_plan(c, c->plan, kPlanStep, seqs, rows, nullptr, nullptr, 1, st)) return e;
    return run_attend(c, layer, q, out, nullptr, c->plan, st);
}

int mla_step_begin(mla_ctx* c, uint32_t n_seq, const uint32_t* seq_ids, const uint32_t* n_new, void* stream)
{
    if (!c || (n_seq && !seq_ids)) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (c->in_step) return fail(c, MLA_ERR_STATE, "step_begin while a step is open");
    auto st = static_cast<cudaStream_t>(stream);
    std::vector<uint32_t> seqs(seq_ids, seq_ids + n_seq);
    std::vector<uint32_t> nn(n_seq, 1);
    if (n_new) nn.assign(n_new, n_new + n_seq);
    uint64_t total = 0;
    for (uint32_t i = 0; i < n_seq; i++) {
        if (!c->pt->seq(seqs[i])) return fail(c, MLA_ERR_INVALID, "unknown sequence id " + std::to_string(seqs[i]));
        for (uint32_t j = 0; j < i; j++)
            if (seqs[j] == seqs[i]) return fail(c, MLA_ERR_INVALID, "sequence listed twice in one step");
        total += std::max<uint32_t>(nn[i], 1);
    }
    if (total > c->cfg.max_rows) return fail(c, MLA_ERR_CAPACITY, "step has " + std::to_string(total) + " rows, max_rows is " + std::to_string(c->cfg.max_rows));
    // reserve first (all-or-nothing per sequence; on failure earlier reservations stay, harmless)
    uint32_t max_pos = 0;
    for (uint32_t i = 0; i < n_seq; i++) {
        const auto* s = c->pt->seq(seqs[i]);
        if (int e = pt_code(c, c->pt->reserve(seqs[i], s->len + nn[i]))) return e;
        if (nn[i]) max_pos = std::max(max_pos, s->base_pos + s->len + nn[i] - 1);
    }
    if (total) if (int e = ensure_rope_rows(c, max_pos + 1, st)) return e;
    auto& rows = c->rows;
    rows.clear();
    rows.reserve(total);
    c->chunks.clear();
    c->has_chunks = false;
    c->step_new_rows = 0;
    for (uint32_t i = 0; i < n_seq; i++) {
        const auto* s = c->pt->seq(seqs[i]);
        if (nn[i] == 0) {                                              // query-only row
            if (c->q_rope_in_kernel)
                return fail(c, MLA_ERR_UNSUPPORTED, "a query-only row has no position of its own: rotate q on the caller's side "
                                                    "(mla_set_q_rope(ctx, 0)) for KV-range shards that do not own the tail");
            rows.push_back({i, s->len, 0, ~uint64_t(0)});
        }
        if (nn[i] >= kPrefillMin && c->kernel != MLA_KERNEL_MMA) {
            c->chunks.push_back({i, uint32_t(rows.size()), nn[i], s->len, s->base_pos});
            c->has_chunks = true;
        }
        for (uint32_t t = 0; t < nn[i]; t++) {
            const uint32_t local = s->len + t;
            rows.push_back({i, local + 1, s->base_pos + local, c->pt->slot(seqs[i], local)});
        }
        c->step_new_rows += nn[i];
    }
    c->step_rows = uint32_t(rows.size());
    c->stack.ready = c->stack_tail.ready = false;
    c->step_seqs = std::move(seqs);
    c->step_nnew = std::move(nn);
    if (int e = build_plan(c, c->plan, kPlanStep, c->step_seqs, rows, nullptr, nullptr, 1, st)) return e;
    if (c->has_chunks)
        if (int e = rest_plan(c, st)) return e;
    c->in_step = true;
    return MLA_OK;
}

int mla_step_append(mla_ctx* c, uint32_t layer, const void* kv_a, void* stream)
{
    if (!c || !kv_a) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_append outside step_begin/step_end");
    if (int e = check_layer(c, layer, true)) return e;
    return run_append(c, layer, kv_a, c->plan.m, static_cast<cudaStream_t>(stream));
}

int mla_step_attend(mla_ctx* c, uint32_t layer, const void* q, void* out, void* stream)
{
    if (!c || !q || !out) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_attend outside step_begin/step_end");
    if (int e = check_layer(c, layer, true)) return e;
    return run_attend(c, layer, q, out, nullptr, c->plan, static_cast<cudaStream_t>(stream));
}

int mla_step_layers(mla_ctx* c, uint32_t layer_begin, uint32_t n_layers, const void* kv_a, const void* q, void* out,
                    void* stream)
{
    if (!c || !kv_a || !q || !out) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_layers outside step_begin/step_end");
    if (uint64_t(layer_begin) + n_layers > c->cfg.n_layers) return fail(c, MLA_ERR_INVALID, "layer range out of bounds");
    auto st = static_cast<cudaStream_t>(stream);
    const size_t rows = c->step_rows, H = c->cfg.n_heads;
    const size_t kv_b = rows * mla::kRow * 2, q_b = rows * H * mla::kQDim * 2, o_b = rows * H * mla::kVDim * 2;
    for (uint32_t i = 0; i < n_layers; i++)
        if (int e = check_layer(c, layer_begin + i, true)) return e;
    // Layers whose inputs are all at hand need not queue up one behind the other: a group of them is ONE absorb, one
    // attention and one merge launch, planned together, so that a step of few rows fills the machine.
    uint32_t group = 1;
    if (!c->has_chunks && rows && c->kernel != MLA_KERNEL_MMA) group = uint32_t(std::min<uint64_t>(n_layers, c->ws_rows / rows));
    // The group's plan is uploaded by this call: not into a captured graph, whose replays would read the upload ring again
    // long after it went on.  A captured call goes layer by layer with the plan of mla_step_begin.
    if (group > 1 && capturing(st)) group = 1;
    if (group > 1) {
        const uint32_t n_groups = (n_layers + group - 1) / group;
        group = (n_layers + n_groups - 1) / n_groups;
        // both plans go up ahead of the first launch: an upload between two launches ends their overlap
        auto plan_of = [&](uint32_t n) -> Plan& { return n == group ? c->stack : c->stack_tail; };
        bool own_upload = false;               // by this call, so that nothing stands between it and the first launch
        for (uint32_t n : {group, n_layers % group})
            if (Plan& p = plan_of(n); n && (!p.ready || p.m.layers != n)) {
                if (int e = build_plan(c, p, n == group ? kPlanStack : kPlanStackTail, c->step_seqs, c->rows, nullptr, nullptr, n, st)) return e;
                own_upload = true;
            }
        for (uint32_t i = 0; i < n_layers; i += group) {
            const uint32_t n = std::min(group, n_layers - i);
            Plan& p = plan_of(n);
            if (int e = run_attend(c, layer_begin + i, static_cast<const char*>(q) + i * q_b, static_cast<char*>(out) + i * o_b, nullptr, p, st,
                                   static_cast<const char*>(kv_a) + i * kv_b, i > 0, own_upload && i == 0))
                return e;
        }
        return MLA_OK;
    }
    for (uint32_t i = 0; i < n_layers; i++) {
        const uint32_t layer = layer_begin + i;
        // the caller's kv_a for ALL layers existed before this call: from the second layer on, the kernel ahead of the
        // layer's first launch is this library's own and kv_a was complete before it started
        if (int e = run_layer(c, layer, static_cast<const char*>(kv_a) + i * kv_b, static_cast<const char*>(q) + i * q_b,
                              static_cast<char*>(out) + i * o_b, st, i > 0))
            return e;
    }
    return MLA_OK;
}

int mla_step_attend_partial(mla_ctx* c, uint32_t layer, const void* q, float* partial, void* stream)
{
    if (!c || !q || !partial) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_attend_partial outside step_begin/step_end");
    if (int e = check_layer(c, layer, true)) return e;
    return run_attend(c, layer, q, nullptr, partial, c->plan, static_cast<cudaStream_t>(stream));
}

int mla_step_layer_partial(mla_ctx* c, uint32_t layer, const void* kv_a, const void* q, float* partial, void* stream)
{
    if (!c || !q || !partial) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_layer_partial outside step_begin/step_end");
    if (int e = check_layer(c, layer, true)) return e;
    if (c->has_chunks) return fail(c, MLA_ERR_UNSUPPORTED, "a step with prefill chunks has no partial form");
    if (c->step_new_rows && !kv_a) return fail(c, MLA_ERR_INVALID, "the step appends rows on this GPU: kv_a is needed");
    auto st = static_cast<cudaStream_t>(stream);
    if (!c->step_new_rows) kv_a = nullptr;           // query-only rows: nothing to append, kv_a is never read
    return run_attend(c, layer, q, nullptr, partial, c->plan, st, kv_a);
}

int mla_merge_partials(mla_ctx* c, uint32_t layer, uint32_t n_parts, uint32_t rows, const float* partials,
                       void* out, void* stream)
{
    if (!c || !partials || !out || n_parts == 0) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (int e = check_layer(c, layer, true)) return e;
    mla::StepMeta m{};
    m.rows = rows;
    m.layers = 1;
    auto st = static_cast<cudaStream_t>(stream);
    const int e = mla::launch_merge_tc5(int(c->cfg.dtype), partials, m, n_parts, &c->w_uv_map, out, c->cfg.n_heads, layer, uint32_t(c->sm_count), c->status_dev,
                                        launch_stream(c, st));
    if (e != 0) return fail(c, MLA_ERR_CUDA, std::string("merge launch: ") + cudaGetErrorString(cudaError_t(e)));
    if (rows) launched(c, st);
    c->launches += rows ? 1 : 0;
    CU_TRY(c, cudaGetLastError());
    return MLA_OK;
}

static bool is_pinned(const void* p)
{
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost;
}

int mla_step_layer_host(mla_ctx* c, uint32_t layer, const void* kv_a_host, const void* q_host, void* out_host,
                        void* stream)
{
    if (!c || !kv_a_host || !q_host || !out_host) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_layer_host outside step_begin/step_end");
    if (int e = check_layer(c, layer, true)) return e;
    auto st = static_cast<cudaStream_t>(stream);
    const size_t R = c->cfg.max_rows, H = c->cfg.n_heads, rows = c->step_rows, L = c->cfg.n_layers;
    const size_t kv_cap = R * mla::kRow * 2, q_cap = R * H * mla::kQDim * 2, o_cap = R * H * mla::kVDim * 2;
    const size_t kv_b = rows * mla::kRow * 2, q_b = rows * H * mla::kQDim * 2, o_b = rows * H * mla::kVDim * 2;
    if (!c->d_kv) {
        // one device slot per layer: the layers of a step then queue up without waiting for
        // each other's copies
        CU_TRY(c, cudaMalloc(&c->d_kv, L * kv_cap));
        CU_TRY(c, cudaMalloc(&c->d_q, L * q_cap));
        CU_TRY(c, cudaMalloc(&c->d_out, L * o_cap));
    }
    char* d_kv = static_cast<char*>(c->d_kv) + layer * kv_cap;
    char* d_q = static_cast<char*>(c->d_q) + layer * q_cap;
    char* d_out = static_cast<char*>(c->d_out) + layer * o_cap;
    const bool direct = is_pinned(kv_a_host) && is_pinned(q_host) && is_pinned(out_host);
    if (direct) {
        // page-locked caller buffers: fully asynchronous; out_host is complete when mla_step_end returns
        if (!c->copy_in) {
            CU_TRY(c, cudaStreamCreateWithFlags(&c->copy_in, cudaStreamNonBlocking));
            CU_TRY(c, cudaStreamCreateWithFlags(&c->copy_out, cudaStreamNonBlocking));
            c->host_ev.resize(L);
            for (auto& ev : c->host_ev) {
                CU_TRY(c, cudaEventCreateWithFlags(&ev.in, cudaEventDisableTiming));
                CU_TRY(c, cudaEventCreateWithFlags(&ev.compute, cudaEventDisableTiming));
                CU_TRY(c, cudaEventCreateWithFlags(&ev.out, cudaEventDisableTiming));
            }
        }
        auto& ev = c->host_ev[layer];
        // this layer's device slots were last read / written by its previous use
        if (ev.used) CU_TRY(c, cudaStreamWaitEvent(c->copy_in, ev.compute, 0));
        CU_TRY(c, cudaMemcpyAsync(d_kv, kv_a_host, kv_b, cudaMemcpyHostToDevice, c->copy_in));
        CU_TRY(c, cudaMemcpyAsync(d_q, q_host, q_b, cudaMemcpyHostToDevice, c->copy_in));
        CU_TRY(c, cudaEventRecord(ev.in, c->copy_in));
        CU_TRY(c, cudaStreamWaitEvent(st, ev.in, 0));
        if (ev.used) CU_TRY(c, cudaStreamWaitEvent(st, ev.out, 0));
        if (int e = run_layer(c, layer, d_kv, d_q, d_out, st)) return e;
        CU_TRY(c, cudaEventRecord(ev.compute, st));
        CU_TRY(c, cudaStreamWaitEvent(c->copy_out, ev.compute, 0));
        CU_TRY(c, cudaMemcpyAsync(out_host, d_out, o_b, cudaMemcpyDeviceToHost, c->copy_out));
        CU_TRY(c, cudaEventRecord(ev.out, c->copy_out));
        ev.used = ev.pending = true;
        return MLA_OK;
    }
    if (!c->h_in) {
        CU_TRY(c, cudaMallocHost(&c->h_in, kv_cap + q_cap));
        CU_TRY(c, cudaMallocHost(&c->h_out, o_cap));
    }
    // pageable caller buffers: staged through page-locked memory, synchronous
    CU_TRY(c, cudaStreamSynchronize(st));
    std::memcpy(c->h_in, kv_a_host, kv_b);
    std::memcpy(static_cast<char*>(c->h_in) + kv_cap, q_host, q_b);
    CU_TRY(c, cudaMemcpyAsync(d_kv, c->h_in, kv_b, cudaMemcpyHostToDevice, st));
    CU_TRY(c, cudaMemcpyAsync(d_q, static_cast<char*>(c->h_in) + kv_cap, q_b, cudaMemcpyHostToDevice, st));
    if (int e = run_layer(c, layer, d_kv, d_q, d_out, st)) return e;
    CU_TRY(c, cudaMemcpyAsync(c->h_out, d_out, o_b, cudaMemcpyDeviceToHost, st));
    CU_TRY(c, cudaStreamSynchronize(st));
    std::memcpy(out_host, c->h_out, o_b);
    return MLA_OK;
}

int mla_step_end(mla_ctx* c)
{
    if (!c) return MLA_ERR_INVALID;
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_end without step_begin");
    // The step closes and the counters move whatever happens below (the rows were written by kernels already
    // queued); the first error is reported after that.
    c->in_step = false;
    int rc = MLA_OK;
    cudaSetDevice(c->cfg.device);
    for (auto& ev : c->host_ev)              // outputs of mla_step_layer_host must have landed in the caller's buffers
        if (ev.pending) {
            const cudaError_t e = cudaEventSynchronize(ev.out);
            if (e != cudaSuccess && rc == MLA_OK)
                rc = fail(c, MLA_ERR_CUDA, std::string("cudaEventSynchronize(output copy): ") + cudaGetErrorString(e));
            ev.pending = false;
        }
    for (size_t i = 0; i < c->step_seqs.size(); i++)
        if (int e = pt_code(c, c->pt->advance(c->step_seqs[i], c->step_nnew[i])))
            if (rc == MLA_OK) rc = e;
    return rc;
}

int mla_step_info(const mla_ctx* c, uint32_t* rows, uint32_t* segments)
{
    if (!c) return MLA_ERR_INVALID;
    if (rows) *rows = c->step_rows;
    // of one layer of the step (or of the last explicit call), whatever groups of layers mla_step_layers launches
    if (segments) *segments = c->plan.m.segs;
    return MLA_OK;
}

int mla_step_balance(const mla_ctx* c, uint32_t* workers, uint32_t* min_pages, uint32_t* max_pages)
{
    if (!c) return MLA_ERR_INVALID;
    if (workers) *workers = c->plan_workers;
    if (min_pages) *min_pages = c->plan_min_pages;
    if (max_pages) *max_pages = c->plan_max_pages;
    return MLA_OK;
}

int mla_launch_count(const mla_ctx* c, uint64_t* n)
{
    if (!c || !n) return MLA_ERR_INVALID;
    *n = c->launches;
    return MLA_OK;
}

int mla_set_q_rope(mla_ctx* c, int in_kernel)
{
    if (!c) return MLA_ERR_INVALID;
    if (c->in_step) return fail(c, MLA_ERR_STATE, "mla_set_q_rope inside step_begin/step_end");
    c->q_rope_in_kernel = in_kernel != 0;
    return MLA_OK;
}

int mla_selftest_wait_timeout(mla_ctx* c, uint64_t limit_cycles, void* stream, uint32_t* waited_cycles)
{
    if (!c) return MLA_ERR_INVALID;
    USE_DEVICE(c);
    if (limit_cycles == 0 || limit_cycles > 2000000000ull)
        return fail(c, MLA_ERR_INVALID, "limit_cycles must be in 1 .. 2e9 (about a second)");
    auto st = static_cast<cudaStream_t>(stream);
    uint32_t* report = nullptr;
    CU_TRY(c, cudaMalloc(&report, 16));
    mla::launch_wait_timeout_selftest(static_cast<long long>(limit_cycles), c->status_dev, report, st);
    mla::launch_lost_share_selftest(static_cast<long long>(std::min<uint64_t>(limit_cycles, 1000000)), c->status_dev, report + 2, st);
    c->launches += 2;
    uint32_t host[4] = {1, 0, 1, 1};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, report, 16, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(report);
    if (e != cudaSuccess) return fail(c, MLA_ERR_CUDA, std::string("wait-timeout self-test: ") + cudaGetErrorString(e));
    if (waited_cycles) *waited_cycles = host[1];
    if (host[0] != 0) return fail(c, MLA_ERR_DEVICE, "the self-test's wait did not give up");
    if (host[2] != 0 || host[3] != 0) return fail(c, MLA_ERR_DEVICE, "a block of the self-test took a share that never came for complete");
    return MLA_OK;
}

int mla_profile_enable(mla_ctx* c, int on)
{
    if (!c) return MLA_ERR_INVALID;
    USE_DEVICE(c);
    if (on && c->prof_events.empty()) {
        c->prof_events.resize(8192);
        for (auto& pe : c->prof_events) {
            CU_TRY(c, cudaEventCreate(&pe.first));
            CU_TRY(c, cudaEventCreate(&pe.second));
        }
    }
    c->profiling = on != 0;
    c->prof_stride = on > 1 ? uint32_t(on) : 1;
    c->prof_seq = 0;
    return MLA_OK;
}

int mla_profile_read(mla_ctx* c, uint32_t* launches, float* total_ms)
{
    if (!c || !launches || !total_ms) return MLA_ERR_INVALID;
    USE_DEVICE(c);
    float sum = 0.0f;
    for (size_t i = 0; i < c->prof_used; i++) {
        CU_TRY(c, cudaEventSynchronize(c->prof_events[i].second));
        float ms = 0.0f;
        CU_TRY(c, cudaEventElapsedTime(&ms, c->prof_events[i].first, c->prof_events[i].second));
        sum += ms;
    }
    *launches = uint32_t(c->prof_used);
    *total_ms = sum;
    c->prof_used = 0;
    return MLA_OK;
}

const char* mla_kernel_name(const mla_ctx* c)
{
    if (!c) return "";
    return c->kernel == MLA_KERNEL_TCGEN05_PAIR128 ? "tcgen05-pair128" : c->kernel == MLA_KERNEL_TCGEN05 ? "tcgen05"
         : c->kernel == MLA_KERNEL_TCGEN05_T16 ? "tcgen05-t16" : "mma";
}

int mla_read_rows(mla_ctx* c, uint32_t layer, uint32_t id, uint32_t row_begin, uint32_t n, void* host_out, void* stream)
{
    if (!c || !host_out) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (int e = check_layer(c, layer, false)) return e;
    const auto* s = c->pt->seq(id);
    if (!s) return fail(c, MLA_ERR_INVALID, "unknown sequence id");
    if (uint64_t(row_begin) + n > uint64_t(s->pages.size()) * mla::kPage)
        return fail(c, MLA_ERR_INVALID, "rows were never appended");
    auto st = static_cast<cudaStream_t>(stream);
    const size_t rb = mla::kRow * 2;
    for (uint32_t r = 0; r < n;) {   // one copy per page run
        const uint32_t row = row_begin + r;
        const uint32_t in_page = std::min<uint32_t>(n - r, mla::kPage - row % mla::kPage);
        CU_TRY(c, cudaMemcpyAsync(static_cast<char*>(host_out) + size_t(r) * rb,
                                  layer_pool(c, layer) + c->pt->slot(id, row) * rb, size_t(in_page) * rb,
                                  cudaMemcpyDeviceToHost, st));
        r += in_page;
    }
    CU_TRY(c, cudaStreamSynchronize(st));
    return MLA_OK;
}

int mla_write_rows(mla_ctx* c, uint32_t layer, uint32_t id, uint32_t row_begin, uint32_t n, const void* dev_rows,
                   void* stream)
{
    if (!c || (n && !dev_rows)) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (int e = check_layer(c, layer, false)) return e;
    if (!c->pt->seq(id)) return fail(c, MLA_ERR_INVALID, "unknown sequence id");
    if (c->in_step) return fail(c, MLA_ERR_STATE, "write_rows is not allowed while a step is open");
    if (int e = pt_code(c, c->pt->reserve(id, row_begin + n))) return e;
    auto st = static_cast<cudaStream_t>(stream);
    std::vector<uint32_t> seqs{id};
    std::vector<RowSpec> none;
    if (int e = build_plan(c, c->plan, kPlanStep, seqs, none, nullptr, nullptr, 0, st)) return e;
    mla::launch_write_rows(dev_rows, layer_pool(c, layer), c->pool_slots, c->plan.m.tables, row_begin, n,
                           c->status_dev, st);
    c->launches += n ? 1 : 0;
    CU_TRY(c, cudaGetLastError());
    return MLA_OK;
}

}  // extern "C"

// ---- attention block: the projections around the op -----------------------------------------------------------
namespace {

// out_i[rows][N_i] = act[rows][K] . W_i[N_i][K]^T, rounded to the storage type; residual: added to what out holds
// norm_w: act's rows go through the RMSNorm first, by way of norm_out where the projection does not do it itself
// exchanged: of the projection before, then of this one (launch_gemm_tc5)
int project(mla_ctx* c, const void* act, uint32_t rows, uint32_t K, std::initializer_list<mla::GemmWeight> weights, bool residual, cudaStream_t st,
            const void* norm_w = nullptr, void* norm_out = nullptr, bool* exchanged = nullptr)
{
    mla::GemmCall g;
    g.A = act;
    g.M = rows;
    g.K = K;
    for (const auto& w : weights) g.w[g.n_weights++] = w;
    g.packed = true;
    g.residual = residual;
    g.norm_w = norm_w;
    g.norm_out = norm_out;
    g.eps = c->cfg.rms_norm_eps;
    g.exchange_near = exchanged && *exchanged;
    const int rc = mla::launch_gemm_tc5(int(c->cfg.dtype), g, c->gemm_ws, c->status_dev, launch_stream(c, st), c->launches, exchanged);
    if (rc == -1) return fail(c, MLA_ERR_INVALID, "projection operands must be 16-byte aligned with row lengths that are multiples of 8");
    if (rc != 0) return fail(c, MLA_ERR_CUDA, std::string("projection launch: ") + cudaGetErrorString(cudaError_t(rc)));
    if (rows) launched(c, st);
    return MLA_OK;
}

int block_of(mla_ctx* c, uint32_t layer, const BlockW** out)
{
    if (layer >= c->cfg.n_layers) return fail(c, MLA_ERR_INVALID, "layer " + std::to_string(layer) + " out of range");
    if (!c->blocks[layer].set) return fail(c, MLA_ERR_STATE, "block weights of layer " + std::to_string(layer) + " were never registered");
    *out = &c->blocks[layer];
    return MLA_OK;
}

int project_in(mla_ctx* c, const BlockW& b, uint32_t rows, const void* hidden, void* q, void* kv_a, cudaStream_t st)
{
    const uint32_t E = b.embed, H = c->cfg.n_heads, QD = H * uint32_t(mla::kQDim);
    if (int e = grow(c, &c->blk_hidden2, &c->blk_hidden2_cap, size_t(rows) * E * 2)) return e;
    const mla::GemmWeight kv = gemm_weight(b.kv_a_map, uint32_t(mla::kRow), kv_a);
    if (!b.q_lora) return project(c, hidden, rows, E, {gemm_weight(b.q_map, QD, q), kv}, false, st, b.attn_norm, c->blk_hidden2);
    if (int e = grow(c, &c->blk_qa, &c->blk_qa_cap, size_t(rows) * b.q_lora * 2)) return e;
    bool exchanged = false;
    if (int e = project(c, hidden, rows, E, {gemm_weight(b.q_a_map, b.q_lora, c->blk_qa), kv}, false, st, b.attn_norm, c->blk_hidden2, &exchanged)) return e;
    return project(c, c->blk_qa, rows, b.q_lora, {gemm_weight(b.q_b_map, QD, q)}, false, st, b.q_a_norm, c->blk_qa, &exchanged);
}

}  // namespace

extern "C" {

int mla_set_block_weights(mla_ctx* c, uint32_t layer, const mla_block_weights* w)
{
    if (!c || !w) return fail(c, MLA_ERR_INVALID, "null argument");
    if (layer >= c->cfg.n_layers) return fail(c, MLA_ERR_INVALID, "layer " + std::to_string(layer) + " out of range");
    USE_DEVICE(c);
    const uint32_t E = w->embedding_length, R = w->q_lora_rank, H = c->cfg.n_heads;
    if (E == 0 || E % 8 || R % 8) return fail(c, MLA_ERR_INVALID, "embedding_length and q_lora_rank must be multiples of 8");
    if (!w->attn_norm || !w->kv_a_mqa || !w->wo || (R ? (!w->q_a || !w->q_a_norm || !w->q_b) : !w->q))
        return fail(c, MLA_ERR_INVALID, "missing projection weight for this q_lora_rank");
    BlockW& b = c->blocks[layer];
    const uint32_t QD = H * uint32_t(mla::kQDim), VD = H * uint32_t(mla::kVDim);
    auto put = [&](void** dst, const void* src, size_t n) -> int {
        if (*dst) { cudaFree(*dst); *dst = nullptr; }
        if (!src) return MLA_OK;
        CU_TRY(c, cudaMalloc(dst, n * 2));
        CU_TRY(c, cudaMemcpy(*dst, src, n * 2, cudaMemcpyHostToDevice));
        return MLA_OK;
    };
    if (int e = ensure_gemm_workspace(c)) return e;
    // matrices are staged row-major, a run of 128-row tiles at a time, and repacked on the device
    void* stage = nullptr;
    constexpr size_t kStageBytes = 32ull << 20;
    auto stage_rows = [&](uint32_t K) { return uint32_t(std::max<size_t>(1, kStageBytes / (size_t(K) * 2 * 128)) * 128); };
    auto stage_bytes = [&](uint32_t N, uint32_t K) { return size_t(std::min(N, stage_rows(K))) * K * 2; };
    CU_TRY(c, cudaMalloc(&stage, std::max({R ? stage_bytes(R, E) : 0, R ? stage_bytes(QD, R) : stage_bytes(QD, E), stage_bytes(uint32_t(mla::kRow), E),
                                           stage_bytes(E, VD)})));
    auto put_matrix = [&](void** dst, mla::GemmWeightMaps* maps, const void* src, uint32_t N, uint32_t K) -> int {
        if (*dst) { cudaFree(*dst); *dst = nullptr; }
        if (!src) return MLA_OK;
        CU_TRY(c, cudaMalloc(dst, mla::gemm_tc5_packed_values(N, K) * 2));
        for (uint32_t r0 = 0, n; r0 < N; r0 += n) {
            n = std::min(N - r0, stage_rows(K));
            CU_TRY(c, cudaMemcpy(stage, static_cast<const char*>(src) + size_t(r0) * K * 2, size_t(n) * K * 2, cudaMemcpyHostToDevice));
            if (int rc = mla::launch_gemm_pack(stage, static_cast<char*>(*dst) + mla::gemm_tc5_packed_values(r0, K) * 2, n, K, nullptr))
                return fail(c, MLA_ERR_CUDA, std::string("weight packing: ") + cudaGetErrorString(cudaError_t(rc)));
        }
        if (!mla::gemm_tc5_packed_maps(maps, int(c->cfg.dtype), *dst, N, K)) return fail(c, MLA_ERR_CUDA, "cuTensorMapEncodeTiled(projection weights) failed");
        return MLA_OK;
    };
    b.set = false;
    int e = put(&b.attn_norm, w->attn_norm, E);
    if (!e) e = put(&b.q_a_norm, R ? w->q_a_norm : nullptr, R);
    if (!e) e = put_matrix(&b.q_a, &b.q_a_map, R ? w->q_a : nullptr, R, E);
    if (!e) e = put_matrix(&b.q_b, &b.q_b_map, R ? w->q_b : nullptr, QD, R);
    if (!e) e = put_matrix(&b.q, &b.q_map, R ? nullptr : w->q, QD, E);
    if (!e) e = put_matrix(&b.kv_a, &b.kv_a_map, w->kv_a_mqa, uint32_t(mla::kRow), E);
    if (!e) e = put_matrix(&b.wo, &b.wo_map, w->wo, E, VD);
    const cudaError_t done = cudaDeviceSynchronize();            // the packing runs on the default stream, the projections need not
    cudaFree(stage);
    if (e) return e;
    CU_TRY(c, done);
    b.embed = E;
    b.q_lora = R;
    b.set = true;
    return MLA_OK;
}

int mla_block_project_in(mla_ctx* c, uint32_t layer, uint32_t rows, const void* hidden, void* q, void* kv_a, void* stream)
{
    if (!c || (rows && (!hidden || !q || !kv_a))) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    const BlockW* b = nullptr;
    if (int e = block_of(c, layer, &b)) return e;
    if (rows == 0) return MLA_OK;
    return project_in(c, *b, rows, hidden, q, kv_a, static_cast<cudaStream_t>(stream));
}

int mla_block_project_out(mla_ctx* c, uint32_t layer, uint32_t rows, const void* attn_out, void* hidden, void* stream)
{
    if (!c || (rows && (!attn_out || !hidden))) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    const BlockW* b = nullptr;
    if (int e = block_of(c, layer, &b)) return e;
    if (rows == 0) return MLA_OK;
    // hidden = hidden + W_o . attn_out
    return project(c, attn_out, rows, c->cfg.n_heads * uint32_t(mla::kVDim), {gemm_weight(b->wo_map, b->embed, hidden)}, true,
                   static_cast<cudaStream_t>(stream));
}

int mla_step_block(mla_ctx* c, uint32_t layer, void* hidden, void* stream)
{
    if (!c || !hidden) return fail(c, MLA_ERR_INVALID, "null argument");
    USE_DEVICE(c);
    if (!c->in_step) return fail(c, MLA_ERR_STATE, "step_block outside step_begin/step_end");
    if (!c->q_rope_in_kernel)
        return fail(c, MLA_ERR_STATE, "the block's q projection is not rotated: enable mla_set_q_rope(ctx, 1) first");
    if (int e = check_layer(c, layer, true)) return e;
    const BlockW* b = nullptr;
    if (int e = block_of(c, layer, &b)) return e;
    auto st = static_cast<cudaStream_t>(stream);
    const uint32_t rows = c->step_rows, H = c->cfg.n_heads;
    if (rows == 0) return MLA_OK;
    const size_t q_bytes = size_t(rows) * H * mla::kQDim * 2, kv_bytes = size_t(rows) * mla::kRow * 2, out_bytes = size_t(rows) * H * mla::kVDim * 2;
    if (int e = grow(c, &c->blk_rows, &c->blk_rows_cap, q_bytes + kv_bytes + out_bytes)) return e;
    char *q = static_cast<char*>(c->blk_rows), *kv = q + q_bytes, *out = kv + kv_bytes;          // rows are multiples of 128 bytes
    if (int e = project_in(c, *b, rows, hidden, q, kv, st)) return e;
    if (int e = run_layer(c, layer, kv, q, out, st)) return e;
    return project(c, out, rows, H * uint32_t(mla::kVDim), {gemm_weight(b->wo_map, b->embed, hidden)}, true, st);
}

}  // extern "C"
