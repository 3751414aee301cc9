// Split-KV absorbed MLA attention for 128-head groups on a PAIR of SMs, 128-token super-tiles
// (thread-block cluster of 2, tcgen05.mma.cta_group::2), sm_100a.
//
// Each block has 64 heads, its 256 latent dims of V, and O^T for its dims x all 128 heads.  A tile is two pages, and the pair's score
// MMA has N = 128: block r stages the whole K of page r (the B operand's rows 64r .. 64r+63).
//
// Shared memory is exactly full (Q' 72 KB, K 72 KB, V 64 KB, P 16 KB, 3 KB of barriers and scratch), so K and V are not double-buffered
// as a whole: every pair of K sub-tiles [64 tokens][2 x 64 dims], the rope sub-tile and every V buffer [page][128-dim chunk] is
// re-loaded as soon as the MMAs that read it have completed.  The dynamic shared segment must start 1 KB-aligned because there is
// no slack to round up (checked; the status word says so if not).
//
// TMEM: O^T 2 x 128 columns; two score tiles of two partial sums of 64 columns, one per issuing warp.  Each accumulator has ONE
// issuing thread and the softmax adds the partials in a fixed order, so the result is bit-reproducible from run to run and under any
// page permutation.
//
// Warps: 0 K producer, 1-2 score issuers (pairs {0,2}, {1,3} and the rope sub-tile), 3-4 value issuers (one per chunk), 5 V producer,
// 6-13 softmax.  The softmax computes its exponentials optimistically against the current reference maximum while the
// cluster round that tells whether any head of the pair must move its maximum is in flight; only in that rare case they are redone
// and O^T rescaled.  Waiting threads sleep in the barrier unit (try_wait with a time hint) rather than re-poll: shared-memory
// bandwidth is what the MMA operand fetches and the TMA fills compete for.  All waits are bounded.
//
// What bounds it, from clock64 marks in a traced build (32 sequences x 8191 tokens): the period of a tile is 2,900 cycles, of which the
// MMAs (36 of 44 cycles, 16 of 77) need 2,816; HBM needs 1.67 us for it, 3,280 cycles at 1.965 GHz.  Before, K was released in three
// rounds of four sub-tiles and the softmax read four partial score tiles, and the period was 3,530: a K load takes 2,200 cycles and
// nothing waited for it but the next tile.  Long lists run into the power cap (SM clock 1.2 to 1.5 GHz) and follow energy
// instead: with a quarter of the score MMAs / of the value MMAs / without the V loads / the exponentials 4 layers of 64 x 16383 take
// 1,144 / 1,165 / 1,229 / 1,276 us instead of 1,305.  Before / now: the kernel alone at full clocks, one layer of 64 x 16384 tokens, 262 /
// 241 us; under the cap 4 layers of 64 x 16383 1,332 to 1,374 / 1,281 to 1,305 on three GPUs, where runs of one side differ by 1 to 5 %; eight
// launches of 8 x 16383 tokens 492 / 468, one sequence of 131,072 tokens 243 / 231 (1.5 % and 2 % of it because no array is
// indexed by the tile's parity and no wait ends with a vote: they sat on the chain from scores to P).
// Not better: K 6 pairs deep with 2 V buffers (period 5,040) or 5 with 3 (3,710), where V, 1,400 cycles from L2, holds P up; the
// other block's V loaded over K pairs that have been read, two tiles in flight (4,010).
#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int PAGES = 2;                            // pages per super-tile
constexpr int TILE = PAGES * kPage;                 // 128 tokens
constexpr int ROWS = 64;                            // rows of a block's operand tiles: tokens of a page, heads
constexpr int NSUB = kRow / 64;                     // 9
constexpr int SUB_BYTES = kPage * 128;              // 8,192: [64 tokens or heads][64 values]
constexpr int Q_BYTES = NSUB * SUB_BYTES;           // 73,728
constexpr int PAIR_BYTES = 2 * SUB_BYTES;           // 16,384: sub-tiles 2i, 2i+1 of a page
constexpr int P_BYTES = ROWS * 128;                 // 8,192 per page
constexpr int PAGE_BYTES = kPage * kRow * 2;
constexpr int OFF_Q = 0;
constexpr int OFF_K = OFF_Q + Q_BYTES;
constexpr int OFF_V = OFF_K + 4 * PAIR_BYTES;                  // [page][chunk]
constexpr int OFF_ROPE = OFF_V + PAGES * 2 * PAIR_BYTES;
constexpr int OFF_P = OFF_ROPE + SUB_BYTES;                 // [page]
constexpr int OFF_MISC = OFF_P + PAGES * P_BYTES;
constexpr int MISC_BYTES = 3072;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES;           // 232,448 = all of it: no alignment slack
static_assert(SMEM_BYTES == 232448, "shared-memory plan must fill the 227 KB exactly");

// misc area layout (bytes from OFF_MISC)
constexpr int M_BAR = 0;          // mbarriers, 8 B each
constexpr int M_TMEM = 384;       // tmem base
constexpr int M_ABORT = 388;
constexpr int M_FLAG = 392;       // [2] "some head of the pair must move its maximum", by tile parity
constexpr int M_ALPHA = 512;      // [2][128] floats: scale factor per head of the pair, by tile parity
constexpr int M_HMAX = 1536;      // [4][64] floats: tile maximum of each token quarter per head
constexpr int M_LSUM = 1536;      // [3][64] floats: the other quarters' partial sums at the epilogue (the same
                                  // bytes as M_HMAX: a barrier of the softmax group separates the two uses)

constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t COL_O = 0;       // 2 chunks x 128 head columns
constexpr uint32_t COL_S = 256;     // 2 score tiles x 2 partial sums x 64 columns

constexpr int N_QK = 2, N_PV = 2;
constexpr int FIRST_SOFTMAX_WARP = 2 + N_QK + N_PV;
constexpr int NUM_THREADS = 32 * (FIRST_SOFTMAX_WARP + 8);
constexpr int SOFTMAX_THREADS = 256;
constexpr int PAIR_SOFTMAX_WARPS = 16;
constexpr float RESCALE_THRESHOLD = 8.0f;

// L2 prefetch (kernel argument prefetch_tiles, 0 = off): every block pulls "its" page towards L2 that many tiles ahead, a quarter
// (contiguous bytes) with every pair it loads.  Only for short work lists: one sequence of 131,072 tokens takes 237 us with it and
// 240 without, 4 layers of 32 x 8191 tokens 375 and 365.
enum { B_QFULL = 0, B_QEMPTY, B_KFULL, B_KEMPTY = B_KFULL + 4, B_VFULL = B_KEMPTY + 4, B_VEMPTY = B_VFULL + 4, B_RFULL = B_VEMPTY + 4,
       B_REMPTY, B_SFULL, B_SEMPTY = B_SFULL + 2, B_PFULL = B_SEMPTY + 2, B_PEMPTY, B_OFULL, B_SYNCA0, B_SYNCA1, B_SYNCB0, B_SYNCB1, B_COUNT };
static_assert(B_COUNT * 8 <= M_TMEM, "barriers overflow their area");


struct SegInfo : SegDesc {
    uint32_t n_pages, n_tiles;
};
__device__ __forceinline__ SegInfo load_seg(const StepMeta& m, uint32_t seg) {
    SegInfo s;
    static_cast<SegDesc&>(s) = load_seg_desc(m.seg + seg);
    s.n_pages = (s.n_tok + kPage - 1) / kPage;
    s.n_tiles = (s.n_pages + PAGES - 1) / PAGES;      // super-tiles
    return s;
}

// HG: heads per block, 64 or 48.  With up to 96 head rows (launch_decode_tc5_pair128) P and O^T have 96 columns instead of 128, which is a
// quarter less for the value MMAs and the states: 80 heads, 4 layers of 32 x 8191 tokens 337 -> 327 us, 64 x 16383 1,290 -> 1,254; 16 heads x 16
// sequences x 5 verify rows 316 -> 309, x 6 331 -> 321; 96 heads 343 -> 335, and no call slower by more than runs differ.
template <typename T, int HG>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
decode_tc5_pair128_kernel(const __grid_constant__ CUtensorMap map_sub, const __grid_constant__ CUtensorMap map_kv64,
                          const __grid_constant__ CUtensorMap map_q, const unsigned char* __restrict__ pool,
                          uint32_t layer0, uint32_t n_pages, StepMeta m, float* __restrict__ recs, uint32_t H,
                          float scale_log2, uint32_t prefetch_tiles, const unsigned char* __restrict__ next_weights,
                          uint32_t next_weights_bytes, uint32_t* __restrict__ status)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t base = smem_u32(sm);
    const uint32_t sQ = base + OFF_Q, sK = base + OFF_K, sV = base + OFF_V, sRope = base + OFF_ROPE, sP = base + OFF_P;
    const uint32_t sBar = base + OFF_MISC + M_BAR;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + M_TMEM);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + M_ABORT);
    volatile uint32_t* need_flag = reinterpret_cast<volatile uint32_t*>(sm + OFF_MISC + M_FLAG);
    float* alpha_all = reinterpret_cast<float*>(sm + OFF_MISC + M_ALPHA);
    float* half_max = reinterpret_cast<float*>(sm + OFF_MISC + M_HMAX);
    float* l_other = reinterpret_cast<float*>(sm + OFF_MISC + M_LSUM);
    auto bar = [&](int i) { return sBar + 8u * uint32_t(i); };

    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t rank = cluster_rank();                 // 0 = pair leader (issues the MMAs)
    const uint32_t worker = blockIdx.x / 2;
    const uint32_t hpair = blockIdx.y * (2 * HG);        // first head of the pair's 128 (96)
    const uint32_t h0 = hpair + rank * HG;               // first head of this block's 64 (48)
    const uint32_t seg_begin = m.cta_seg_begin[worker], seg_end = m.cta_seg_begin[worker + 1];

    // The swizzled operand tiles need 1 KB alignment and the plan leaves no room to round up.
    // Both blocks of a pair see the same offset, so they take this exit together.
    grid_launch_dependents();
    if ((base & 1023u) != 0) {
        grid_dependency_wait();          // also this exit keeps the stream's "every kernel waits before it completes" chain
        if (tid == 0) atomicOr(status, ST_BAD_ALIGNMENT);
        return;
    }

    if (tid == 64) { prefetch_map(&map_q); prefetch_map(&map_sub); prefetch_map(&map_kv64); }
    if (warp == 0) {
        if (lane == 0) {
            *abort_flag = 0;
            need_flag[0] = 0;
            need_flag[1] = 0;
        }
        for (int i = int(lane); i < B_COUNT; i += 32) {
            const uint32_t count = i == B_QEMPTY || i == B_SFULL || i == B_SFULL + 1 ? uint32_t(N_QK)
                                 : i == B_PEMPTY || i == B_OFULL ? uint32_t(N_PV)
                                 : i < B_SEMPTY ? 1u : uint32_t(PAIR_SOFTMAX_WARPS);          // SEMPTY, PFULL, SYNCA0/1, SYNCB0/1
            mbar_init(bar(i), count);
        }
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    // both blocks' barriers must exist before either sends a remote arrive or a TMA completion
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    // The step's metadata is in place when this kernel starts (the rule stands in mla_common.cuh), so it may be
    // read ahead of the wait: the dependent loads that describe the first segment (descriptor -> page ids) then overlap
    // the previous kernel's tail instead of delaying the first TMA.
    SegInfo seg0{};
    const uint32_t* tbl0 = nullptr;
    uint32_t page0[PAGES] = {0, 0};
    if (seg_begin < seg_end) {
        seg0 = load_seg(m, seg_begin);
        tbl0 = m.tables + seg0.tbl;
        if (seg0.n_tiles) {
#pragma unroll
            for (int r = 0; r < PAGES; r++) page0[r] = tbl0[min(uint32_t(r), seg0.n_pages - 1)];
        }
    }
    auto seg_info = [&](uint32_t seg) -> SegInfo { return seg == seg_begin ? seg0 : load_seg(m, seg); };
    auto seg_table = [&](uint32_t seg, const SegInfo& si) -> const uint32_t* {
        return seg == seg_begin ? tbl0 : m.tables + si.tbl;
    };
    auto page_ptr = [&](const SegInfo& si, uint32_t page) -> const unsigned char* {
        return pool + (size_t(layer0 + si.layer) * n_pages + page) * (kPage * kRow * 2);
    };
    // L2 is the point of coherence, so pulling cache lines towards it ahead of the wait is safe even for the page
    // that the append of this layer-step is still writing: the first tiles' loads then find their pages in L2.
    if (warp == N_QK + N_PV + 1 && lane == 0 && seg_begin < seg_end) {
        for (uint32_t jj = 0; jj < min(2u, seg0.n_tiles); jj++) {
            const uint32_t pgid = tbl0[min(PAGES * jj + rank, seg0.n_pages - 1)];
            if (pgid < n_pages) bulk_prefetch_l2(page_ptr(seg0, pgid), kPage * kRow * 2);
        }
    }
    grid_dependency_wait();          // queries, new cache rows and the state records belong to earlier kernels until here

    // Page of super-tile j that block `r` stages as K (and whose tokens are columns 64r .. 64r+63 of
    // the score tile).  A segment with an odd page count repeats its last page in the second half:
    // finite data whose scores the softmax masks.
    auto page_of = [&](const uint32_t* tbl, const SegInfo& s, uint32_t j, uint32_t r) -> uint32_t {
        if (tbl == tbl0 && j == 0) return r ? page0[1] : page0[0];
        const uint32_t i = min(PAGES * j + r, s.n_pages - 1);
        return tbl[i];
    };

    if (warp == 0) {
        // ===================== TMA producer for Q' and K =====================
        if (lane == 0) {
            const uint32_t leader_qfull = map_to_rank(bar(B_QFULL), 0);
            const uint32_t leader_kfull = map_to_rank(bar(B_KFULL), 0), leader_rfull = map_to_rank(bar(B_RFULL), 0);
            uint32_t t = 0, nseg = 0;
            bool ok = true;
            for (uint32_t seg = seg_begin; seg < seg_end && ok; seg++) {
                const SegInfo s = seg_info(seg);
                if (s.n_tiles == 0 || s.heads <= hpair) continue;
                const uint32_t* tbl = seg_table(seg, s);
                ok = mbar_wait<kSleep>(bar(B_QEMPTY), (nseg & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                if (rank == 0) mbar_expect_tx(bar(B_QFULL), 2 * Q_BYTES);
                tma_load_3d_pair(sQ, &map_q, leader_qfull, 0, int(s.q_row * H + h0), 0);      // all 9 sub-tiles at once
                for (uint32_t j = 0; j < s.n_tiles && ok; j++, t++) {
                    uint32_t page = page_of(tbl, s, j, rank);
                    const uint32_t ahead = prefetch_tiles > 0 && j + prefetch_tiles < s.n_tiles ? page_of(tbl, s, j + prefetch_tiles, rank) : n_pages;
                    if (page >= n_pages) {
                        atomicOr(status, ST_BAD_PAGE);
                        page = 0;
                    }
                    const int slot0 = int(page * kPage), layer = int(layer0 + s.layer);
#pragma unroll 1
                    for (uint32_t i = 0; i < 4; i++) {
                        if (ahead < n_pages) bulk_prefetch_l2(page_ptr(s, ahead) + i * (PAGE_BYTES / 4), PAGE_BYTES / 4);
                        ok = mbar_wait<kSleep>(bar(B_KEMPTY + i), (t & 1) ^ 1, abort_flag, status);
                        if (!ok) break;
                        if (rank == 0) mbar_expect_tx(bar(B_KFULL + i), 2 * PAIR_BYTES);
                        tma_load_4d_pair(sK + i * PAIR_BYTES, &map_kv64, leader_kfull + 8 * i, 0, slot0, int(2 * i), layer);
                    }
                    if (!ok) break;
                    ok = mbar_wait<kSleep>(bar(B_REMPTY), (t & 1) ^ 1, abort_flag, status);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(bar(B_RFULL), 2 * SUB_BYTES);
                    tma_load_3d_pair(sRope, &map_sub, leader_rfull, kRank, slot0, layer);
                }
                nseg++;
            }
        }
    } else if (warp == N_QK + N_PV + 1) {
        // ===================== TMA producer for V =====================
        if (lane == 0) {
            const uint32_t leader_vfull = map_to_rank(bar(B_VFULL), 0);
            uint32_t t = 0;
            bool ok = true;
            for (uint32_t seg = seg_begin; seg < seg_end && ok; seg++) {
                const SegInfo s = seg_info(seg);
                if (s.n_tiles == 0 || s.heads <= hpair) continue;
                const uint32_t* tbl = seg_table(seg, s);
                for (uint32_t j = 0; j < s.n_tiles && ok; j++, t++) {
#pragma unroll 1
                    for (uint32_t v = 0; v < 4; v++) {           // page v / 2, chunk v % 2
                        uint32_t page = page_of(tbl, s, j, v / 2);
                        if (page >= n_pages) page = 0;           // flagged by the K producer
                        ok = mbar_wait<kSleep>(bar(B_VEMPTY + v), (t & 1) ^ 1, abort_flag, status);
                        if (!ok) break;
                        if (rank == 0) mbar_expect_tx(bar(B_VFULL + v), 2 * PAIR_BYTES);
                        // all 64 tokens of the page, this block's 128 dims of the chunk = sub-tiles 4 * chunk + 2r, +1
                        tma_load_4d_pair(sV + v * PAIR_BYTES, &map_kv64, leader_vfull + 8 * v, 0, int(page * kPage),
                                         int(4 * (v % 2) + 2 * rank), int(layer0 + s.layer));
                    }
                }
            }
            // This thread's loads are all issued about a tile before the block finishes.  The next kernel but one of
            // the stream (the following layer's absorb) starts by streaming that layer's W_UK from HBM; pulling this
            // block's share of it towards L2 now turns that stream into L2 hits (the bytes move while the last tiles
            // compute and the partial states are merged).  Any thread of the grid could do it; this one is idle.
            if (next_weights != nullptr) {
                const uint32_t nblk = gridDim.x * gridDim.y, me = blockIdx.y * gridDim.x + blockIdx.x;
                const uint32_t share = ((next_weights_bytes + nblk - 1) / nblk + 15u) & ~15u;
                const uint32_t off = me * share;
                if (off < next_weights_bytes) bulk_prefetch_l2(next_weights + off, min(share, next_weights_bytes - off) & ~15u);
            }
        }
    } else if (warp <= N_QK + N_PV) {
        // ===================== MMA issuers (pair leader only) =====================
        if (rank == 0) {
            constexpr uint32_t IDESC_QK = instr_desc(Fmt<T>::v, 128, TILE, 0, 0);        // 64 head rows, 64 tokens per block
            constexpr uint32_t IDESC_PV = instr_desc(Fmt<T>::v, 256, 2 * HG, 1, 0);      // 128 dims per block
            constexpr uint32_t HI = desc_hi(1024);
            const bool is_qk = warp <= N_QK;
            const uint32_t part = is_qk ? warp - 1 : warp - 1 - N_QK;
            const uint32_t qk_a = desc_lo(sQ, 16), pv_b = desc_lo(sP, 16);
            uint32_t t = 0, nseg = 0;
            bool ok = true;
            for (uint32_t seg = seg_begin; seg < seg_end && ok; seg++) {
                const SegInfo s = seg_info(seg);
                if (s.n_tiles == 0 || s.heads <= hpair) continue;
                if (is_qk) ok = mbar_wait<kSleepCluster>(bar(B_QFULL), nseg & 1, abort_flag, status);
                for (uint32_t j = 0; j < s.n_tiles && ok; j++, t++) {
                    if (is_qk) {
                        // score issuer p: pairs p, p + 2, the last one also the rope sub-tile, into its own 64 columns
                        ok = mbar_wait<kSleepCluster>(bar(B_SEMPTY + (t & 1)), ((t >> 1) & 1) ^ 1, abort_flag, status);
                        const uint32_t d = tmem + COL_S + ((t & 1) * N_QK + part) * (TILE / 2);
#pragma unroll
                        for (uint32_t e = 0; e < 4 / N_QK; e++) {
                            const uint32_t i = part + N_QK * e;
                            ok = ok && mbar_wait<kSleep>(bar(B_KFULL + i), t & 1, abort_flag, status);
                            if (!ok) break;
                            tc_fence_after();
                            const uint32_t b0 = desc_lo(sK + i * PAIR_BYTES, 16);
                            if (elect_one()) {
#pragma unroll
                                for (int cc = 0; cc < 2; cc++)
#pragma unroll
                                    for (int k = 0; k < 4; k++)
                                        tc_mma_pair(d, qk_a + (((2 * i + cc) * SUB_BYTES + k * 32) >> 4), HI, b0 + ((cc * SUB_BYTES + k * 32) >> 4),
                                                    HI, IDESC_QK, (e == 0 && cc == 0 && k == 0) ? 0u : 1u);
                                tc_commit_pair(bar(B_KEMPTY + i));
                            }
                            __syncwarp();
                        }
                        if (!ok) break;
                        const bool last = part == uint32_t(N_QK - 1);
                        if (last) {
                            ok = mbar_wait<kSleep>(bar(B_RFULL), t & 1, abort_flag, status);
                            if (!ok) break;
                            tc_fence_after();
                        }
                        const uint32_t br = desc_lo(sRope, 16);
                        if (elect_one()) {
                            if (last) {
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    tc_mma_pair(d, qk_a + ((8 * SUB_BYTES + k * 32) >> 4), HI, br + ((k * 32) >> 4), HI, IDESC_QK, 1u);
                                tc_commit_pair(bar(B_REMPTY));
                            }
                            tc_commit_pair(bar(B_SFULL + (t & 1)));
                            if (j + 1 == s.n_tiles) tc_commit_pair(bar(B_QEMPTY));
                        }
                        __syncwarp();
                    } else {
                        // chunk `part` of O^T += V^T P^T over the tile's two pages
                        ok = mbar_wait<kSleepCluster>(bar(B_PFULL), t & 1, abort_flag, status);
#pragma unroll 1
                        for (uint32_t pg = 0; pg < uint32_t(PAGES) && ok; pg++) {
                            const uint32_t v = 2 * pg + part;
                            ok = mbar_wait<kSleep>(bar(B_VFULL + v), t & 1, abort_flag, status);
                            if (!ok) break;
                            tc_fence_after();
                            const uint32_t a0 = desc_lo(sV + v * PAIR_BYTES, SUB_BYTES);
                            const uint32_t fresh = (j == 0 && pg == 0) ? 0u : 1u;
                            if (elect_one()) {
#pragma unroll
                                for (int k = 0; k < kPage / 16; k++)
                                    tc_mma_pair(tmem + COL_O + part * (2 * HG), a0 + ((k * 2048) >> 4), HI,
                                                pv_b + ((pg * P_BYTES + k * 32) >> 4), HI, IDESC_PV, k == 0 ? fresh : 1u);
                                tc_commit_pair(bar(B_VEMPTY + v));
                                if (pg + 1 == uint32_t(PAGES)) {
                                    tc_commit_pair(bar(B_PEMPTY));
                                    if (j + 1 == s.n_tiles) tc_commit_pair(bar(B_OFULL));
                                }
                            }
                            __syncwarp();
                        }
                    }
                }
                nseg++;
            }
        }
    } else {
        // ===================== softmax / correction / epilogue (both blocks, 8 warps) =====================
        // S of a pair MMA with 64 rows per block: head row r sits in TMEM lane r (tokens of the first
        // page) and lane 64+r (second page), 64 columns each.  Two warps share each lane quarter and
        // split its columns, so a thread owns (head, 32 tokens): token quarter tq = 2*page + group.
        const uint32_t sw_id = warp - FIRST_SOFTMAX_WARP;      // 0..7
        const uint32_t grp = sw_id / 4;                       // column group within the lane quarter
        const uint32_t q4 = warp % 4;
        const uint32_t lane_base = (q4 * 32u) << 16;
        const uint32_t half = q4 / 2;                         // page within the tile
        const uint32_t tq = 2 * half + grp;                   // tokens 32*tq .. 32*tq+31 of the tile
        const uint32_t hl = 32 * (q4 % 2) + lane;             // head within this block's 64
        const uint32_t st_id = tid - (NUM_THREADS - SOFTMAX_THREADS);
        const uint32_t peer = rank ^ 1;
        const uint32_t r_sempty = map_to_rank(bar(B_SEMPTY), 0);          // and the second one 8 bytes on
        const uint32_t r_pfull = map_to_rank(bar(B_PFULL), 0);
        const uint32_t r_synca = map_to_rank(bar(B_SYNCA0), peer), r_syncb = map_to_rank(bar(B_SYNCB0), peer);     // likewise
        const uint32_t r_flag = map_to_rank(base + OFF_MISC + M_FLAG, peer);
        const uint32_t r_alpha = map_to_rank(base + OFF_MISC + M_ALPHA, peer);
        float m_used = -INFINITY, l_part = 0.0f;
        uint32_t t = 0, nseg = 0, na = 0, nb = 0;         // na / nb, bit par: phase of SYNCA[par] / SYNCB[par]
        bool fail = false;
        auto wait_w = [&](uint32_t b, uint32_t parity) {              // completion of tensor-core / TMA work
            fail |= !mbar_wait<kSleep>(b, parity, abort_flag, status);
            __syncwarp();
        };
        auto wait_x = [&](uint32_t b, uint32_t parity) {              // rounds that carry the twin's DSMEM writes
            fail |= !mbar_wait<kSleepCluster>(b, parity, abort_flag, status);
            __syncwarp();
        };
        auto group_or = [&](bool pred) -> bool {              // barrier over this block's softmax threads + OR
            uint32_t r;
            asm volatile(
                "{\n.reg .pred pi, po;\n"
                "setp.ne.b32 pi, %1, 0;\n"
                "barrier.cta.red.or.pred po, 1, 256, pi;\n"
                "selp.u32 %0, 1, 0, po;\n}\n"
                : "=r"(r) : "r"(uint32_t(pred)) : "memory");
            return r != 0;
        };
        bool stop = false;
        for (uint32_t seg = seg_begin; seg < seg_end && !stop; seg++) {
            const SegInfo s = seg_info(seg);
            if (s.heads <= hpair) continue;                   // a smaller group than the plan's largest: none of its rows here
            if (s.n_tiles == 0) {
                // nothing to attend: each block writes its 256 dims of every head, and (m, l) of its own heads
                for (uint32_t h = 0; h < 2 * HG; h++) {
                    if (hpair + h >= s.heads) break;
                    float* rc = recs + (size_t(seg) * m.rec_stride + hpair + h) * kPart;
                    const uint32_t dim = (st_id / 128) * 256 + rank * 128 + (st_id % 128);
                    rc[2 + dim] = 0.0f;
                    if (st_id == 0 && h / HG == rank) { rc[0] = -INFINITY; rc[1] = 0.0f; }
                }
                continue;
            }
            m_used = -INFINITY;
            l_part = 0.0f;
            const bool mine = HG == ROWS || hl < uint32_t(HG);          // with 48 heads the last rows of the score tile are the twin's
            const int lim = mine ? seg_visible(s, h0 + hl, H) : 0;
            for (uint32_t j = 0; j < s.n_tiles; j++, t++) {
                const uint32_t par = t & 1;
                wait_w(bar(B_SFULL + par), (t >> 1) & 1);
                uint32_t sv[32];
                tc_fence_after();
                {
                    uint32_t sw[32];
                    const uint32_t col = tmem + lane_base + COL_S + par * N_QK * (TILE / 2) + grp * 32;
                    tc_ld32(col, sv);
                    tc_ld32(col + TILE / 2, sw);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) sv[i] = __float_as_uint(__uint_as_float(sv[i]) + __uint_as_float(sw[i]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {                       // orders only TMEM reads: no memory release needed
                    if (rank == 0) mbar_arrive(bar(B_SEMPTY + par));
                    else mbar_arrive_cluster_relaxed(r_sempty + 8 * par);
                }
                // Scores stay unscaled in registers: the scale rides in the FMA in front of each exponential, and
                // the mask pass runs only on a segment's last, partly filled tile.
                const int valid = lim - int(j * TILE);
                if (valid < TILE) {
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (int(tq * 32) + i >= valid) sv[i] = __float_as_uint(-INFINITY);
                }
                float mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < 32; i++) mx = fmaxf(mx, __uint_as_float(sv[i]));
                mx *= scale_log2;
                // The first tile of a segment sets every head's reference maximum, but there is no O^T to rescale yet
                // (its PV starts a fresh accumulation), so the twin block has nothing to learn from it: the four
                // token quarters of a head meet inside the block and the two cluster rounds are skipped.  Both blocks
                // of a pair walk the same segments, so they skip the same rounds.
                const bool first = j == 0;
                if (first) {
                    half_max[tq * ROWS + hl] = mx;
                    if (group_or(fail)) { stop = true; break; }
                    m_used = fmaxf(fmaxf(half_max[hl], half_max[ROWS + hl]), fmaxf(half_max[2 * ROWS + hl], half_max[3 * ROWS + hl]));
                }
                // does any head of the pair have to move its reference maximum on this tile?
                const bool need = !first && (mx > m_used + RESCALE_THRESHOLD);
                const bool warp_need = __any_sync(0xffffffffu, need);
                if (lane == 0 && !first) {
                    if (warp_need) {
                        atomicOr(const_cast<uint32_t*>(&need_flag[par]), 1u);
                        asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;\n" ::"r"(r_flag + 4 * par), "r"(1u) : "memory");
                        mbar_arrive_local_release_cluster(bar(B_SYNCA0 + par));
                        mbar_arrive_cluster(r_synca + 8 * par);
                    } else {
                        mbar_arrive(bar(B_SYNCA0 + par));
                        mbar_arrive_cluster_relaxed(r_synca + 8 * par);
                    }
                }
                // a row that has seen no token yet (a segment that only later rows of its group reach): p = 0
                float m_eff = m_used == -INFINITY ? 0.0f : m_used;
                // optimistic: exponentials against the current maximum while the cluster round is in
                // flight; they stand unless some head of the pair raised the flag
                float sum = 0.0f;
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float p0 = fast_ex2(fmaf(__uint_as_float(sv[i]), scale_log2, -m_eff));
                    const float p1 = fast_ex2(fmaf(__uint_as_float(sv[i + 1]), scale_log2, -m_eff));
                    sum += p0 + p1;
                    pk[i / 2] = Elem<T>::pack2(p0, p1);
                }
                bool slow = false;
                if (!first) {
                    wait_x(bar(B_SYNCA0 + par), (na >> par) & 1);
                    na ^= 1u << par;
                    if (group_or(fail)) { stop = true; break; }
                    slow = need_flag[par] != 0;
                }
                if (slow) {
                    // exchange the token quarters' maxima inside the block, decide per head, publish the
                    // scale factors to both blocks, and redo the exponentials
                    float alpha = 1.0f;
                    half_max[tq * ROWS + hl] = mx;
                    group_or(false);
                    // Everyone here has read the flag, and the twin's writes of this round have landed.  It is cleared ahead of this thread's
                    // arrival below: whoever next raises it, two tiles from now, the twin too, has waited for that arrival first.  (The
                    // arrival for P does not order it: on a segment's last tile the twin may pass a first tile, which has no round, and be there.)
                    if (st_id == 0) need_flag[par] = 0;
                    const float mrow = fmaxf(fmaxf(half_max[hl], half_max[ROWS + hl]), fmaxf(half_max[2 * ROWS + hl], half_max[3 * ROWS + hl]));
                    if (mrow > m_used + RESCALE_THRESHOLD) { alpha = fast_ex2(m_used - mrow); m_used = mrow; }
                    if (tq == 0 && mine) {
                        alpha_all[par * 128 + rank * HG + hl] = alpha;
                        asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;\n"
                                     ::"r"(r_alpha + 4 * (par * 128 + rank * HG + hl)), "f"(alpha) : "memory");
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive_local_release_cluster(bar(B_SYNCB0 + par));
                        mbar_arrive_cluster(r_syncb + 8 * par);
                    }
                    wait_x(bar(B_SYNCB0 + par), (nb >> par) & 1);
                    nb ^= 1u << par;
                    l_part *= alpha;
                    m_eff = m_used == -INFINITY ? 0.0f : m_used;
                    sum = 0.0f;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float p0 = fast_ex2(fmaf(__uint_as_float(sv[i]), scale_log2, -m_eff));
                        const float p1 = fast_ex2(fmaf(__uint_as_float(sv[i + 1]), scale_log2, -m_eff));
                        sum += p0 + p1;
                        pk[i / 2] = Elem<T>::pack2(p0, p1);
                    }
                }
                l_part += sum;
                // PV of the previous tile must be complete: O is stable and P is free
                wait_w(bar(B_PEMPTY), (t - 1) & 1);
                tc_fence_after();
                if (slow) {
                    // O^T[this block's dims][128 heads] *= alpha[head]; each warp group takes one chunk
#pragma unroll 1
                    for (int c = 0; c < 2 * HG / 32; c++) {
                        uint32_t o[32];
                        const uint32_t col = COL_O + grp * (2 * HG) + c * 32;
                        tc_ld32(tmem + lane_base + col, o);
                        tc_wait_ld();
                        const float* al = alpha_all + par * 128 + c * 32;
#pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * al[i]);
                        tc_st32(tmem + lane_base + col, o);
                    }
                    tc_wait_st();
                }
                {
                    // row hl of the page's K-major swizzled P tile, this thread's 32 tokens = 16-byte chunks 4*grp .. 4*grp+3
                    unsigned char* prow = sm + OFF_P + half * P_BYTES + hl * 128;
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        const uint4 v = make_uint4(pk[ch * 4], pk[ch * 4 + 1], pk[ch * 4 + 2], pk[ch * 4 + 3]);
                        *reinterpret_cast<uint4*>(prow + (((4 * grp + ch) ^ (hl & 7)) << 4)) = v;
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (rank == 0) mbar_arrive(bar(B_PFULL));
                    else mbar_arrive_remote(r_pfull);
                }
            }
            if (stop) break;
            // ---- epilogue: O^T (this block's 256 dims x 128 heads) -> acc[head][dim]; (m, l) of own heads
            wait_w(bar(B_OFULL), nseg & 1);
            group_or(false);                   // the maxima scratch is free: its bytes now carry the partial sums
            if (tq != 0) l_other[(tq - 1) * ROWS + hl] = l_part;
            if (group_or(fail)) { stop = true; break; }
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 2 * HG / 32; c++) {                      // warp group `grp` owns chunk `grp`
                uint32_t o[32];
                tc_ld32(tmem + lane_base + COL_O + grp * (2 * HG) + c * 32, o);
                tc_wait_ld();
                const uint32_t dim = grp * 256 + rank * 128 + q4 * 32 + lane;
                const uint32_t hb = hpair + c * 32;
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    if (hb + i < s.heads) recs[(size_t(seg) * m.rec_stride + hb + i) * kPart + 2 + dim] = __uint_as_float(o[i]);
                }
            }
            if (tq == 0 && mine && h0 + hl < s.heads) {
                float* rc = recs + (size_t(seg) * m.rec_stride + h0 + hl) * kPart;
                rc[0] = m_used;
                rc[1] = l_part + l_other[hl] + l_other[ROWS + hl] + l_other[2 * ROWS + hl];
            }
            tc_fence_before();
            group_or(false);                   // the scratch is reused by the next segment
            nseg++;
        }
    }

    // Neither block may leave while its twin can still signal its barriers, write its scratch or
    // feed a pair MMA from its shared memory.
    tc_fence_before();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}
}  // namespace

int decode_tc5_pair128_configure()
{
    auto set = [](auto kernel) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        // every kernel of a layer-step asks for the same (maximal) shared-memory carve-out, so the SMs are not
        // re-partitioned between consecutive launches
        return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    };
    cudaError_t e = set(decode_tc5_pair128_kernel<__half, 64>);
    if (e == cudaSuccess) e = set(decode_tc5_pair128_kernel<__half, 48>);
    if (e == cudaSuccess) e = set(decode_tc5_pair128_kernel<__nv_bfloat16, 64>);
    if (e == cudaSuccess) e = set(decode_tc5_pair128_kernel<__nv_bfloat16, 48>);
    return int(e);
}

// tmaps: the context's tensor-map array (kMapPoolSub = one K sub-tile, kMapPoolV = V boxes, kMapQueries = Q').
// pool: the whole cache pool (linear L2 prefetch).
int launch_decode_tc5_pair128(int dtype, const void* tmaps, const void* pool, uint32_t layer0, uint32_t n_pages,
                              const StepMeta& m, float* recs, uint32_t H, uint32_t prefetch_tiles, const void* next_weights,
                              uint32_t next_weights_bytes, uint32_t* status, cudaStream_t st)
{
    if (m.ctas == 0) return 0;
    const CUtensorMap* maps = static_cast<const CUtensorMap*>(tmaps);
    const float scale_log2 = 1.4426950408889634f / sqrtf(float(kQDim));
    const bool narrow = m.rec_stride <= 96;
    dim3 grid(2 * m.ctas, narrow ? 1 : (m.rec_stride + 127) / 128);          // clusters of 2 along x
    auto go = [&](auto kernel) {
        return int(launch_pdl(kernel, grid, dim3(NUM_THREADS), SMEM_BYTES, st, maps[kMapPoolSub], maps[kMapPoolV], maps[kMapQueries],
                              static_cast<const unsigned char*>(pool), layer0, n_pages, m, recs, H, scale_log2, prefetch_tiles,
                              static_cast<const unsigned char*>(next_weights), next_weights_bytes, status));
    };
    if (dtype == 0) return narrow ? go(decode_tc5_pair128_kernel<__half, 48>) : go(decode_tc5_pair128_kernel<__half, 64>);
    return narrow ? go(decode_tc5_pair128_kernel<__nv_bfloat16, 48>) : go(decode_tc5_pair128_kernel<__nv_bfloat16, 64>);
}

}  // namespace mla
