// Split-KV absorbed MLA attention for up to 64 head rows on the 5th-generation tensor cores of sm_100a, in the transposed
// orientation: the tokens of a page are the M rows, the head rows the N columns (NH = 16, 32, 48 or 64 of them).
//
// One persistent block per SM walks its list of KV segments (runs of whole pages of one query group); per page of 64 tokens:
//
//   TMA      page [64 tok][576] -> shared memory as 9 swizzled sub-tiles [64 tok][64 dims]: four pairs into a ring of pair slots,
//            the rope sub-tile into a ring of its own, each slot with its own barriers
//   QK       S^T[64 tok x NH] = K[64 x 576] . Q'^T        36 x tcgen05.mma  M=64  N=NH K=16
//                                A = cache sub-tiles (K-major), B = Q' (K-major)
//   softmax  two groups of four warps, half of the head rows each; a thread holds two tokens of a quarter of its group's rows.  The first
//            page of a segment sets the reference maxima; on later pages the exponentials are computed against them at once and stand
//            unless a vote finds a score more than 2^8 above its reference (then maxima are found, O^T rescaled, exponentials redone)
//   PV       O^T[512 dims x NH] += V^T[512 x 64 tok] . P^T   16 x tcgen05.mma M=128 N=NH K=16
//                                A = the SAME cache sub-tiles read MN-major, B = P^T [NH][64 tok] (K-major)
//
// What bounds it: HBM brings a page to every SM in 1.67 us (73.7 KB x 148 at 6.54 TB/s).  The MMAs of a page take 1,450 (16 rows) to
// 1,920 cycles (64; measured alone an MMA takes the larger of N/2 cycles and its operands' bytes / 128, with 16 columns 3 more).  From the
// request of a pair to the end of the PV MMAs that free its slot it is 5,000 to 7,000 cycles, about 2,300 of them the load; so the pages
// that fit beside Q' and P set the pace where they are few (2.75 pages with 16 rows, 2.5, 2.25, 2 with 64).  A page does not sit in one stage
// buffer: whole-page stages leave one load in flight while the other page is consumed.  With pair slots a score MMA starts as soon as
// its pair has landed and a slot is free as soon as the PV MMAs of its chunk are done.
// 8 layers of 32 sequences x 8191 tokens, bf16, absorb and merge included: 16 heads 410 -> 382 us (0.97 of the HBM rate), 32 heads 567 ->
// 426, 48 heads 547 -> 441, 64 heads 558 -> 502, against a kernel of four warps with a barrier for every maximum (16) and one with the
// heads as M rows and whole-page stages (17 to 64).
//
// Tensor memory: O^T in 4 x NH columns, then the score tiles.
// Warp roles: warp 0 = TMA producer, PARTS warps = score issuers, one = value issuer (warp 1 also owns the tensor memory), eight = softmax,
// correction and epilogue (warp w touches TMEM lanes 32*(w%4) .. +31).
// Output per (segment, head row): m (reference maximum, log2 domain), l, acc[512] — 514 floats.
//
// Every mbarrier wait is bounded: after ~2 s a waiter raises ST_WAIT_TIMEOUT in the status word, sets the block's abort flag and
// every role leaves its loops; TMEM is freed on all paths.
#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int TILE = 64;                          // tokens per tile = one page
constexpr int NSUB = kRow / 64;                   // 9 sub-tiles of 64 dims
constexpr int SUB_BYTES = TILE * 128;             // 8 KB
constexpr int PAIR_BYTES = 2 * SUB_BYTES;         // 16 KB: sub-tiles 2i, 2i+1 of a page
constexpr int PAGE_BYTES = kPage * kRow * 2;
constexpr int MAX_ROWS = 64;
constexpr int MISC_BYTES = 1600;
constexpr int M_TMEM = 304, M_ABORT = 308, M_ALPHA = 320, M_HMAX = 576;   // alpha [NH]; hmax [4][NH], at the end of a segment lsum [4][NH]
static_assert(M_ALPHA + MAX_ROWS * 4 <= M_HMAX && M_HMAX + 4 * MAX_ROWS * 4 <= MISC_BYTES, "scratch overflows its area");
constexpr int SMEM_MAX = 232448;

constexpr int SOFTMAX_WARPS = 8;
constexpr float RESCALE_THRESHOLD = 8.0f;         // log2 units

template <int NH>
struct Plan {
    static constexpr int Q_SUB = NH * 128;                                   // [NH rows][64 dims]
    static constexpr int Q_BYTES = NSUB * Q_SUB;
    static constexpr int P_BYTES = NH * 128;                                 // [NH rows][64 tok]
    static constexpr int SUBS = (SMEM_MAX - MISC_BYTES - Q_BYTES - P_BYTES) / SUB_BYTES;
    // a page takes four pair slots for longer than its rope slot; one rope slot where a second would cost a pair slot
    static constexpr int ROPES = SUBS % 2 ? (SUBS >= 20 ? 3 : 1) : 2;
    static constexpr int PAIRS = (SUBS - ROPES) / 2;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_PAIRS = OFF_Q + Q_BYTES;
    static constexpr int OFF_ROPE = OFF_PAIRS + PAIRS * PAIR_BYTES;
    static constexpr int OFF_P = OFF_ROPE + ROPES * SUB_BYTES;
    static constexpr int OFF_MISC = OFF_P + P_BYTES;
    static constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES;
    // Score-issuing warps, each with partial score tiles of its own that the softmax adds in a fixed order (an accumulator has one issuing
    // thread, so results repeat bit for bit), and score tiles in flight.  One warp issues as fast as the tensor core takes these
    // shapes, but its waits for the four pairs and its code, four times as long, stand one behind the other: with 1 / 2 / 4 issuers 8 layers of
    // 32 x 8191 tokens take 439 / - / 426 us with 32 rows, 468 / 441 / 446 with 48, 522 / 502 / 514 with 64; 27 blocks of 16 heads x 4
    // rows, where a block has a page or two and the instructions come in cold, 714 / 697 / 697.
    static constexpr int PARTS = NH <= 32 ? 4 : 2;
    static constexpr int S_TILES = NH <= 32 ? 1 : 2;
    static constexpr int FIRST_SOFTMAX_WARP = 2 + PARTS;
    static constexpr int NUM_THREADS = 32 * (FIRST_SOFTMAX_WARP + SOFTMAX_WARPS);
    static constexpr uint32_t COL_S = 4 * NH;
    static constexpr uint32_t TMEM_COLS = (4 + S_TILES * PARTS) * NH <= 128 ? 128 : (4 + S_TILES * PARTS) * NH <= 256 ? 256 : 512;
    // barrier slots (8 bytes each)
    enum { B_QFULL = 0, B_QEMPTY, B_KF, B_KE = B_KF + PAIRS, B_RF = B_KE + PAIRS, B_RE = B_RF + ROPES, B_SFULL = B_RE + ROPES,
           B_SEMPTY = B_SFULL + S_TILES, B_PFULL = B_SEMPTY + S_TILES, B_PEMPTY, B_OFULL, B_COUNT };
    static_assert(SMEM_BYTES <= SMEM_MAX && PAIRS >= 6, "shared memory of one block");
    static_assert(OFF_PAIRS % 1024 == 0 && OFF_ROPE % 1024 == 0 && OFF_P % 1024 == 0, "swizzled tiles need 1 KB alignment");
    static_assert((4 + S_TILES * PARTS) * NH <= 512, "tensor memory");
    // A barrier wait names its phase by one bit: an issuer may wait for a slot's next filling only when the one before has landed, although
    // another issuer waited for that one.  It works on page t when all have worked on page t - S_TILES; a filling earlier is PAIRS pairs back.
    static_assert(PAIRS >= 4 * S_TILES, "phases of the pair ring");
    static_assert(B_COUNT * 8 <= M_TMEM, "barriers overflow their area");
};

struct SegInfo : SegDesc {
    uint32_t n_tiles;
};

__device__ __forceinline__ SegInfo load_seg(const StepMeta& m, uint32_t seg) {
    SegInfo s;
    static_cast<SegDesc&>(s) = load_seg_desc(m.seg + seg);
    s.n_tiles = (s.n_tok + TILE - 1) / TILE;
    return s;
}

// N columns of 16 TMEM lanes (16x256b): block k of 8 columns gives registers 4k..4k+3 = (lane i/4, columns 8k + 2(i%4), +1), then
// (lane i/4 + 8, the same columns)
template <int N>
__device__ __forceinline__ void load_scores(uint32_t taddr, uint32_t (&r)[N / 2]) {
    constexpr int B = N / 8;
    constexpr int at2 = B & 4, at1 = B & 6;
    if constexpr (B & 4) tc_ld16x256(taddr, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
    if constexpr (B & 2) tc_ld16x256(taddr + 8 * at2, *reinterpret_cast<uint32_t(*)[8]>(&r[4 * at2]));
    if constexpr (B & 1) tc_ld16x256(taddr + 8 * at1, *reinterpret_cast<uint32_t(*)[4]>(&r[4 * at1]));
}

template <typename T, int NH>
__global__ void __launch_bounds__(Plan<NH>::NUM_THREADS, 1)
decode_tc5_kernel(const __grid_constant__ CUtensorMap map_pair, const __grid_constant__ CUtensorMap map_sub,
                  const __grid_constant__ CUtensorMap map_q, const unsigned char* __restrict__ pool, uint32_t layer0, uint32_t n_pages,
                  StepMeta m, float* __restrict__ recs, uint32_t H, float scale_log2, uint32_t* __restrict__ status)
{
    using L = Plan<NH>;
    constexpr int PAIRS = L::PAIRS, ROPES = L::ROPES, PARTS = L::PARTS, S_TILES = L::S_TILES, FIRST_SOFTMAX_WARP = L::FIRST_SOFTMAX_WARP;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t base = smem_u32(sm);
    const uint32_t sQ = base + L::OFF_Q, sPairs = base + L::OFF_PAIRS, sRope = base + L::OFF_ROPE, sP = base + L::OFF_P;
    const uint32_t sBar = base + L::OFF_MISC;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L::OFF_MISC + M_TMEM);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L::OFF_MISC + M_ABORT);
    float* alpha_s = reinterpret_cast<float*>(sm + L::OFF_MISC + M_ALPHA);
    float* hmax_s = reinterpret_cast<float*>(sm + L::OFF_MISC + M_HMAX);
    auto bar = [&](int i) { return sBar + 8u * uint32_t(i); };

    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t cta = blockIdx.x, h0 = blockIdx.y * NH;
    const uint32_t seg_begin = m.cta_seg_begin[cta], seg_end = m.cta_seg_begin[cta + 1];

    grid_launch_dependents();
    if ((base & 1023u) != 0) {           // the swizzled tiles need it and the plan leaves no room to round up
        grid_dependency_wait();          // also this exit keeps the stream's "every kernel waits before it completes" chain
        if (tid == 0) atomicOr(status, ST_BAD_ALIGNMENT);
        return;
    }
    if (tid == 64) { prefetch_map(&map_q); prefetch_map(&map_pair); prefetch_map(&map_sub); }
    if (warp == 0) {
        if (lane == 0) *abort_flag = 0;
        for (int i = int(lane); i < L::B_COUNT; i += 32) mbar_init(bar(i), i >= L::B_SEMPTY && i <= L::B_PFULL ? SOFTMAX_WARPS : i == L::B_QEMPTY || (i >= L::B_SFULL && i < L::B_SEMPTY) ? PARTS : 1);
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc<L::TMEM_COLS>(tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    // The first pages of the block's first segment towards L2 while the absorb launch ends: L2 is the point of coherence, so this is
    // safe even for the page that the append is still writing.  8 layers of 64 heads x 16 sequences, one launch series each: 375 ->
    // 365 us.  The first segment's descriptor is read here too, not behind the wait (the step's metadata is in place when this kernel
    // starts: the rule stands in mla_common.cuh).
    SegInfo seg0{};
    if (seg_begin < seg_end) seg0 = load_seg(m, seg_begin);
    auto seg_info = [&](uint32_t seg) -> SegInfo { return seg == seg_begin ? seg0 : load_seg(m, seg); };
    auto page_at = [&](const SegInfo& s, uint32_t page) { return pool + (size_t(layer0 + s.layer) * n_pages + page) * PAGE_BYTES; };
    if (warp == 0 && lane == 0 && seg_begin < seg_end) {
        const SegInfo& s = seg0;
        for (uint32_t j = 0; j < min(2u, s.n_tiles); j++) {
            const uint32_t page = m.tables[s.tbl + j];
            if (page < n_pages) bulk_prefetch_l2(page_at(s, page), PAGE_BYTES);
        }
    }
    // queries, new cache rows and the state records belong to earlier kernels of the stream, which may still run
    grid_dependency_wait();

    if (warp == 0) {
        // ===================== TMA producer =====================
        if (lane == 0) {
            uint32_t ps = 0, pph = 1, rs = 0, rph = 1, nseg = 0;         // next pair / rope slot and the parity that says it is free
            bool ok = true;
            for (uint32_t seg = seg_begin; seg < seg_end && ok; seg++) {
                const SegInfo s = seg_info(seg);
                if (s.n_tiles == 0 || s.heads <= h0) continue;
                ok = mbar_wait(bar(L::B_QEMPTY), (nseg & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                mbar_expect_tx(bar(L::B_QFULL), L::Q_BYTES);
                tma_load_3d(sQ, &map_q, bar(L::B_QFULL), 0, int(s.q_row * H + h0), 0);          // all 9 sub-tiles in one box
                const uint32_t* tbl = m.tables + s.tbl;
                for (uint32_t j = 0; j < s.n_tiles && ok; j++) {
                    uint32_t page = tbl[j];
                    const uint32_t next = j + 1 < s.n_tiles ? tbl[j + 1] : n_pages;
                    if (page >= n_pages) {
                        atomicOr(status, ST_BAD_PAGE);
                        page = 0;
                    }
#pragma unroll 1
                    for (int i = 0; i < 4; i++) {
                        // a quarter of the next page towards L2 (contiguous bytes, not this pair's)
                        if (next < n_pages) bulk_prefetch_l2(page_at(s, next) + i * (PAGE_BYTES / 4), PAGE_BYTES / 4);
                        ok = mbar_wait(bar(L::B_KE + ps), pph, abort_flag, status);
                        if (!ok) break;
                        mbar_expect_tx(bar(L::B_KF + ps), PAIR_BYTES);
                        tma_load_4d(sPairs + ps * PAIR_BYTES, &map_pair, bar(L::B_KF + ps), 0, int(page * kPage), 2 * i, int(layer0 + s.layer));
                        if (++ps == PAIRS) { ps = 0; pph ^= 1; }
                    }
                    if (!ok) break;
                    ok = mbar_wait(bar(L::B_RE + rs), rph, abort_flag, status);
                    if (!ok) break;
                    mbar_expect_tx(bar(L::B_RF + rs), SUB_BYTES);
                    tma_load_3d(sRope + rs * SUB_BYTES, &map_sub, bar(L::B_RF + rs), kRank, int(page * kPage), int(layer0 + s.layer));
                    if (++rs == ROPES) { rs = 0; rph ^= 1; }
                }
                nseg++;
            }
        }
    } else if (warp < FIRST_SOFTMAX_WARP) {
        // ===================== MMA issuers =====================
        // A warp runs the loop uniformly (operands stay in uniform registers) and one elected lane issues.
        constexpr uint32_t IDESC_QK = instr_desc(Fmt<T>::v, TILE, NH, 0, 0);          // M = 64 tokens
        constexpr uint32_t IDESC_PV = instr_desc(Fmt<T>::v, 128, NH, 1, 0);
        constexpr uint32_t HI = desc_hi(1024);          // every operand: 8-row groups 1024 B apart
        const bool is_qk = warp <= uint32_t(PARTS);
        const uint32_t part = warp - 1;
        const uint32_t qk_b = desc_lo(sQ, 16), pv_b = desc_lo(sP, 16);
        // slot and phase of the page's first pair, of its rope sub-tile, and the score tile with the parity that says it is free
        uint32_t t = 0, nseg = 0, ps = 0, pph = 0, rs = 0, rph = 0, sb = 0, sph = 1;
        bool ok = true;
        for (uint32_t seg = seg_begin; seg < seg_end && ok; seg++) {
            const SegInfo s = seg_info(seg);
            if (s.n_tiles == 0 || s.heads <= h0) continue;
            if (is_qk) ok = mbar_wait(bar(L::B_QFULL), nseg & 1, abort_flag, status);
            for (uint32_t j = 0; j < s.n_tiles && ok; j++, t++) {
                if (is_qk) {
                    // score issuer i: pairs i * 4 / PARTS on; the last one also the rope sub-tile
                    constexpr uint32_t EACH = 4 / PARTS;
                    ok = mbar_wait(bar(L::B_SEMPTY + sb), sph, abort_flag, status);
                    const uint32_t d = tmem + L::COL_S + (sb * PARTS + part) * NH;
#pragma unroll
                    for (uint32_t e = 0; e < EACH; e++) {
                        const uint32_t i = part * EACH + e;
                        uint32_t slot = ps + i, ph = pph;
                        if (slot >= uint32_t(PAIRS)) { slot -= PAIRS; ph ^= 1; }
                        ok = ok && mbar_wait(bar(L::B_KF + slot), ph, abort_flag, status);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t a0 = desc_lo(sPairs + slot * PAIR_BYTES, 16);
                        if (elect_one()) {
#pragma unroll
                            for (int cc = 0; cc < 2; cc++)
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    tc_mma(d, a0 + ((cc * SUB_BYTES + k * 32) >> 4), HI, qk_b + (((2 * i + cc) * L::Q_SUB + k * 32) >> 4), HI,
                                           IDESC_QK, (e == 0 && cc == 0 && k == 0) ? 0u : 1u);
                        }
                        __syncwarp();
                    }
                    if (!ok) break;
                    const bool last = part == uint32_t(PARTS - 1);
                    if (last) {
                        ok = mbar_wait(bar(L::B_RF + rs), rph, abort_flag, status);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const uint32_t ar = desc_lo(sRope + rs * SUB_BYTES, 16);
                    if (elect_one()) {
                        if (last) {
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                tc_mma(d, ar + ((k * 32) >> 4), HI, qk_b + ((8 * L::Q_SUB + k * 32) >> 4), HI, IDESC_QK, 1u);
                            tc_commit(bar(L::B_RE + rs));
                        }
                        tc_commit(bar(L::B_SFULL + sb));
                        if (j + 1 == s.n_tiles) tc_commit(bar(L::B_QEMPTY));
                    }
                    __syncwarp();
                    if (++rs == ROPES) { rs = 0; rph ^= 1; }
                    if (++sb == S_TILES) { sb = 0; sph ^= 1; }
                } else {
                    // chunks of O^T = pairs of the page read MN-major.  The pairs have landed: P exists only after the score issuer
                    // waited for them.
                    ok = mbar_wait(bar(L::B_PFULL), t & 1, abort_flag, status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t fresh = j == 0 ? 0u : 1u;
                    if (elect_one()) {
#pragma unroll 1
                        for (uint32_t c = 0; c < 4; c++) {
                            const uint32_t slot = ps + c >= uint32_t(PAIRS) ? ps + c - PAIRS : ps + c;
                            const uint32_t a0 = desc_lo(sPairs + slot * PAIR_BYTES, SUB_BYTES);
#pragma unroll
                            for (int k = 0; k < TILE / 16; k++)
                                tc_mma(tmem + c * NH, a0 + ((k * 2048) >> 4), HI, pv_b + ((k * 32) >> 4), HI, IDESC_PV, k == 0 ? fresh : 1u);
                            tc_commit(bar(L::B_KE + slot));
                        }
                        tc_commit(bar(L::B_PEMPTY));
                        if (j + 1 == s.n_tiles) tc_commit(bar(L::B_OFULL));
                    }
                    __syncwarp();
                }
                ps += 4;
                if (ps >= uint32_t(PAIRS)) { ps -= PAIRS; pph ^= 1; }
            }
            nseg++;
        }
    } else {
        // ===================== softmax / correction / epilogue =====================
        // S^T (M=64 layout) keeps token rows 16q .. 16q+15 in TMEM lanes 0-15 of sub-partition q.  A 16x256b load spreads them over
        // the warp: thread i holds tokens 16q + i/4 and + 8 of columns 8k + 2(i%4), +1 for every block k of 8 head rows.
        // The groups of four warps share nothing but the barriers of the issuers.  A failed (timed-out / aborted) wait never makes
        // a thread leave early on its own: it goes on, with whatever is there, to the group's next barrier, where failures are OR-reduced
        // and the group's 128 threads leave together.
        constexpr int NW = NH / 2, NB = NW / 8, NV = 2 * NB;  // head columns, blocks of them and head rows per thread of a group
        const uint32_t q4 = warp % 4;                         // TMEM sub-partition of this warp
        const uint32_t grp = (warp - FIRST_SOFTMAX_WARP) / 4;
        const uint32_t lane_base = (q4 * 32u) << 16;
        const uint32_t qd = lane & 3, tr = lane >> 2;         // column pair within a block, token row within the warp's 16 (and + 8)
        auto head_of = [&](int v) { return uint32_t(grp * NW + 8 * (v >> 1) + 2 * qd + (v & 1)); };
        const uint32_t tok_a = 16 * q4 + tr;
        // where this lane's row of a stored 8 x 8 block lies: blocks come as (k, tokens 0-7), (k, 8-15), (k+1, 0-7), (k+1, 8-15)
        const uint32_t p_row = sP + (grp * NW + 8 * (lane >> 4) + (lane & 7)) * 128 + (((2 * q4 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4);
        // References are scores as they are, unscaled, so that the difference to the largest one is exactly 0 however large they are: with the scale
        // in an FMA against a scaled reference it was the rounding of that, beyond 2^32 an exponential of infinity or 0 (and no faster).
        float m_ref[NV], psum[NV];                            // m_ref: 0 for the rows of `none`, whose reference is -infinity
        uint32_t none = 0, t = 0, nseg = 0, sb = 0, sph = 0;
        float over_by = RESCALE_THRESHOLD;
        bool fail = false;
        auto wait_w = [&](uint32_t b, uint32_t parity) {
            fail |= !mbar_wait(b, parity, abort_flag, status);
            __syncwarp();
        };
        auto group_or = [&](bool pred) -> bool {              // barrier over the group's 128 threads + OR
            uint32_t r;
            asm volatile(
                "{\n.reg .pred pi, po;\n"
                "setp.ne.b32 pi, %1, 0;\n"
                "barrier.cta.red.or.pred po, %2, 128, pi;\n"
                "selp.u32 %0, 1, 0, po;\n}\n"
                : "=r"(r) : "r"(uint32_t(pred)), "r"(1 + grp) : "memory");
            return r != 0;
        };
        uint32_t sv[NW / 2];                                  // scores, unscaled: sv[4k + 2e' + e]: head 8k + 2qd + e, token tok_a + 8e'
        auto publish_max = [&] {                              // maxima of this warp's 16 tokens
#pragma unroll
            for (int v = 0; v < NV; v++) {
                float x = fmaxf(__uint_as_float(sv[4 * (v >> 1) + (v & 1)]), __uint_as_float(sv[4 * (v >> 1) + 2 + (v & 1)]));
                x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 4));
                x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 8));
                x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 16));
                if (tr == 0) hmax_s[q4 * NH + head_of(v)] = x;
            }
        };
        auto tile_max = [&](int v) {
            const float* hm = hmax_s + head_of(v);
            return fmaxf(fmaxf(hm[0], hm[NH]), fmaxf(hm[2 * NH], hm[3 * NH]));
        };
        uint32_t pk[NW / 4];                                  // pk[2k + e']: the two head rows of block k, token tok_a + 8e'
        float add[NV];
        auto exponentials = [&]() -> bool {                   // true: some score lies too far above its reference
            float top = -INFINITY;
#pragma unroll
            for (int k = 0; k < NB; k++) {
                float p[4];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float me = m_ref[2 * k + e];
                    const float xa = (__uint_as_float(sv[4 * k + e]) - me) * scale_log2, xb = (__uint_as_float(sv[4 * k + 2 + e]) - me) * scale_log2;
                    top = fmaxf(top, fmaxf(xa, xb));
                    p[e] = fast_ex2(xa);
                    p[2 + e] = fast_ex2(xb);
                    add[2 * k + e] = p[e] + p[2 + e];
                }
                pk[2 * k] = Elem<T>::pack2(p[0], p[1]);
                pk[2 * k + 1] = Elem<T>::pack2(p[2], p[3]);
            }
            return top > over_by;
        };
        // A row without a maximum (one that sees no token of the segment, or only scores of -infinity so far) has p = 0 against a reference of
        // 0.  Its thread takes the slow path on every page with a score above -infinity, so that the row's first one becomes its reference.
        auto set_ref = [&](int v, float mt) {
            const bool empty = mt == -INFINITY;
            m_ref[v] = empty ? 0.0f : mt;
            none = (none & ~(1u << v)) | (uint32_t(empty) << v);
        };
        bool stop = false;
        for (uint32_t seg = seg_begin; seg < seg_end && !stop; seg++) {
            const SegInfo s = seg_info(seg);
            if (s.heads <= h0) continue;                      // a smaller group than the plan's largest: none of its rows here
            if (s.n_tiles == 0) {
                // nothing to attend: the state of an empty range
                const uint32_t st = tid - 32 * FIRST_SOFTMAX_WARP;
                for (uint32_t h = 0; h < uint32_t(NH); h++) {
                    if (h0 + h >= s.heads) break;
                    float* rc = recs + (size_t(seg) * m.rec_stride + h0 + h) * kPart;
                    for (uint32_t d = st; d < kRank; d += 32 * SOFTMAX_WARPS) rc[2 + d] = 0.0f;
                    if (st == 0) { rc[0] = -INFINITY; rc[1] = 0.0f; }
                }
                continue;
            }
#pragma unroll
            for (int v = 0; v < NV; v++) psum[v] = 0.0f;
            none = 0;
            const int lim_first = seg_visible(s, 0, H);       // the group's first row sees the fewest tokens
            for (uint32_t j = 0; j < s.n_tiles; j++, t++) {
                const bool cut = int(j * TILE) + TILE > lim_first;       // some row does not see all of this page
                int valid[NV];
                if (cut) {
#pragma unroll
                    for (int v = 0; v < NV; v++) valid[v] = seg_visible(s, h0 + head_of(v), H) - int(j * TILE);
                }
                wait_w(bar(L::B_SFULL + sb), sph);
                tc_fence_after();
                {
                    uint32_t part_s[PARTS][NW / 2];
#pragma unroll
                    for (int p = 0; p < PARTS; p++) load_scores<NW>(tmem + lane_base + L::COL_S + (sb * PARTS + p) * NH + grp * NW, part_s[p]);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < NW / 2; i++) {
                        float x = __uint_as_float(part_s[0][i]);
#pragma unroll
                        for (int p = 1; p < PARTS; p++) x += __uint_as_float(part_s[p][i]);
                        sv[i] = __float_as_uint(x);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(L::B_SEMPTY + sb));
                if (++sb == S_TILES) { sb = 0; sph ^= 1; }
                if (cut) {
#pragma unroll
                    for (int v = 0; v < NV; v++) {
                        if (int(tok_a) >= valid[v]) sv[4 * (v >> 1) + (v & 1)] = __float_as_uint(-INFINITY);
                        if (int(tok_a) + 8 >= valid[v]) sv[4 * (v >> 1) + 2 + (v & 1)] = __float_as_uint(-INFINITY);
                    }
                }
                bool slow = false;
                if (j == 0) {
                    publish_max();
                    if (group_or(fail)) { stop = true; break; }
                    // a column beyond the group's rows has scores of nobody: no exponential, no vote
#pragma unroll
                    for (int v = 0; v < NV; v++) set_ref(v, h0 + head_of(v) < s.heads ? tile_max(v) : INFINITY);
                    over_by = none ? -INFINITY : RESCALE_THRESHOLD;
                    exponentials();
                } else {
                    slow = group_or(exponentials() || fail);
                    if (slow) {
                        if (group_or(fail)) { stop = true; break; }
                        publish_max();
                        group_or(false);
#pragma unroll
                        for (int v = 0; v < NV; v++) {
                            const float mt = tile_max(v), mr = (none >> v) & 1 ? -INFINITY : m_ref[v];
                            float alpha = 1.0f;
                            const float up = (mt - mr) * scale_log2;
                            if (up > RESCALE_THRESHOLD) { alpha = fast_ex2(-up); set_ref(v, mt); }
                            psum[v] *= alpha;
                            if (q4 == 0 && tr == 0) alpha_s[head_of(v)] = alpha;
                        }
                        over_by = none ? -INFINITY : RESCALE_THRESHOLD;
                        exponentials();
                    }
                }
#pragma unroll
                for (int v = 0; v < NV; v++) psum[v] += add[v];
                // PV of the previous tile must be complete: O is stable and P is free
                wait_w(bar(L::B_PEMPTY), (t - 1) & 1);
                if (slow) {
                    if (group_or(fail)) { stop = true; break; }
                    tc_fence_after();
                    // O^T[dim lane][head column] *= alpha[head], this group's columns
#pragma unroll 1
                    for (int c = 0; c < 4 * NB; c++) {
                        uint32_t o[8];
                        const uint32_t hc = grp * NW + (c % NB) * 8, col = tmem + lane_base + (c / NB) * NH + hc;
                        tc_ld8(col, o);
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha_s[hc + i]);
                        tc_st8(col, o);
                    }
                    tc_wait_st();
                }
                // P^T [NH][64 tok], K-major with the 128-byte swizzle: row = head, 16-byte chunk = tok / 8
#pragma unroll
                for (int k = 0; k + 1 < NB; k += 2) store_matrix_t4(p_row + k * 1024, pk[2 * k], pk[2 * k + 1], pk[2 * k + 2], pk[2 * k + 3]);
                if constexpr (NB & 1) store_matrix_t2(p_row + (NB - 1) * 1024, pk[2 * NB - 2], pk[2 * NB - 1]);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(L::B_PFULL));
            }
            if (stop) break;
            // ---- epilogue of the segment: O^T -> acc[head][dim], plus (m, l).  Every warp has read the maxima when PV is done.
            wait_w(bar(L::B_OFULL), nseg & 1);
#pragma unroll
            for (int v = 0; v < NV; v++) {
                float x = psum[v];
                x += __shfl_xor_sync(0xffffffffu, x, 4);
                x += __shfl_xor_sync(0xffffffffu, x, 8);
                x += __shfl_xor_sync(0xffffffffu, x, 16);
                if (tr == 0) hmax_s[q4 * NH + head_of(v)] = x;
            }
            if (group_or(fail)) { stop = true; break; }
            tc_fence_after();
            const size_t rec = size_t(seg) * m.rec_stride + h0;
            constexpr int TRIP = NW <= 16 ? 4 : NW <= 32 ? 2 : 1;          // chunks per trip to tensor memory
#pragma unroll 1
            for (int c0 = 0; c0 < 4; c0 += TRIP) {
                uint32_t o[TRIP][NW];
#pragma unroll
                for (int c = 0; c < TRIP; c++) tc_ld_columns<NW>(tmem + lane_base + (c0 + c) * NH + grp * NW, o[c]);
                tc_wait_ld();
                float* rc = recs + (rec + grp * NW) * kPart + 2 + c0 * 128 + q4 * 32 + lane;
#pragma unroll
                for (int i = 0; i < NW; i++) {
                    if (h0 + grp * NW + i >= s.heads) break;
#pragma unroll
                    for (int c = 0; c < TRIP; c++) rc[i * kPart + c * 128] = __uint_as_float(o[c][i]);
                }
            }
            if (q4 == 0 && tr == 0) {
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const uint32_t h = head_of(v);
                    if (h0 + h < s.heads) {
                        float* rc = recs + (rec + h) * kPart;
                        rc[0] = (none >> v) & 1 ? -INFINITY : m_ref[v] * scale_log2;
                        rc[1] = (hmax_s[h] + hmax_s[NH + h]) + (hmax_s[2 * NH + h] + hmax_s[3 * NH + h]);
                    }
                }
            }
            // the scratch and the score / O columns are reused by the next segment: everyone is done reading
            if (seg + 1 < seg_end) group_or(false);
            tc_fence_before();
            nseg++;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<L::TMEM_COLS>(tmem);
    }
}

template <typename T, int NH>
int configure()
{
    return int(cudaFuncSetAttribute(decode_tc5_kernel<T, NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, Plan<NH>::SMEM_BYTES));
}
template <typename T>
int configure_all()
{
    for (int e : {configure<T, 16>(), configure<T, 32>(), configure<T, 48>(), configure<T, 64>()})
        if (e) return e;
    return 0;
}

template <typename T, int NH>
int launch(const CUtensorMap* maps, const unsigned char* pool, uint32_t layer0, uint32_t n_pages, const StepMeta& m, float* recs, uint32_t H,
           uint32_t* status, cudaStream_t st)
{
    const float scale_log2 = 1.4426950408889634f / sqrtf(float(kQDim));
    return int(launch_pdl(decode_tc5_kernel<T, NH>, dim3(m.ctas, (m.rec_stride + NH - 1) / NH), dim3(Plan<NH>::NUM_THREADS), Plan<NH>::SMEM_BYTES, st,
                          maps[kMapPoolV], maps[kMapPoolSub], maps[query_map(NH)], pool, layer0, n_pages, m, recs, H, scale_log2, status));
}
template <typename T>
int launch_for(uint32_t columns, const CUtensorMap* maps, const unsigned char* pool, uint32_t layer0, uint32_t n_pages, const StepMeta& m,
               float* recs, uint32_t H, uint32_t* status, cudaStream_t st)
{
    switch (columns) {
    case 16: return launch<T, 16>(maps, pool, layer0, n_pages, m, recs, H, status, st);
    case 32: return launch<T, 32>(maps, pool, layer0, n_pages, m, recs, H, status, st);
    case 48: return launch<T, 48>(maps, pool, layer0, n_pages, m, recs, H, status, st);
    default: return launch<T, 64>(maps, pool, layer0, n_pages, m, recs, H, status, st);
    }
}

}  // namespace

int decode_tc5_configure(int dtype) { return dtype == 0 ? configure_all<__half>() : configure_all<__nv_bfloat16>(); }

int launch_decode_tc5(int dtype, uint32_t columns, const void* tmaps, const void* pool, uint32_t layer0, uint32_t n_pages, const StepMeta& m,
                      float* recs, uint32_t H, uint32_t* status, cudaStream_t st)
{
    if (m.ctas == 0) return 0;
    const CUtensorMap* maps = static_cast<const CUtensorMap*>(tmaps);
    const auto* pl = static_cast<const unsigned char*>(pool);
    return dtype == 0 ? launch_for<__half>(columns, maps, pl, layer0, n_pages, m, recs, H, status, st)
                      : launch_for<__nv_bfloat16>(columns, maps, pl, layer0, n_pages, m, recs, H, status, st);
}

}  // namespace mla
