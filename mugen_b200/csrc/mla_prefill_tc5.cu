// Causal attention of a prefill chunk on the 5th-generation tensor cores, sm_100a.
//
// The reference runs its absorbed routine once per chunk token with a growing length (src/core/model/
// transformer.cpp:1325-1337: token t of a chunk appended at start_position attends rows [0, start_position + t + 1)).
// Any mathematically equal form within the attention tolerance may stand in for it; for MANY query tokens over the
// same cache the cheap form is the expanded one: the latent rows are expanded ONCE per layer into per-head keys and
// values with the same weights,
//     k[t][h] = ( W_UK_h . c_kv[t]  (128 dims) , k_rope[t] (64 dims, shared by all heads) ),   v[t][h] = W_UV_h . c_kv[t],
// (two dense projections, mla_gemm_tc5.cu), and every (128 query tokens x one head) tile then runs flash attention
// over 192-dim keys and 128-dim values: 2 x (192 + 128) flops per (query, key, head) pair instead of the absorbed
// form's 2 x (576 + 512), and each staged key/value tile serves 128 query tokens instead of one.
//
// One block per (tile of 128 query tokens, head); scores, probabilities and the output accumulate in tensor memory:
//   Q        [128 queries][192 dims] rotated and written once into shared memory by the softmax threads
//   TMA      per step of KT = 128 keys K [128][192] (two boxes of expanded nope dims + the rope dims straight from the two
//            cache pages) and V [128][128], rings of two each, every ring with a thread of its own (one thread for both starts
//            K of step t + 1 only after the PV of step t - 2 has freed V's buffer: 2,300 instead of 1,850 cycles per step);
//            a K buffer is free as soon as the score MMAs that read it complete, a V buffer one softmax later
//   QK       S[128 queries x 128 keys] = Q . K^T         12 x tcgen05.mma M128 N128 K16, two score tiles in flight; a tile is
//            free for the step after next as soon as its group has loaded it into registers (P has columns of its own: with Q
//            in tensor memory there is no room for them, P overwrites its scores and QK of step t + 2 waits for PV of step t)
//   softmax  two groups of four warps take the key steps in turn (group g: steps g, g + 2, ..), one thread per query row and
//            all 128 keys of it, so that one group's exponentials run while the other waits for its scores or stores P.
//            Causal mask, log2-domain online softmax with lazy rescaling (threshold 2^8).  What a step needs from the one
//            before is the row's reference maximum alone (one float through shared memory, warp to warp); every group sums
//            its own steps' probabilities and the epilogue adds the two.  P goes back to tensor memory in the storage type
//   PV       O[128 queries x 128 value dims] += P . V    8 x tcgen05.mma M128 N128 K16, A = P in tensor memory, B = the
//            staged V tile read MN-major (no transpose)
//   rescale  a row whose maximum moved rescales its own O row (its own lane) after the previous PV completes; nothing else
//            waits for that PV, and no block-wide agreement is needed
//   epilogue O / l -> out[query][head][128], rounded once to the storage type
// What bounds it is the softmax: 16,384 exponentials per step take the special-function units 1,200 cycles (measured 9.5
// cycles per warp instruction), the float and conversion instructions around them about 4.7 issue slots per value, against
// 1,300 cycles of MMAs; a step takes 1,800.  (An eighth or a quarter of the exponentials as polynomials on the float pipe is
// 5 % slower; a pair of blocks sharing K and V by cta_group::2 halves the L2 feed and is 15 % slower, its barriers are a
// cluster hop away.)  128 heads, chunks of 4096 tokens at 8192: 3.47 -> 2.83 ms, 990 -> 1,214 TFLOP/s.
// Warps: 0 K producer, 1 score-MMA issuer, 2 PV-MMA issuer (two issuers keep the tensor pipe fed while one of them
// waits), 3 V producer, 4.. softmax / correction / epilogue.  All waits are bounded.
#include <cuda.h>

#include <algorithm>

#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int QT = 128, KT = 128;                      // queries per block, keys per step
constexpr int SUB = KT * 128;                          // [128 queries or keys][64 dims]
constexpr int Q_BYTES = 3 * SUB;                       // 192 dims
constexpr int STAGES = 2, K_STAGE = 3 * SUB, V_STAGE = 2 * SUB;        // K: 192 dims, V: 128 dims of KT keys
constexpr int OFF_Q = 0, OFF_K = OFF_Q + Q_BYTES, OFF_V = OFF_K + STAGES * K_STAGE, OFF_MISC = OFF_V + STAGES * V_STAGE;
constexpr int VP = kVDim / 2;                          // value dims that a thread of a group normalises of its row
// reference maximum of each row after step t: [2 step parities][128 rows]; row sums and maxima of the groups: [2][128] each
constexpr int M_MREF = 320, M_LSUM = M_MREF + 2 * QT * 4, M_MLAST = M_LSUM + 2 * QT * 4, M_TMEM = M_MLAST + 2 * QT * 4, M_ABORT = M_TMEM + 4,
              MISC_BYTES = M_TMEM + 64;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024;       // + slack for 1 KB alignment
constexpr int NUM_SOFTMAX = 2 * QT;
constexpr int FIRST_SOFTMAX_WARP = 4;
constexpr int NUM_THREADS = 32 * FIRST_SOFTMAX_WARP + NUM_SOFTMAX;
// tensor memory columns: a score tile and a tile of P (16-bit pairs) per softmax group, O
constexpr int S_BUFS = 2;
constexpr uint32_t TMEM_COLS = 512, COL_S = 0, COL_P = COL_S + S_BUFS * KT, COL_O = COL_P + S_BUFS * KT / 2;
static_assert(COL_O + kVDim <= TMEM_COLS, "tensor memory columns");
constexpr float RESCALE_THRESHOLD = 8.0f;
enum { B_QFULL = 0, B_KFULL, B_KEMPTY = B_KFULL + STAGES, B_VFULL = B_KEMPTY + STAGES, B_VEMPTY = B_VFULL + STAGES,
       B_SFULL = B_VEMPTY + STAGES, B_SEMPTY = B_SFULL + S_BUFS, B_PFULL = B_SEMPTY + S_BUFS, B_PVDONE = B_PFULL + S_BUFS,
       B_OFULL = B_PVDONE + S_BUFS, B_MREF, B_COUNT = B_MREF + 8 };       // B_MREF: [2 step parities][4 warps of a group]
static_assert(B_COUNT * 8 <= M_MREF && B_COUNT <= 32, "barriers overflow their area");
static_assert(SMEM_BYTES <= 232448, "over the shared memory of one block");

// Two floats at a time (sm_100 has packed f32 arithmetic; every half rounds as the scalar instruction does)
struct F2 {
    uint64_t v;
    __device__ __forceinline__ F2(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
    __device__ __forceinline__ void get(float& lo, float& hi) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
};
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(a.v) : "l"(b.v), "l"(c.v)); return a; }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v)); return a; }

template <typename T>
__global__ void __launch_bounds__(NUM_THREADS, 1)
prefill_tc5_kernel(const T* __restrict__ q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ CUtensorMap map_r, const PrefillTile* __restrict__ tiles, const uint32_t* __restrict__ pages,
                   uint32_t H, uint32_t layer, uint32_t n_pages, const float* __restrict__ cos_sin, uint32_t cs_rows, T* __restrict__ out,
                   float scale_log2, uint32_t* __restrict__ status)
{
    extern __shared__ unsigned char prefill_smem[];
    const uint32_t raw = smem_u32(prefill_smem);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = prefill_smem + (base - raw);
    const uint32_t sQ = base + OFF_Q, sK = base + OFF_K, sV = base + OFF_V, sBar = base + OFF_MISC;
    auto bar = [&](int i) { return sBar + 8u * uint32_t(i); };
    float* mref_s = reinterpret_cast<float*>(sm + OFF_MISC + M_MREF);
    float* lsum_s = reinterpret_cast<float*>(sm + OFF_MISC + M_LSUM);
    float* mlast_s = reinterpret_cast<float*>(sm + OFF_MISC + M_MLAST);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + M_TMEM);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + M_ABORT);

    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    // the list is sorted, tiles that see the most keys first; the step's metadata is in place when this kernel starts (mla_common.cuh)
    PrefillTile a;
    {
        const uint4* p = reinterpret_cast<const uint4*>(tiles + blockIdx.x);
        const uint4 x = __ldg(p), y = __ldg(p + 1);
        a.q_row = x.x; a.n_q = x.y; a.pos = x.z; a.total = x.w; a.row0 = y.x; a.rope_pos = y.y;
    }
    const uint32_t h = blockIdx.y, total = a.total;
    const uint32_t kv_end = min(total, a.pos + QT);                // keys any query of this tile may see
    const uint32_t n_kv = (kv_end + KT - 1) / KT;

    auto arrive = [&](int i) {      // one arrival per warp
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(i));
    };
    grid_launch_dependents();
    if (tid == 64) { prefetch_map(&map_k); prefetch_map(&map_v); prefetch_map(&map_r); }
    if (warp == 0 && lane < B_COUNT) {
        const int i = int(lane);
        mbar_init(bar(i), i == B_QFULL ? 8u : i >= B_SEMPTY && i < B_PFULL + S_BUFS ? 4u : 1u);
    }
    if (warp == 0) mbar_init_fence();
    if (tid == 0) *abort_flag = 0;
    if (warp == 1) tc_alloc<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The expanded keys and values come from the kernel just before.  The queries were there before that one passed its own wait, and only
    // then does it let this kernel start (gemm_pair_kernel): they are loaded ahead of the wait (27 blocks over a 777-token prompt 1632 ->
    // 1619 us, 300 tokens x 16 blocks 778 -> 771).
    if (warp < FIRST_SOFTMAX_WARP) grid_dependency_wait();

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            constexpr int PG = KT / kPage;
            const uint32_t* pg_list = pages + a.row0 / kPage;
            uint32_t page[PG], next[PG];                             // page ids are requested a step ahead of their use
#pragma unroll
            for (int i = 0; i < PG; i++) next[i] = __ldg(pg_list + i);
            for (uint32_t t = 0; t < n_kv && ok; t++) {
#pragma unroll
                for (int i = 0; i < PG; i++) {
                    page[i] = next[i];
                    if (page[i] >= n_pages) { atomicOr(status, ST_BAD_PAGE); page[i] = 0; }
                    next[i] = __ldg(pg_list + min(t + 1, n_kv - 1) * PG + i);
                }
                const int st = int(t % STAGES), row = int(a.row0 + t * KT);
                ok = mbar_wait(bar(B_KEMPTY + st), ((t / STAGES) & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                const uint32_t kd = sK + st * K_STAGE;
                mbar_expect_tx(bar(B_KFULL + st), K_STAGE);
                tma_load_2d(kd, &map_k, bar(B_KFULL + st), int(h * kNope), row);
                tma_load_2d(kd + SUB, &map_k, bar(B_KFULL + st), int(h * kNope + 64), row);
#pragma unroll
                for (int i = 0; i < PG; i++)                         // the rope keys of each page
                    tma_load_3d(kd + 2 * SUB + i * kPage * 128, &map_r, bar(B_KFULL + st), kRank, int(page[i] * kPage), int(layer));
            }
        }
    } else if (warp == 3) {
        if (lane == 0) {
            bool ok = true;
            for (uint32_t t = 0; t < n_kv && ok; t++) {
                const int st = int(t % STAGES), row = int(a.row0 + t * KT);
                ok = mbar_wait(bar(B_VEMPTY + st), ((t / STAGES) & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                const uint32_t vd = sV + st * V_STAGE;
                mbar_expect_tx(bar(B_VFULL + st), V_STAGE);
                tma_load_2d(vd, &map_v, bar(B_VFULL + st), int(h * kVDim), row);
                tma_load_2d(vd + SUB, &map_v, bar(B_VFULL + st), int(h * kVDim + 64), row);
            }
        }
    } else if (warp == 1) {
        // ---- score MMAs: a score tile is free again as soon as its group has loaded it into registers
        constexpr uint32_t IDESC_QK = instr_desc(Fmt<T>::v, QT, KT, 0, 0), HI = desc_hi(1024);
        bool ok = mbar_wait(bar(B_QFULL), 0, abort_flag, status);
        for (uint32_t t = 0; t < n_kv && ok; t++) {
            const int ks = int(t % STAGES), b = int(t % S_BUFS);
            ok = mbar_wait(bar(B_KFULL + ks), (t / STAGES) & 1, abort_flag, status) &&
                 mbar_wait(bar(B_SEMPTY + b), ((t / S_BUFS) & 1) ^ 1, abort_flag, status);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t qa = desc_lo(sQ), kb = desc_lo(sK + ks * K_STAGE);
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        tc_mma(tmem + COL_S + b * KT, qa + ((c * SUB + k * 32) >> 4), HI, kb + ((c * SUB + k * 32) >> 4), HI, IDESC_QK,
                               (c == 0 && k == 0) ? 0u : 1u);
                tc_commit(bar(B_SFULL + b));
                tc_commit(bar(B_KEMPTY + ks));
            }
            __syncwarp();
        }
    } else if (warp == 2) {
        // ---- O += P(t) . V(t)
        constexpr uint32_t IDESC_PV = instr_desc(Fmt<T>::v, QT, kVDim, 0, 1), HI = desc_hi(1024);
        bool ok = true;
        for (uint32_t t = 0; t < n_kv && ok; t++) {
            const int vs = int(t % STAGES);
            ok = mbar_wait(bar(B_VFULL + vs), (t / STAGES) & 1, abort_flag, status) &&
                 mbar_wait(bar(B_PFULL + t % S_BUFS), (t / S_BUFS) & 1, abort_flag, status);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t vb = desc_lo(sV + vs * V_STAGE, SUB), pa = tmem + COL_P + (t % S_BUFS) * (KT / 2);
#pragma unroll
                for (int k = 0; k < KT / 16; k++)    // keys 16k..: 8 columns
                    tc_mma_ts(tmem + COL_O, pa + 8 * k, vb + ((k * 2048) >> 4), HI, IDESC_PV, (t == 0 && k == 0) ? 0u : 1u);
                tc_commit(bar(B_VEMPTY + vs));
                tc_commit(bar(B_PVDONE + (t % S_BUFS)));
                if (t + 1 == n_kv) tc_commit(bar(B_OFULL));
            }
            __syncwarp();
        }
    } else {
        // ===== softmax / correction / epilogue: the query row is this thread's tensor-memory lane; `part` is its group =====
        const uint32_t q4 = warp % 4, part = (warp - FIRST_SOFTMAX_WARP) / 4, r = q4 * 32 + lane;
        const uint32_t lane_base = (q4 * 32u) << 16;
        const uint32_t my_pos = a.pos + r;                               // last key this query may see
        {   // The query rows into the operand tiles: neighbouring lanes take neighbouring 16-byte pieces of a row.  (A thread per half row
            // makes every load of a warp 32 cache lines of 16 bytes used, and the 32 loads of cosines and sines more of them: 6.7 us
            // from the wait to the last query of a block, 2.4 now; with the stores at the end 27 blocks over a 777-token prompt 2020 ->
            // 1900 us.)
            const uint32_t st = tid - 32 * FIRST_SOFTMAX_WARP;
            const size_t pitch = size_t(H) * kQDim;
            const T* q0 = q + (size_t(a.q_row) * H + h) * kQDim;
            auto put = [&](uint32_t row, uint32_t ch, const uint4& v) {          // ch: 16-byte piece of the row
                *reinterpret_cast<uint4*>(sm + OFF_Q + (ch / 8) * SUB + row * 128 + (((ch % 8) ^ (row & 7)) << 4)) = v;
            };
            constexpr uint32_t NP = kNope / 8, RP = kRope / 16;                  // pieces of the plain dims, pairs of pieces of the rope dims
            uint4 v[QT * NP / NUM_SOFTMAX], x0[QT * RP / NUM_SOFTMAX], x1[QT * RP / NUM_SOFTMAX];
#pragma unroll
            for (int k = 0; k < int(QT * NP / NUM_SOFTMAX); k++) {
                const uint32_t row = (st + k * NUM_SOFTMAX) / NP, ch = st % NP;
                v[k] = row < a.n_q ? __ldg(reinterpret_cast<const uint4*>(q0 + row * pitch) + ch) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int k = 0; k < int(QT * RP / NUM_SOFTMAX); k++) {
                const uint32_t row = (st + k * NUM_SOFTMAX) / RP, ch = NP + st % RP;
                x0[k] = row < a.n_q ? __ldg(reinterpret_cast<const uint4*>(q0 + row * pitch) + ch) : make_uint4(0u, 0u, 0u, 0u);
                x1[k] = row < a.n_q ? __ldg(reinterpret_cast<const uint4*>(q0 + row * pitch) + ch + RP) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int k = 0; k < int(QT * NP / NUM_SOFTMAX); k++) put((st + k * NUM_SOFTMAX) / NP, st % NP, v[k]);
#pragma unroll
            for (int k = 0; k < int(QT * RP / NUM_SOFTMAX); k++) {
                const uint32_t row = (st + k * NUM_SOFTMAX) / RP, i = (st % RP) * 8, pos = a.rope_pos + row;
                if (cos_sin != nullptr && row < a.n_q) {
                    // q-side RoPE (NeoX pairs (i, i + 32), the append's table and rounding: reference transformer.cpp:1204-1240)
                    if (pos >= cs_rows) {
                        atomicOr(status, ST_BAD_SLOT);
                    } else {
                        const float4* tb = reinterpret_cast<const float4*>(cos_sin + size_t(pos) * kRope + i);
                        const float4 c0 = __ldg(tb), c1 = __ldg(tb + 1), s0 = __ldg(tb + 8), s1 = __ldg(tb + 9);
                        const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                        const T *f0 = reinterpret_cast<const T*>(&x0[k]), *f1 = reinterpret_cast<const T*>(&x1[k]);
                        uint32_t y0[4], y1[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float a0 = Elem<T>::to_f32(f0[2 * j]), a1 = Elem<T>::to_f32(f0[2 * j + 1]), b0 = Elem<T>::to_f32(f1[2 * j]), b1 = Elem<T>::to_f32(f1[2 * j + 1]);
                            y0[j] = Elem<T>::pack2(__fsub_rn(__fmul_rn(a0, cs[2 * j]), __fmul_rn(b0, sn[2 * j])), __fsub_rn(__fmul_rn(a1, cs[2 * j + 1]), __fmul_rn(b1, sn[2 * j + 1])));
                            y1[j] = Elem<T>::pack2(__fadd_rn(__fmul_rn(b0, cs[2 * j]), __fmul_rn(a0, sn[2 * j])), __fadd_rn(__fmul_rn(b1, cs[2 * j + 1]), __fmul_rn(a1, sn[2 * j + 1])));
                        }
                        x0[k] = make_uint4(y0[0], y0[1], y0[2], y0[3]);
                        x1[k] = make_uint4(y1[0], y1[1], y1[2], y1[3]);
                    }
                }
                put(row, NP + st % RP, x0[k]);
                put(row, NP + RP + st % RP, x1[k]);
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            arrive(B_QFULL);
            grid_dependency_wait();          // the outputs: an earlier kernel may still read the buffer
        }
        float m_run = -INFINITY, l_run = 0.0f;       // the row's reference maximum, and the sum of this group's steps relative to it
        bool fail = false;
        auto wait_w = [&](uint32_t b, uint32_t parity) {
            if (!fail) fail = !mbar_wait(b, parity, abort_flag, status);
            fail = __any_sync(0xffffffffu, fail);
        };
        auto group_or = [&](bool pred) -> bool {              // barrier over the softmax threads + OR
            uint32_t rr;
            asm volatile(
                "{\n.reg .pred pi, po;\n"
                "setp.ne.b32 pi, %1, 0;\n"
                "barrier.cta.red.or.pred po, 1, %2, pi;\n"
                "selp.u32 %0, 1, 0, po;\n}\n"
                : "=r"(rr) : "r"(uint32_t(pred)), "n"(NUM_SOFTMAX) : "memory");
            return rr != 0;
        };
        for (uint32_t t = part; t < n_kv; t += 2) {
            const uint32_t b = part;                                     // = t % S_BUFS
            const uint32_t s_addr = tmem + lane_base + COL_S + b * KT, p_addr = tmem + lane_base + COL_P + b * (KT / 2);
            wait_w(bar(B_SFULL + b), (t / 2) & 1);
            if (fail) break;
            tc_fence_after();
            float sv[KT];
#pragma unroll
            for (int c = 0; c < KT / 32; c++) tc_ld32(s_addr + 32 * c, reinterpret_cast<uint32_t (&)[32]>(sv[32 * c]));
            tc_wait_ld();
            tc_fence_before();
            arrive(B_SEMPTY + int(b));
            const uint32_t k0 = t * KT;
            if (k0 + KT > my_pos + 1 || k0 + KT > total) {               // causal / end mask (only near the diagonal)
                const uint32_t end = min(my_pos + 1, total);
#pragma unroll
                for (int i = 0; i < KT; i++) if (k0 + uint32_t(i) >= end) sv[i] = -INFINITY;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < KT; i += 8)
#pragma unroll
                for (int j = 0; j < 4; j++) mx4[j] = fmaxf(fmaxf(mx4[j], sv[i + j]), sv[i + 4 + j]);
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
            float m_prev = -INFINITY;                                    // the row's reference after step t - 1
            if (t > 0) {
                wait_w(bar(B_MREF + ((t - 1) & 1) * 4 + q4), ((t - 1) / 2) & 1);
                if (fail) break;
                m_prev = mref_s[((t - 1) & 1) * QT + r];
            }
            const bool need = m_prev != -INFINITY && mx > m_prev + RESCALE_THRESHOLD;
            const float m_new = m_prev == -INFINITY || need ? mx : m_prev;
            // the other group has read what this slot held (it could not have posted step t - 1 otherwise)
            mref_s[(t & 1) * QT + r] = m_new;
            arrive(B_MREF + int((t & 1) * 4 + q4));
            if (m_new != m_run) {                                        // this group's sum follows (-infinity: nothing summed yet)
                l_run = m_run == -INFINITY ? 0.0f : l_run * fast_ex2(m_run - m_new);
                m_run = m_new;
            }
            const float mref = m_run == -INFINITY ? 0.0f : m_run;         // a row whose keys so far are all masked: p = 0
            if (t >= S_BUFS) {                                           // P(t - 2) has been read
                wait_w(bar(B_PVDONE + b), (t / S_BUFS - 1) & 1);
                if (fail) break;
                tc_fence_after();
            }
            const F2 scale2(scale_log2, scale_log2), mref2(-mref, -mref);
            F2 sum2[2] = {F2(0.0f, 0.0f), F2(0.0f, 0.0f)};
#pragma unroll
            for (int c = 0; c < KT / 32; c++) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const F2 x = fma2(F2(sv[32 * c + 2 * i], sv[32 * c + 2 * i + 1]), scale2, mref2);
                    float p0, p1;
                    x.get(p0, p1);
                    p0 = fast_ex2(p0);
                    p1 = fast_ex2(p1);
                    sum2[i & 1] = add2(sum2[i & 1], F2(p0, p1));
                    pk[i] = Elem<T>::pack2(p0, p1);
                }
                tc_st16(p_addr + 16 * c, pk);
            }
            float s0, s1, s2, s3;
            sum2[0].get(s0, s1);
            sum2[1].get(s2, s3);
            l_run += (s0 + s1) + (s2 + s3);
            // tcgen05.ld / .st are warp-wide: the warp rescales when any of its rows needs it (the others multiply by 1)
            if (__any_sync(0xffffffffu, need)) {
                wait_w(bar(B_PVDONE + ((t - 1) & 1)), ((t - 1) / 2) & 1);        // PV of the previous step complete: this row of O is stable
                if (fail) break;
                tc_fence_after();
                const float alpha = need ? fast_ex2(m_prev - m_new) : 1.0f;
#pragma unroll 1
                for (uint32_t c = 0; c < kVDim / 32; c++) {
                    uint32_t o[32];
                    tc_ld32(tmem + lane_base + COL_O + c * 32, o);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tc_st32(tmem + lane_base + COL_O + c * 32, o);
                }
            }
            tc_wait_st();
            tc_fence_before();
            arrive(B_PFULL + int(b));
        }
        wait_w(bar(B_OFULL), 0);
        lsum_s[part * QT + r] = l_run;
        mlast_s[part * QT + r] = m_run;
        const bool bad = group_or(fail);
        if (!bad) {
            tc_fence_after();
            const float ma = mlast_s[r], mb = mlast_s[QT + r], m_end = fmaxf(ma, mb);     // O stands relative to the later one, the larger
            float l = 0.0f;
            if (ma != -INFINITY) l += lsum_s[r] * fast_ex2(ma - m_end);
            if (mb != -INFINITY) l += lsum_s[QT + r] * fast_ex2(mb - m_end);
            const float linv = l > 0.0f ? 1.0f / l : 0.0f;
            // by way of the query tile's shared memory (its MMAs are done), so that the lanes of a warp store whole rows
            unsigned char* box = sm + OFF_Q + r * (kVDim * 2);
#pragma unroll 1
            for (uint32_t c = 0; c < VP / 32; c++) {
                uint32_t o[32];
                tc_ld32(tmem + lane_base + COL_O + part * VP + c * 32, o);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        w[i] = Elem<T>::pack2(__uint_as_float(o[8 * j + 2 * i]) * linv, __uint_as_float(o[8 * j + 2 * i + 1]) * linv);
                    *reinterpret_cast<uint4*>(box + (((part * (VP / 8) + c * 4 + j) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            asm volatile("barrier.cta.sync 1, %0;\n" ::"n"(NUM_SOFTMAX) : "memory");
            constexpr uint32_t OP = kVDim / 8;                           // 16-byte pieces of an output row
            // read again: the loop above has no registers to carry these
            uint32_t st, q_row, n_q;
            asm volatile("mov.u32 %0, %%tid.x;\n" : "=r"(st));
            asm volatile("ld.global.v2.u32 {%0, %1}, [%2];\n" : "=r"(q_row), "=r"(n_q) : "l"(tiles + blockIdx.x) : "memory");
            st -= 32 * FIRST_SOFTMAX_WARP;
            T* dst = out + (size_t(q_row) * H + blockIdx.y) * kVDim;
#pragma unroll
            for (int k = 0; k < int(QT * OP / NUM_SOFTMAX); k++) {
                const uint32_t row = (st + k * NUM_SOFTMAX) / OP, ch = st % OP;
                if (row < n_q)
                    reinterpret_cast<uint4*>(dst + row * size_t(H) * kVDim)[ch] = *reinterpret_cast<const uint4*>(sm + OFF_Q + row * (kVDim * 2) + ((ch ^ (row & 7)) << 4));
            }
        }
        tc_fence_before();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

}  // namespace

int prefill_tc5_configure()
{
    cudaError_t e = cudaFuncSetAttribute(prefill_tc5_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(prefill_tc5_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    return int(e);
}

// Returns a cudaError_t value, or -1 when a tensor map cannot be built.
int launch_prefill_tc5(int dtype, const PrefillCall& p, uint32_t* status, cudaStream_t st)
{
    if (p.n_tiles == 0) return 0;
    if ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.out)) & 15u) return int(cudaErrorMisalignedAddress);
    alignas(64) CUtensorMap mk, mv;
    if (!make_matrix_map(&mk, dtype, p.kx, p.rows, uint64_t(p.H) * kNope, KT) ||
        !make_matrix_map(&mv, dtype, p.vx, p.rows, uint64_t(p.H) * kVDim, KT))
        return -1;
    const float scale_log2 = 1.4426950408889634f / sqrtf(float(kQDim));
    dim3 grid(p.n_tiles, p.H);
    auto go = [&](auto kernel, auto* q, auto* out) {
        return int(launch_pdl(kernel, grid, dim3(NUM_THREADS), SMEM_BYTES, st, q, mk, mv, *p.pool_map, p.tiles, p.pages, p.H, p.layer, p.n_pages,
                              p.cos_sin, p.cs_rows, out, scale_log2, status));
    };
    return dtype == 0 ? go(prefill_tc5_kernel<__half>, static_cast<const __half*>(p.q), static_cast<__half*>(p.out))
                      : go(prefill_tc5_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(p.q), static_cast<__nv_bfloat16*>(p.out));
}

}  // namespace mla
