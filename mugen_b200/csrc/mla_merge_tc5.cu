// Merge of split-KV partial states + W_UV projection on the 5th-generation tensor cores, sm_100a.
//
//   o_c[row][512] = sum_p 2^(m_p - M) acc_p / sum_p 2^(m_p - M) l_p        (float, per head)
//   out[row][128] = o_c . W_UV_h^T
//
// What bounds it is W_UV (131 KB per layer and head, read once) and the partial states, so the kernel streams both:
// persistent blocks, one per SM, each with an equal run of (layer, head) units.  W_UV_h (128 outputs x 512 dims) arrives by
// TMA as eight sub-tiles [128 outputs][64 dims] in a ring of eight and is the M side of the MMA (tcgen05.mma M128 N32 or
// N16, K16): it stays in shared memory for all row tiles of its unit and its buffers are re-loaded for the next unit as the
// last tile's MMAs release them.  The N side is a tile of 16 or 8 rows of o_c, split into hi = T(o) and lo = T(o - hi)
// that stand side by side, so that W passes through the tensor core once for both (two MMAs per step, hi then lo, took 1.7 us
// of a tile of 8 rows against 0.9; 27 blocks of 16 heads x 4 rows 796 -> 775 us with what follows from it, 8 layers of 128 heads x
// 8 sequences by calls 1.5 % faster, one sequence of 131,072 tokens 1.8 %)
// (together ~16 mantissa bits for bf16, ~22 for fp16, so the float state is not rounded to the storage type before the
// projection), two buffers in turn: sixteen warps reduce the next tile's partial states while the tensor core works on
// this one's.
// Reduction: G = 8, 4, 2 or 1 warps per row for blocks of up to 2, 4, 8 or more rows, each with its share of the 512 dims,
// so that 128 bytes of loads are in flight per lane whatever the mix of rows and parts; weights come from one pass over
// (m, l), 32 parts at a time, and no exchange between warps is needed.
// (One block per head and 16 or 64 rows with load, reduction and MMAs in sequence: 27 layers x 16 heads x 1 row took 24 us
// for 57 MB.)
#include <algorithm>
#include <type_traits>

#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int W_SUB = kVDim * 128;             // 16,384: [128 outputs][64 dims]
constexpr int NSUB = kRank / 64;               // 8
constexpr int OFF_A = NSUB * W_SUB;            // two buffers of operand tiles: [sub-tile][hi rows, lo rows][64 dims]
constexpr int OFF_MISC = OFF_A + 2 * NSUB * 32 * 128;
constexpr int MISC_BYTES = 256;
constexpr int SMEM_BYTES = OFF_MISC + MISC_BYTES + 1024;   // + slack to round the base up to 1 KB
constexpr int RED_WARPS = 16;
// A tile takes 32 MMAs of 40 cycles (their 128 weight rows from shared memory), whoever issues them; what an issuer adds is its waits
// and its code, which comes in cold.  With few rows four issuers take two sub-tiles each into accumulators of their own, which the
// epilogue adds in a fixed order (27 blocks of 16 heads x 4 rows: 996 -> 970 us with the absorb's issuers).  With more than 8
// rows (G = 1) the reduction takes longer and needs the registers: two issuers there (3 layers x 128 heads x 128 sequences of 64
// tokens: one 218 us, two 205, four 244 with 160 bytes of spills; 2 layers x 128 heads x 128 verify rows: 305, 297, 324).
// An accumulator takes two sub-tiles whoever issues them: G follows from how many layers and heads share a launch, and a row's sums
// must not.
constexpr int ACCS = NSUB / 2;
template <int G>
struct Roles {        // warps: W producer, MMA issuers, 4 epilogue, then the reduction
    // rows per tile; hi and lo of them side by side are the N side, so that a sub-tile of W goes through the tensor core once
    static constexpr int MT = G == 1 ? 16 : 8, NB = 2 * MT, A_SUB = NB * 128, A_BUF = NSUB * A_SUB;
    static constexpr int ISSUERS = G == 1 ? 2 : 4, FIRST_EPI = 1 + ISSUERS, FIRST_RED = FIRST_EPI + 4, THREADS = 32 * (FIRST_RED + RED_WARPS);
    static constexpr uint32_t TMEM_COLS = 2 * ACCS * NB;
};

struct MergeArgs {
    const float* recs;
    const RowParts* parts;              // nullptr: n_parts records per row, [part][row][head]
    uint32_t rec_stride, n_parts;
    uint32_t rows, H, layer0;
    uint32_t r_parts, units, run;       // a head's rows are cut into r_parts units; units of all layers; units per block
    const uint32_t* att_row;
};

// One row's merged state by one warp: dims dim0 + 64*k + 2*lane (+1), k < DL/2.  acc comes back normalised.
// Index: of a float within 32 parts, 64 bits where a caller's partials need them (launch_merge_tc5).
template <int DL, typename Index>
__device__ __forceinline__ void reduce_row(const MergeArgs& a, const RowParts& rp, uint32_t h, uint32_t dim0, uint32_t lane, float (&acc)[DL])
{
    constexpr int Q = DL / 2, PB = 32 / DL;      // loads per part, parts per batch
    float M = -INFINITY, L = 0.0f;
#pragma unroll
    for (int k = 0; k < DL; k++) acc[k] = 0.0f;
    const Index stride = Index(a.rec_stride) * kPart;
    const float* rec0 = a.recs + size_t(rp.rec_off + h) * kPart;
    if (DL == 16 && rp.end - rp.begin == 1) {
        // One part, as most rows of a large step have: nothing to exchange, and the bits of the path below for every state (an empty part
        // adds nothing, whatever its sums hold; a maximum of infinity makes NaN).  Only where a
        // block has many rows (a warp per row): 27 layers of 64 sequences x 8 verify rows of 16 heads 1,070 -> 998 us, 4 layers of 128 heads x
        // 100 sequences of 300 tokens 206 -> 190.  With fewer rows per block 8 x 128 heads by calls take 0.7 % longer.
        const float* rec = rec0 + size_t(rp.begin) * stride;
        const float* src = rec + 2 + dim0 + 2 * lane;
        const float2 ml = *reinterpret_cast<const float2*>(rec);
#pragma unroll
        for (int k = 0; k < Q; k++) {
            const float2 f = *reinterpret_cast<const float2*>(src + 64 * k);
            acc[2 * k] = f.x;
            acc[2 * k + 1] = f.y;
        }
        const bool live = ml.x > -INFINITY;                    // not so for NaN either
        const float w = 1.0f + (ml.x - ml.x), l = w * ml.y, inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
        for (int k = 0; k < DL; k++) acc[k] = live ? fmaf(w, acc[k], 0.0f) * inv : 0.0f;
        return;
    }
    for (uint32_t c0 = rp.begin; c0 < rp.end; c0 += 32) {
        const uint32_t n = min(32u, rp.end - c0);
        const float* rec = rec0 + size_t(c0) * stride;
        const float* src = rec + 2 + dim0 + 2 * lane;
        float v[PB][Q][2];
        auto load = [&](uint32_t p0) {
#pragma unroll
            for (int i = 0; i < PB; i++)
#pragma unroll
                for (int k = 0; k < Q; k++)
                    if (p0 + i < n) {
                        const float* at = src + (p0 + i) * stride + 64 * k;
                        const float2 f = *reinterpret_cast<const float2*>(at);
                        v[i][k][0] = f.x;
                        v[i][k][1] = f.y;
                    }
        };
        float2 ml = lane < n ? *reinterpret_cast<const float2*>(rec + lane * stride) : make_float2(-INFINITY, 0.0f);
        load(0);
        float mx = ml.x;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float Mn = fmaxf(M, mx);
        if (Mn == -INFINITY) continue;                         // warp-uniform: nothing attended so far
        const float sc = exp2f(M - Mn), w = exp2f(ml.x - Mn);
        float wl = w * ml.y;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) wl += __shfl_xor_sync(0xffffffffu, wl, off);
        L = fmaf(L, sc, wl);
#pragma unroll
        for (int k = 0; k < DL; k++) acc[k] *= sc;
        M = Mn;
        for (uint32_t p0 = 0; p0 < n; p0 += PB) {
            if (p0) load(p0);
#pragma unroll
            for (int i = 0; i < PB; i++) {
                const float wi = __shfl_sync(0xffffffffu, w, int((p0 + i) & 31));
                if (p0 + i >= n) continue;
#pragma unroll
                for (int k = 0; k < DL; k++) acc[k] = fmaf(wi, v[i][k / 2][k % 2], acc[k]);
            }
        }
    }
    const float inv = L > 0.0f ? 1.0f / L : 0.0f;
#pragma unroll
    for (int k = 0; k < DL; k++) acc[k] *= inv;
}

template <typename T, int G, typename Index = uint32_t>
__global__ void __launch_bounds__(Roles<G>::THREADS, 1)
merge_outproj_tc5_kernel(const __grid_constant__ CUtensorMap map_w, T* __restrict__ out, const MergeArgs a, uint32_t* __restrict__ status)
{
    constexpr int MT = Roles<G>::MT, NB = Roles<G>::NB, A_SUB = Roles<G>::A_SUB, A_BUF = Roles<G>::A_BUF;
    constexpr int ISSUERS = Roles<G>::ISSUERS, FIRST_EPI = Roles<G>::FIRST_EPI, FIRST_RED = Roles<G>::FIRST_RED;
    constexpr uint32_t TMEM_COLS = Roles<G>::TMEM_COLS;
    extern __shared__ unsigned char merge_tc5_smem[];
    const uint32_t raw = smem_u32(merge_tc5_smem);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = merge_tc5_smem + (base - raw);
    const uint32_t bar0 = base + OFF_MISC;        // full[8], empty[8], a_full[2], a_empty[2], acc_full[2], acc_empty[2]
    auto full = [&](uint32_t s) { return bar0 + 8u * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8u * (NSUB + s); };
    auto a_full = [&](uint32_t b) { return bar0 + 8u * (2 * NSUB + b); };
    auto a_empty = [&](uint32_t b) { return bar0 + 8u * (2 * NSUB + 2 + b); };
    auto acc_full = [&](uint32_t b) { return bar0 + 8u * (2 * NSUB + 4 + b); };
    auto acc_empty = [&](uint32_t b) { return bar0 + 8u * (2 * NSUB + 6 + b); };
    static_assert((2 * NSUB + 8) * 8 <= 224, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + 228);
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;

    const uint32_t u0 = blockIdx.x * a.run, u1 = min(a.units, u0 + a.run);
    struct Unit { uint32_t li, h, r0, r1; };                // rows r0 .. r1 - 1 in tiles of MT from r0
    auto unit_of = [&](uint32_t u) -> Unit {
        const uint32_t hu = u / a.r_parts, rp = u % a.r_parts;
        return Unit{hu / a.H, hu % a.H, a.rows * rp / a.r_parts, a.rows * (rp + 1) / a.r_parts};
    };

    grid_launch_dependents();
    if (tid == 0) {
        *abort_flag = 0;
        for (uint32_t s = 0; s < NSUB; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (uint32_t b = 0; b < 2; b++) { mbar_init(a_full(b), 32 * RED_WARPS); mbar_init(a_empty(b), ISSUERS); mbar_init(acc_full(b), ISSUERS); mbar_init(acc_empty(b), 128); }
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---- the weights are constant: their loads do not wait for earlier kernels
        if (lane == 0) {
            bool ok = true;
            uint32_t n = 0;
            for (uint32_t u = u0; u < u1 && ok; u++, n++) {
                const Unit x = unit_of(u);
                for (uint32_t s = 0; s < NSUB && ok; s++) {
                    ok = mbar_wait<kPoll, true>(empty(s), (n & 1) ^ 1, abort_flag, status);
                    if (!ok) break;
                    mbar_expect_tx(full(s), W_SUB);
                    tma_load_2d(base + s * W_SUB, &map_w, full(s), 64 * int(s), int(((a.layer0 + x.li) * a.H + x.h) * kVDim));
                }
            }
            grid_dependency_wait();
        }
    } else if (warp < FIRST_EPI) {
        const uint32_t part = warp - 1;
        constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, kVDim, NB), HI = desc_hi(1024);
        bool ok = true;
        uint32_t n = 0, un = 0;                    // row tiles and units so far
        for (uint32_t u = u0; u < u1 && ok; u++, un++) {
            const Unit x = unit_of(u);
            for (uint32_t r0 = x.r0; r0 < x.r1 && ok; r0 += MT, n++) {
                const uint32_t b = n & 1, par = (n >> 1) & 1;
                ok = mbar_wait<kPoll, true>(a_full(b), par, abort_flag, status) && mbar_wait(acc_empty(b), par ^ 1, abort_flag, status);
                for (uint32_t i = 0; i < NSUB / ISSUERS && ok; i++) {
                    const uint32_t s = part * (NSUB / ISSUERS) + i, d = tmem + (b * ACCS + s / 2) * NB;
                    ok = mbar_wait(full(s), un & 1, abort_flag, status);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t da = desc_lo(base + s * W_SUB), db = desc_lo(base + OFF_A + b * A_BUF + s * A_SUB);
#pragma unroll
                        for (int k = 0; k < 4; k++) tc_mma(d, da + ((k * 32) >> 4), HI, db + ((k * 32) >> 4), HI, IDESC, (s % 2 == 0 && k == 0) ? 0u : 1u);
                        if (r0 + MT >= x.r1) tc_commit(empty(s));          // the unit's last row tile frees the weights
                        if (i + 1 == NSUB / ISSUERS) { tc_commit(a_empty(b)); tc_commit(acc_full(b)); }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < FIRST_RED) {
        // ---- epilogue: lane = output, columns = rows
        grid_dependency_wait();
        const uint32_t q4 = warp % 4;
        bool ok = true;
        uint32_t n = 0;
        for (uint32_t u = u0; u < u1; u++) {
            const Unit x = unit_of(u);
            for (uint32_t r0 = x.r0; r0 < x.r1; r0 += MT, n++) {
                const uint32_t b = n & 1, live = min(uint32_t(MT), x.r1 - r0);
                T* dst = out + (size_t(x.li) * a.rows * a.H + x.h) * kVDim + q4 * 32 + lane;
                // the caller's row of column `lane`, read ahead of the wait
                const uint32_t my_row = r0 + min(lane, live - 1), my_at = a.att_row ? a.att_row[my_row] : my_row;
                ok = ok && mbar_wait(acc_full(b), (n >> 1) & 1, abort_flag, status);
                ok = __all_sync(0xffffffffu, ok);
                tc_fence_after();
                float v[MT];
                {   // the accumulators' sums over hi and lo, always in this order
#pragma unroll
                    for (int k = 0; k < MT; k++) v[k] = 0.0f;
#pragma unroll 1
                    for (int p = 0; p < ACCS; p++) {
                        uint32_t o[NB];
                        tc_ldn(tmem + ((q4 * 32u) << 16) + (b * ACCS + p) * NB, o);
                        tc_wait_ld();
#pragma unroll
                        for (int k = 0; k < MT; k++) v[k] += __uint_as_float(o[k]) + __uint_as_float(o[MT + k]);
                    }
                }
                tc_fence_before();
                mbar_arrive(acc_empty(b));
#pragma unroll
                for (int k = 0; k < MT; k++) {
                    const uint32_t at = __shfl_sync(0xffffffffu, my_at, k);
                    if (ok && uint32_t(k) < live) dst[size_t(at) * a.H * kVDim] = Elem<T>::from_f32(v[k]);
                }
            }
        }
    } else {
        // ---- reduction of the partial states into the operand tiles
        const uint32_t rw = warp - FIRST_RED;
        // a row's part p: a segment of the plan (its RowParts say which, and where in the segment's records the row is), or
        // shard p of a KV-range-sharded sequence.  The plan is in place when this kernel starts (mla_common.cuh).
        auto row_parts = [&](uint32_t li, uint32_t r) -> RowParts {
            if (!a.parts) return RowParts{0, a.n_parts, r * a.H, 0};
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.parts + size_t(li) * a.rows + r));
            return RowParts{v.x, v.y, v.z, 0};
        };
        // Unit, tile and parts of this warp's row come ahead of their use: the divisions of unit_of and the load would each stand
        // between the wait and the first state.
        const uint32_t rr = rw / G, dim0 = (rw % G) * (kRank / G);      // G warps x (16 / G) rows: one pass per tile
        Unit x{};
        RowParts rp{0, 0, 0, 0};
        auto fetch = [&](const Unit& at, uint32_t r0) { if (r0 + rr < at.r1) rp = row_parts(at.li, r0 + rr); };
        if (u0 < u1) { x = unit_of(u0); fetch(x, x.r0); }
        grid_dependency_wait();          // the states belong to the attention kernel
        bool ok = true;
        uint32_t n = 0;
        for (uint32_t u = u0; u < u1; u++) {
            for (uint32_t r0 = x.r0; r0 < x.r1; r0 += MT, n++) {
                const uint32_t b = n & 1, live = min(uint32_t(MT), x.r1 - r0);
                unsigned char* hi = sm + OFF_A + b * A_BUF;
                float acc[16 / G];
                if (rr < live) reduce_row<16 / G, Index>(a, rp, x.h, dim0, lane, acc);
                if (r0 + MT < x.r1) fetch(x, r0 + MT);
                else if (u + 1 < u1) { const Unit y = unit_of(u + 1); fetch(y, y.r0); }
                ok = ok && mbar_wait(a_empty(b), ((n >> 1) & 1) ^ 1, abort_flag, status);      // the MMAs of two tiles ago have read this buffer
                if (rr < live) {
                    const uint32_t so = rr * 128 + (((lane / 4) ^ (rr & 7)) << 4) + (lane % 4) * 4;
#pragma unroll
                    for (int k = 0; k < 8 / G; k++) {
                        const float o0 = acc[2 * k], o1 = acc[2 * k + 1];
                        const T h0 = Elem<T>::from_f32(o0), h1 = Elem<T>::from_f32(o1);
                        unsigned char* p = hi + (dim0 / 64 + k) * A_SUB + so;
                        *reinterpret_cast<uint32_t*>(p) = Elem<T>::pack2(o0, o1);
                        *reinterpret_cast<uint32_t*>(p + MT * 128) = Elem<T>::pack2(o0 - Elem<T>::to_f32(h0), o1 - Elem<T>::to_f32(h1));
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                mbar_arrive(a_full(b));
            }
            if (u + 1 < u1) x = unit_of(u + 1);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

}  // namespace

int merge_tc5_configure()
{
    auto set = [](auto kernel) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        // every kernel of a layer-step asks for the same (maximal) shared-memory carve-out, so the SMs are not
        // re-partitioned between consecutive launches
        return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    };
    cudaError_t e = set(merge_outproj_tc5_kernel<__half, 1, uint64_t>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__half, 1>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__half, 2>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__half, 4>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__half, 8>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__nv_bfloat16, 1, uint64_t>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__nv_bfloat16, 1>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__nv_bfloat16, 2>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__nv_bfloat16, 4>);
    if (e == cudaSuccess) e = set(merge_outproj_tc5_kernel<__nv_bfloat16, 8>);
    return int(e);
}

// w_map: host CUtensorMap over W_UV of all layers ([layers*H*128 outputs][512 dims], box 64 dims x 128 outputs, 128-byte
// swizzle).  m.layers consecutive layers from layer0; out holds them one after the other.  n_parts > 0: the records are
// [n_parts][m.rows][H] instead of the plan's segments.
int launch_merge_tc5(int dtype, const float* recs, const StepMeta& m, uint32_t n_parts, const void* w_map, void* out, uint32_t H,
                     uint32_t layer0, uint32_t sm_count, uint32_t* status, const LaunchStream& st)
{
    if (m.rows == 0) return 0;
    const CUtensorMap* map = static_cast<const CUtensorMap*>(w_map);
    const uint32_t heads = m.layers * H;
    MergeArgs a{recs, n_parts ? nullptr : m.parts, n_parts ? m.rows * H : m.rec_stride, n_parts, m.rows, H, layer0, 1, 0, 0,
                n_parts ? nullptr : m.att_row};
    // A head's rows are cut while that still leaves SMs idle (the parts then read the head's weights through L2): the reduction of
    // the partial states is what takes the time, and a row's is the same whoever else is in its block.
    a.r_parts = std::max(1u, std::min(m.rows, sm_count / heads));
    const uint32_t unit_rows = (m.rows + a.r_parts - 1) / a.r_parts;
    a.units = heads * a.r_parts;
    a.run = (a.units + sm_count - 1) / sm_count;
    dim3 grid((a.units + a.run - 1) / a.run);
    // 32 parts of a plan's records are far below 2^32 floats; of a caller's partials they may be more (128 heads: from 2,040
    // rows on).  64-bit indices everywhere cost 1 % (128 heads x 8 sequences, layer by layer: 510 -> 517 us).
    const bool wide = uint64_t(32) * a.rec_stride * kPart > ~0u;
    auto launch = [&](auto k1, auto k2, auto k4, auto k8, auto k_wide, auto* o) {
        auto go = [&](auto kernel, uint32_t threads) { return int(launch_pdl(kernel, grid, dim3(threads), SMEM_BYTES, st, *map, o, a, status)); };
        constexpr uint32_t T1 = Roles<1>::THREADS, TN = Roles<2>::THREADS;
        if (wide) return go(k_wide, T1);
        // (Sixteen warps for a single row were slower however many parts it has: their loop over parts is 32 wide, and 4-byte loads.
        // One layer, 16 heads x 8 rows in blocks of one row: 1 part 5.4 us, 4.5 with eight warps on it; 64 parts 7.7, 7.3.)
        return unit_rows <= 2 ? go(k8, TN) : unit_rows <= 4 ? go(k4, TN) : unit_rows <= 8 ? go(k2, TN) : go(k1, T1);
    };
    auto pick = [&](auto* o) {
        using T = std::remove_pointer_t<decltype(o)>;
        return launch(merge_outproj_tc5_kernel<T, 1>, merge_outproj_tc5_kernel<T, 2>, merge_outproj_tc5_kernel<T, 4>, merge_outproj_tc5_kernel<T, 8>,
                      merge_outproj_tc5_kernel<T, 1, uint64_t>, o);
    };
    return dtype == 0 ? pick(static_cast<__half*>(out)) : pick(static_cast<__nv_bfloat16*>(out));
}

}  // namespace mla
