// Dense projections around the attention op on the 5th-generation tensor cores, sm_100a:
//
//   C[M][N] = A[M][K] . W[N][K]^T        A = activations (row-major, K contiguous), W = a weight matrix exactly as the
//                                        reference keeps it for its matvec kernels (one output per row, K contiguous:
//                                        src/metal/kernel_sources.h:55-98), 16-bit operands, float accumulation in TMEM.
//
// Used for the steps of the reference's MLA decode driver that surround the attention (src/core/model/transformer.cpp:
// 3849-3929, 4002-4015): q_a / q_b (or full q), kv_a_mqa, Wo — M is the step's row count there, so the op streams the
// weight once and is HBM-bound — and for the expansion of latent rows into per-head keys and values in the chunked
// prefill path (M = tokens, K = 512).  Up to two weight matrices over the same activations share a launch (q and kv_a;
// W_UK and W_UV).
//
// Work = (output tile, k-block of 64) units in one line; every worker (a block, or a pair of blocks) gets an equal run of
// them, so a launch is balanced whatever its tile count.  A tile cut by a run boundary is finished by the worker that
// arrives last at the tile's counter: every contributor leaves its float partial in global memory (L2), the last one adds
// them in the order of the runs (bit-reproducible) and stores.  Where that costs more than it saves, pairs take whole tiles, or cut
// only what does not fill a round of all pairs (pick_shape).
//   up to 128 rows   gemm_rows_kernel, one block per SM: 128 weight rows are the M side of the MMA, the rows of A its N side
//                    (16, 32, 64 or 128 columns): the bytes in flight are weight bytes, and a step of 4 rows does not pay
//                    for 128.  HBM-bound.
//   more rows        gemm_pair_kernel on SM pairs (tcgen05.mma.cta_group::2): 256 rows of A x 256 or 128 outputs per tile, each
//                    block holding 128 rows of A and half of the outputs' weight rows: 32 KB from L2 for a k-block of 4.2
//                    MFLOP per block, where one block per 128 x 256 tile needs 48 (930 TFLOP/s = 10.7 TB/s from L2, which
//                    bounds that form).  2048 rows x 7168 outputs, K = 16384, run at 1,404 TFLOP/s, what cuBLAS
//                    sustains on the card.  With few k-blocks or tiles the start, the end and the last wave count: 777 rows x
//                    2048 outputs, K = 2048, 420 TFLOP/s.
//                    Finished tiles leave through shared memory and TMA.
// Calls of up to 32 rows whose tiles are few go to a kernel of their own (mla_gemm_few_tc5.cu).
// The first stages' weight tiles are constant and requested before the grid dependency is waited for.  Projection weights are
// kept packed (gemm_tc5_pack): tiles of 128 outputs x 64 inputs as 16 KB runs, k-block after k-block, so that a block's
// stream of tiles is one stream of consecutive bytes; in the row-major matrix a tile is 128 pieces of 128 bytes that lie
// 2 K bytes apart.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int BM = 128, BK = 64;                         // M side of one block's MMA, k-block
constexpr int A_BYTES = BM * BK * 2;                     // 16,384
// gemm_rows_kernel: a tcgen05.mma costs its issuing warp about 130 cycles whatever its size, 510 per k-block.  HBM does not bring k-blocks
// faster, but those that were requested ahead of the wait are all there behind it.  So with up to 32 rows three warps issue, into
// accumulators of their own that the epilogue adds in their order (three blocks of 128 heads x 32 rows, hidden 7168, with fewer
// stages 374 -> 367 us; input projections of 4 to 32 rows 1 to 5 % shorter, output projections between 2 % shorter and 1.5 % longer).
// With more rows reading three accumulators costs more than that (33 to 128 rows, seven shapes: 3 to 10 % slower); a fourth issuer
// would be the ninth warp of the block and leave a thread 168 registers, of which the sums of cut tiles spill hundreds.
constexpr int rows_issuers(int nt) { return nt <= 32 ? 3 : 1; }
constexpr int rows_threads(int nt) { return 32 * (1 + rows_issuers(nt) + 4); }
constexpr int EPI_WARPS = 8, PAIR_THREADS = 32 * (2 + EPI_WARPS);        // gemm_pair_kernel: two epilogue warps per 32 rows
constexpr int STORE_BYTES = 32 * 128;                    // a warp's box of 64 outputs x 32 rows on its way out
constexpr int MISC_BYTES = 256;
// gemm_rows_kernel: [128 weight rows][NT rows of A] per stage
constexpr int rows_stage(int nt) { return A_BYTES + nt * BK * 2; }
// (More stages are not faster: with what fits, 12 / 11 / 9 / 7, three blocks of 128 heads x 32 rows take 371 us, 367 with these, and
// projections of 33 to 128 rows up to a tenth more.)
constexpr int rows_stages(int nt) { return nt == 128 ? 6 : nt == 64 ? 8 : nt == 32 ? 8 : 9; }
constexpr int rows_smem(int nt) { return rows_stages(nt) * rows_stage(nt) + MISC_BYTES + 1024; }      // + slack for 1 KB alignment
// gemm_pair_kernel: [128 rows of A][NT / 2 weight rows] per block and stage
constexpr int pair_stage(int nt) { return A_BYTES + nt / 2 * BK * 2; }
constexpr int pair_stages(int nt) { return nt == 256 ? 6 : 8; }
constexpr int pair_off_store(int nt) { return pair_stages(nt) * pair_stage(nt); }
constexpr int pair_smem(int nt) { return pair_off_store(nt) + EPI_WARPS * STORE_BYTES + MISC_BYTES + 1024; }
static_assert(BK == 64, "the box width of make_matrix_map");
static_assert(rows_smem(16) <= 232448 && rows_smem(32) <= 232448 && rows_smem(64) <= 232448 && rows_smem(128) <= 232448 && pair_smem(256) <= 232448 && pair_smem(128) <= 232448, "shared memory of one block");

// Pairs with whole tiles take them in turn, so that those which compute at one time stand side by side in the line of tiles and
// ask for the same rows of A, or the same weights, at about the same time: such requests are merged on the way to L2.  How many
// tiles along A's rows stand beside each other (the rest of the rows comes behind all outputs) decides which of the two they share.
// Time over that of consecutive tiles per pair, all of A's rows side by side, in the kernel with four epilogue warps; groups of
// 1 / 2 / 8 / 16 (all, up to 4096 rows); outputs x K; best of three processes, between which one call differs by up to a tenth:
//                     512 rows               1100 rows              2048 rows              3000 rows              4096 rows
//   7168 x 16384   0.86 .95 .95 .95       0.96 .95 .91 .91       0.90 .92 .96 .95       0.99 1.03 1.14 1.04    0.92 .87 1.10 1.05
//   7168 x 12288   0.93 .92 .92 .92       0.94 .94 .90 .90       1.00 1.04 .94 .95      0.88 1.01 1.06 .98     0.94 .92 1.10 1.03
//   7168 x  8192   0.91 .89 .89 .90       0.95 .94 .90 .90       0.99 .99 .94 .94       0.92 .91 .88 .88       0.91 .89 1.00 .95
//   4096 x 16384   0.83 .91 .91 .90       1.09 .97 .93 .93       0.87 .86 .95 .96       0.92 .83 .92 .97       0.95 1.07 1.08 .98
//   4096 x 12288   0.78 .78 .75 .77       1.02 .96 .92 .92       0.94 .94 .93 .93       0.95 .83 .89 .97       0.94 .98 1.06 .96
//   4096 x  8192   0.78 .78 .78 .77       0.93 .94 .88 .88       0.94 .94 .92 .92       0.94 .94 .94 .94       0.95 .94 1.00 .94
//   2048 x 16384   0.80 .83 .83 .78       0.94 .88 .92 .92       0.93 .93 .93 .93       0.88 .84 .82 .95       1.09 1.09 1.09 .95
// All rows side by side are the safe order: 0.95 in the mean over 5000 to 8192 rows, where groups of 1 to 16 reach 1.15 to 1.27.
// Up to K = 8192 nothing is steadily better.  Where A's rows are further apart and not many: one where the outputs are many, or A's
// tiles very few; two in between.  (Expansion of a chunk of 4096 at 8192, groups of 1 / 8 / 16 / all: 357 / 366 / 363 / 361 us.)
inline uint32_t group_of(uint32_t K, uint32_t outputs, uint32_t m_tiles) {
    constexpr uint32_t FAR_K = 9216, MANY_OUTPUTS = 5632;          // between the sizes measured
    if (K < FAR_K || m_tiles > 16) return m_tiles;
    if (outputs >= MANY_OUTPUTS || m_tiles < 4) return 1;
    return m_tiles < 14 ? 2 : m_tiles;
}

struct GemmArgs {
    uint32_t M, kb;                     // rows of A, k-blocks
    uint32_t m_tiles, n_tiles[2];       // tiles along the rows of A, and along the outputs of each weight
    uint32_t N[2], w_row0[2];           // outputs of each weight; first row of the weight inside its map
    uint32_t units, run;                // tiles x k-blocks, and how many of them a worker takes
    uint32_t cut_tiles, stride;         // pairs: the first tiles of the line are cut into equal runs; of the others, whole ones, worker w
                                        // takes the tiles w, w + stride, ..
    uint32_t group_m;                   // tiles along A's rows that stand side by side in the line of tiles
    uint32_t packed;                    // weights in the layout of gemm_tc5_pack
    uint32_t residual;                  // out = T(float(out) + float(T(x))) instead of T(x)
    uint32_t vec_io;                    // outputs start on a 16-byte boundary
    const uint32_t* table;              // paged A: page of every 64 rows, else nullptr
    uint32_t layer, n_pages;
    float* partial;                     // [2 x blocks][NT/4][128] float4
    uint32_t* counters;                 // [tiles], pairs: [tiles][2]; zero between launches
};

// Which weight, tile along A's rows, tile along its outputs.  What GemmArgs holds twice is chosen by a comparison: with an index that is
// known at run time the arguments are copied to the stack first, by every thread, and each use is a load (27 blocks over a 777-token
// prompt 1643 -> 1609 us, 32 rows of 7168 values 378 -> 377).
struct Tile { uint32_t w, m, n; };
__device__ __forceinline__ Tile tile_of(const GemmArgs& a, uint32_t t) {
    Tile r;
    const uint32_t per = a.group_m * (a.n_tiles[0] + a.n_tiles[1]), g = t / per, m0 = g * a.group_m, gm = m0 < a.m_tiles ? min(a.group_m, a.m_tiles - m0) : 1u, nt = (t - g * per) / gm;      // one past the end is asked for, not used
    r.m = m0 + (t - g * per) % gm;
    r.w = nt >= a.n_tiles[0] ? 1u : 0u;
    r.n = nt - (r.w ? a.n_tiles[0] : 0u);
    return r;
}

// The unit that a loading thread stands at.  It walks its units one by one: with the divisions of tile_of for every k-block the
// one loading thread of a block, not the memory behind it, set the pace of the main loop (300 rows, 4096 x 8192: 51.9 us, 41.8
// without; 777 rows, 7168 and 1536 inputs together: 119.6, 104.8; 27 blocks over a 777-token prompt, the output projection: 16.0,
// 14.4).
template <bool kJump>
struct Walk {
    uint32_t vt, k;                     // tile of this worker's line (tile_id makes it a tile of the launch), k-block of it
    Tile t;
    uint32_t left;                      // kJump: units of this worker's run of cut tiles; its whole tiles come behind them
    template <typename TileId>
    __device__ __forceinline__ Walk(const GemmArgs& a, uint32_t u, TileId tile_id, uint32_t run = 0)
        : vt(u / a.kb), k(u % a.kb), t(tile_of(a, tile_id(vt))), left(run) {}
    template <typename TileId>
    __device__ __forceinline__ void next(const GemmArgs& a, TileId tile_id) {
        if (kJump && left != 0 && --left == 0) { vt = a.cut_tiles; k = 0; t = tile_of(a, tile_id(vt)); }
        else if (++k == a.kb) { k = 0; t = tile_of(a, tile_id(++vt)); }
    }
};

// eight 16-bit values at any alignment of the type
template <typename T>
__device__ __forceinline__ uint4 load8(const T* p, bool vec) {
    if (vec) return *reinterpret_cast<const uint4*>(p);
    const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = uint32_t(h[2 * j]) | uint32_t(h[2 * j + 1]) << 16;
    return make_uint4(w[0], w[1], w[2], w[3]);
}
template <typename T>
__device__ __forceinline__ void store8(T* p, const uint4& v, bool vec) {
    if (vec) { *reinterpret_cast<uint4*>(p) = v; return; }
    uint16_t* h = reinterpret_cast<uint16_t*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++) { h[2 * j] = uint16_t(w[j]); h[2 * j + 1] = uint16_t(w[j] >> 16); }
}

template <int CH>
__device__ __forceinline__ void load_acc(uint32_t addr, float (&v)[CH]) {
    uint32_t x[CH];
    tc_ldn(addr, x);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < CH; i++) v[i] = __uint_as_float(x[i]);
}
template <int THREADS>
__device__ __forceinline__ void epilogue_sync() { asm volatile("barrier.cta.sync 1, %0;\n" ::"n"(THREADS) : "memory"); }

// The epilogue threads hand a cut tile's accumulator (row r of it, NT columns, load(c, v) brings CH of them from column c*CH; a thread's
// share are columns c0*CH .. c1*CH - 1) over: partial to global memory, then the tile's counter.  Returns true in the worker that arrived
// last; sum_partials then gives columns c*CH.. of the whole tile.  Worker w's slots are 2w (the tile its run begins in) and
// 2w + 1 (the one it ends in).  last_slot is one word: who writes it for the next cut tile has passed that tile's first barrier, and
// everyone arrives there with this tile's value read.  (With two fences and a third barrier instead of the atomic that releases and
// acquires: 32 heads, hidden 2048, 129 rows, output projection 21.9 us, 20.9 now; 96 heads 29.9, 29.1.)
template <int NT, int CH, int THREADS, typename Load, typename Release>
__device__ __forceinline__ bool hand_over(const GemmArgs& a, uint32_t worker, uint32_t blocks_per_worker, uint32_t rank, uint32_t tile, Load load,
                                          uint32_t r, int c0, int c1, bool first_thread, bool ok, volatile uint32_t* last_slot, Release release)
{
    const uint32_t t0 = tile * a.kb;
    float4* slot = reinterpret_cast<float4*>(a.partial) + size_t(2 * (worker * blocks_per_worker + rank) + (worker * a.run >= t0 ? 0 : 1)) * (NT / 4) * 128;
#pragma unroll 1
    for (int c = c0; c < c1; c++) {
        float v[CH];
        load(c, v);
        if (c + 1 == c1) release();
#pragma unroll
        for (int i = 0; i < CH / 4; i++) __stcg(slot + (c * (CH / 4) + i) * 128 + r, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
    }
    epilogue_sync<THREADS>();
    if (first_thread) {
        const uint32_t n = (t0 + a.kb - 1) / a.run - t0 / a.run + 1;      // workers whose runs meet the tile
        uint32_t* counter = a.counters + tile * blocks_per_worker + rank;
        // releases the partials that the barrier above put behind this thread, acquires those of the workers before
        uint32_t before = 0;
        if (ok) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(before) : "l"(counter) : "memory");
        const uint32_t is_last = ok && before == n - 1 ? 1u : 0u;
        if (is_last) *counter = 0;                                       // as the next launch expects it
        *last_slot = is_last;
    }
    epilogue_sync<THREADS>();
    return *last_slot != 0;
}
template <int NT, int CH>
__device__ __forceinline__ void sum_partials(const GemmArgs& a, uint32_t blocks_per_worker, uint32_t rank, uint32_t tile, uint32_t r, int c, float (&v)[CH])
{
    const uint32_t t0 = tile * a.kb, w0 = t0 / a.run, w1 = (t0 + a.kb - 1) / a.run;
    constexpr int Q = CH / 4, BATCH = 32 / Q;                             // 32 loads of 16 bytes in flight per thread
    const float4* base = reinterpret_cast<const float4*>(a.partial) + c * Q * 128 + r;
#pragma unroll
    for (int i = 0; i < CH; i++) v[i] = 0.0f;
    for (uint32_t w = w0; w <= w1; w += BATCH) {
        float4 p[BATCH][Q];
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            const uint32_t ww = min(w + b, w1);
            const float4* sl = base + size_t(2 * (ww * blocks_per_worker + rank) + (ww * a.run >= t0 ? 0 : 1)) * (NT / 4) * 128;
#pragma unroll
            for (int i = 0; i < Q; i++) p[b][i] = w + b <= w1 ? __ldcg(sl + i * 128) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int b = 0; b < BATCH; b++)
#pragma unroll
            for (int i = 0; i < Q; i++) { v[4 * i] += p[b][i].x; v[4 * i + 1] += p[b][i].y; v[4 * i + 2] += p[b][i].z; v[4 * i + 3] += p[b][i].w; }
    }
}

template <typename T, int NT>
__global__ void __launch_bounds__(rows_threads(NT), 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                 T* __restrict__ out0, T* __restrict__ out1, const GemmArgs a, uint32_t* __restrict__ status)
{
    constexpr int STAGES = rows_stages(NT), STAGE = rows_stage(NT), OFF_MISC = STAGES * STAGE;
    constexpr int ISSUERS = rows_issuers(NT), FIRST_EPI = 1 + ISSUERS;
    constexpr uint32_t TMEM_COLS = ISSUERS == 1 ? 2 * NT : 8 * NT;          // a power of two
    static_assert(TMEM_COLS <= 512 && TMEM_COLS >= 2 * ISSUERS * NT && ISSUERS <= STAGES);
    extern __shared__ unsigned char gemm_smem[];
    const uint32_t raw = smem_u32(gemm_smem);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = gemm_smem + (base - raw);
    const uint32_t bar0 = base + OFF_MISC;                       // full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    auto full = [&](int s) { return bar0 + 8u * uint32_t(s); };
    auto empty = [&](int s) { return bar0 + 8u * uint32_t(STAGES + s); };
    auto acc_full = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + b); };
    auto acc_empty = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
    static_assert((2 * STAGES + 4) * 8 <= 224, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + 228);
    volatile uint32_t* last_slot = reinterpret_cast<volatile uint32_t*>(sm + OFF_MISC + 232);
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t u0 = blockIdx.x * a.run, u1 = min(a.units, u0 + a.run);       // this block's run of units

    grid_launch_dependents();
    if (tid == 64) prefetch_map(&map_a);
    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (uint32_t b = 0; b < 2; b++) { mbar_init(acc_full(b), ISSUERS); mbar_init(acc_empty(b), 128); }
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            auto same = [](uint32_t t) { return t; };
            auto load_w = [&](const Walk<false>& x, int s) {
                tma_load_2d(base + s * STAGE, x.t.w ? &map_w1 : &map_w0, full(s), a.packed ? 0 : int(x.k * BK),
                            a.packed ? int((x.t.n * a.kb + x.k) * BM) : int((x.t.w ? a.w_row0[1] : a.w_row0[0]) + x.t.n * BM));
            };
            auto load_a = [&](const Walk<false>& x, int s) { tma_load_2d(base + s * STAGE + A_BYTES, &map_a, full(s), int(x.k * BK), int(x.t.m * NT)); };
            const uint32_t n = u1 - u0, ahead = min(n, uint32_t(STAGES));
            Walk<false> x(a, u0, same), y = x;
            for (uint32_t i = 0; i < ahead; i++, x.next(a, same)) {
                mbar_expect_tx(full(int(i)), STAGE);
                load_w(x, int(i));
            }
            grid_dependency_wait();      // the activations come from an earlier kernel of the stream
            for (uint32_t i = 0; i < ahead; i++, y.next(a, same)) load_a(y, int(i));
            bool ok = true;
            int s = 0;                   // past the first round whenever the loop runs
            uint32_t par = 0;
            for (uint32_t i = ahead; i < n && ok; i++, y.next(a, same)) {
                ok = mbar_wait(empty(s), par, abort_flag, status);
                if (!ok) break;
                mbar_expect_tx(full(s), STAGE);
                load_w(y, s);
                load_a(y, s);
                if (++s == STAGES) { s = 0; par ^= 1; }
            }
        }
    } else if (warp < FIRST_EPI) {
        // ---- issuer p takes the k-blocks of stages p, p + ISSUERS, .. : a stage belongs to one issuer (mla_few_ring.h has the reason)
        constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, BM, NT);
        grid_dependency_wait();
        const uint32_t p = warp - 1, n = u1 - u0;
        bool ok = true;
        uint32_t nt = 0, i = p, par = 0;              // tiles so far, this issuer's k-block, its phase
        int s = int(p);                               // and stage
        for (uint32_t u = 0; u < n && ok; nt++) {
            const uint32_t end = min(n, ((u0 + u) / a.kb + 1) * a.kb - u0), d = tmem + ((nt & 1) * ISSUERS + p) * NT;
            ok = mbar_wait(acc_empty(nt & 1), ((nt >> 1) & 1) ^ 1, abort_flag, status);
            if (!ok) break;
            if (i >= end && lane == 0) mbar_arrive(acc_full(nt & 1));          // none of this tile's
            __syncwarp();
            for (bool first = true; i < end; first = false) {
                ok = mbar_wait(full(s), par, abort_flag, status);
                if (!ok) break;
                uint32_t next = i + ISSUERS;
                int s2 = s + ISSUERS;
                if (s2 >= STAGES) { next = i + STAGES - s + p; s2 = int(p); }
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t da = desc_lo(base + s * STAGE), db = desc_lo(base + s * STAGE + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; k++)
                        tc_mma(d, da + ((k * 32) >> 4), desc_hi(1024), db + ((k * 32) >> 4), desc_hi(1024), IDESC, (first && k == 0) ? 0u : 1u);
                    tc_commit(empty(s));
                    if (next >= end) tc_commit(acc_full(nt & 1));
                }
                __syncwarp();
                if (s2 <= s) par ^= 1;
                s = s2;
                i = next;
            }
            u = end;
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32*(w%4) .. +31; thread = one weight row (output), columns = rows of A
        grid_dependency_wait();
        const uint32_t q4 = warp % 4, r = q4 * 32 + lane;
        constexpr int CH = NT < 32 ? NT : 32;                     // columns per step
        bool ok = true;
        uint32_t nt = 0;
        for (uint32_t u = u0; u < u1; nt++) {
            const uint32_t tile = u / a.kb, t_end = (tile + 1) * a.kb, end = min(u1, t_end);
            const bool cut = u != tile * a.kb || end != t_end;
            const Tile tl = tile_of(a, tile);
            const uint32_t N = tl.w ? a.N[1] : a.N[0], o = tl.n * BM + r;
            T* out = tl.w ? out1 : out0;
            uint32_t live = (1u << ISSUERS) - 1;              // issuers that have a k-block of this tile
            if (ISSUERS > 1 && end - u < uint32_t(STAGES)) {
                live = 0;
                for (uint32_t i = u - u0; i < end - u0; i++) live |= 1u << (i % STAGES % ISSUERS);
            }
            ok = ok && mbar_wait(acc_full(nt & 1), (nt >> 1) & 1, abort_flag, status);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const uint32_t acc = tmem + ((q4 * 32u) << 16) + (nt & 1) * ISSUERS * NT;
            auto load = [&](int c, float (&v)[CH]) {
                if constexpr (ISSUERS == 1) { load_acc(acc + c * CH, v); return; }
#pragma unroll
                for (int i = 0; i < CH; i++) v[i] = 0.0f;
#pragma unroll
                for (int p = 0; p < ISSUERS; p++) {
                    if (!(live >> p & 1)) continue;
                    float x[CH];
                    load_acc(acc + p * NT + c * CH, x);
#pragma unroll
                    for (int i = 0; i < CH; i++) v[i] += x[i];
                }
            };
            auto release = [&]() { tc_fence_before(); mbar_arrive(acc_empty(nt & 1)); };
            // columns from c*C on of the tile, complete: round and store
            auto finish = [&](int c, const float (&v)[CH]) {
                if (o >= N || !ok) return;
                const uint32_t m0 = tl.m * NT + c * CH, rows = min(uint32_t(CH), a.M > m0 ? a.M - m0 : 0u);
                T* p = out + size_t(m0) * N + o;
                T res[CH];                                         // all of them on their way before the first store
                if (a.residual) {
#pragma unroll
                    for (int i = 0; i < CH; i++) if (uint32_t(i) < rows) res[i] = p[size_t(i) * N];
                }
#pragma unroll
                for (int i = 0; i < CH; i++) {
                    if (uint32_t(i) >= rows) continue;
                    T x = Elem<T>::from_f32(v[i]);
                    if (a.residual) x = Elem<T>::from_f32(Elem<T>::to_f32(res[i]) + Elem<T>::to_f32(x));
                    p[size_t(i) * N] = x;
                }
            };
            if (!cut) {
#pragma unroll 1
                for (int c = 0; c < NT / CH; c++) {
                    float v[CH];
                    load(c, v);
                    if (c + 1 == NT / CH) release();
                    finish(c, v);
                }
            } else if (hand_over<NT, CH, 128>(a, blockIdx.x, 1, 0, tile, load, r, 0, NT / CH, r == 0, ok, last_slot, release)) {
#pragma unroll 1
                for (int c = 0; c < NT / CH; c++) {
                    float v[CH];
                    sum_partials<NT, CH>(a, 1, 0, tile, r, c, v);
                    finish(c, v);
                }
            }
            u = end;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

// kCut: runs may end inside a tile; kResidual: outputs are added to what is there; kTma: outputs leave by TMA.  A launch fetches only
// the instructions that its outputs need.  Without kTma (outputs off a 16-byte boundary: rare) the two others are true and the
// arguments say: 27 layers of a 777-token prompt at 16 heads 1,548 -> 1,539 us, eight layers of 2,300 tokens 889 -> 878.
template <typename T, int NT, bool kPaged, bool kCut, bool kResidual, bool kTma>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                 const __grid_constant__ CUtensorMap map_c0, const __grid_constant__ CUtensorMap map_c1, T* __restrict__ out0, T* __restrict__ out1,
                 const GemmArgs a, uint32_t* __restrict__ status)
{
    constexpr int STAGES = pair_stages(NT), STAGE = pair_stage(NT), OFF_STORE = pair_off_store(NT), OFF_MISC = OFF_STORE + EPI_WARPS * STORE_BYTES;
    constexpr uint32_t TMEM_COLS = 2 * NT;
    extern __shared__ unsigned char gemm_smem[];
    const uint32_t raw = smem_u32(gemm_smem);                     // both blocks of a pair see the same offset
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = gemm_smem + (base - raw);
    const uint32_t bar0 = base + OFF_MISC;                        // full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    auto full = [&](int s) { return bar0 + 8u * uint32_t(s); };
    auto empty = [&](int s) { return bar0 + 8u * uint32_t(STAGES + s); };
    auto acc_full = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + b); };
    auto acc_empty = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
    static_assert((2 * STAGES + 4) * 8 <= 224, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + 228);
    volatile uint32_t* last_slot = reinterpret_cast<volatile uint32_t*>(sm + OFF_MISC + 232);
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t rank = cluster_rank(), worker = blockIdx.x / 2;               // rank 0 issues the MMAs
    // this pair's units: its run [c0, c1) of the cut tiles, then, counted from their end, those of its whole tiles
    const uint32_t tiles = a.units / a.kb, cut_tiles = kCut ? a.cut_tiles : 0u, cut_end = cut_tiles * a.kb;
    const uint32_t c0 = kCut ? min(worker * a.run, cut_end) : 0u, c1 = kCut ? min(c0 + a.run, cut_end) : 0u;
    const uint32_t whole = tiles - cut_tiles > worker ? (tiles - cut_tiles - worker + a.stride - 1) / a.stride : 0u;
    const uint32_t u0 = c0 < c1 ? c0 : cut_end, u1 = cut_end + whole * a.kb;
    auto tile_id = [&](uint32_t vt) -> uint32_t { return kCut && vt < cut_tiles ? vt : cut_tiles + worker + (vt - cut_tiles) * a.stride; };

    if constexpr (!kPaged) grid_launch_dependents();
    if (tid == 64) { prefetch_map(&map_a); prefetch_map(&map_c0); prefetch_map(&map_c1); }
    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (uint32_t b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 2 * EPI_WARPS); }      // the epilogue warps of both blocks
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc_pair<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    // both blocks' barriers must exist before either sends a remote arrive or a TMA completion
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t leader_full = map_to_rank(full(0), 0);
            auto load_w = [&](const Walk<kCut>& x, int s) {            // this block's half of the outputs, in boxes of up to 128 weight rows
                const uint32_t o = x.t.n * NT + rank * (NT / 2);                       // first of this block's outputs
                tma_load_2d_pair(base + s * STAGE + A_BYTES, x.t.w ? &map_w1 : &map_w0, leader_full + 8u * s, a.packed ? 0 : int(x.k * BK),
                                 a.packed ? int(((o / BM) * a.kb + x.k) * BM + o % BM) : int((x.t.w ? a.w_row0[1] : a.w_row0[0]) + o));
            };
            uint32_t cur_m = ~0u, next_m = ~0u, page[2] = {0, 0}, next_page[2] = {0, 0};
            auto page_of = [&](uint32_t i) { return __ldg(a.table + min(i, (a.M + kPage - 1) / kPage - 1)); };   // past the end: the last page again
            auto load_a = [&](const Walk<kCut>& x, int s) {
                const Tile& t = x.t;
                const int k = int(x.k * BK);
                const uint32_t dst = base + s * STAGE;
                if constexpr (kPaged) {
                    if (t.m != cur_m) {                            // the page ids of the next tile are requested a tile ahead
                        if (t.m == next_m) { page[0] = next_page[0]; page[1] = next_page[1]; }
                        else { page[0] = page_of(4 * t.m + 2 * rank); page[1] = page_of(4 * t.m + 2 * rank + 1); }
                        cur_m = t.m;
                        const uint32_t nx = tile_id(x.vt + 1);
                        next_m = nx < tiles ? tile_of(a, nx).m : t.m;
                        next_page[0] = page_of(4 * next_m + 2 * rank);
                        next_page[1] = page_of(4 * next_m + 2 * rank + 1);
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++) {             // two pages of 64 rows
                        uint32_t pg = page[h];
                        if (pg >= a.n_pages) { atomicOr(status, ST_BAD_PAGE); pg = 0; }
                        tma_load_3d_pair(dst + h * (A_BYTES / 2), &map_a, leader_full + 8u * s, k, int(pg * kPage), int(a.layer));
                    }
                } else {
                    tma_load_2d_pair(dst, &map_a, leader_full + 8u * s, k, int(t.m * 2 * BM + rank * BM));
                }
            };
            const uint32_t n = (c1 - c0) + whole * a.kb, ahead = min(n, uint32_t(STAGES));
            Walk<kCut> x(a, u0, tile_id, c1 - c0), y = x;
            for (uint32_t i = 0; i < ahead; i++, x.next(a, tile_id)) {
                if (rank == 0) mbar_expect_tx(full(int(i)), 2 * STAGE);
                load_w(x, int(i));
            }
            grid_dependency_wait();      // the activations come from an earlier kernel of the stream
            for (uint32_t i = 0; i < ahead; i++, y.next(a, tile_id)) load_a(y, int(i));
            bool ok = true;
            int s = 0;                   // past the first round whenever the loop runs
            uint32_t par = 0;
            for (uint32_t i = ahead; i < n && ok; i++, y.next(a, tile_id)) {
                ok = mbar_wait(empty(s), par, abort_flag, status);
                if (!ok) break;
                if (rank == 0) mbar_expect_tx(full(s), 2 * STAGE);
                load_w(y, s);
                load_a(y, s);
                if (++s == STAGES) { s = 0; par ^= 1; }
            }
        }
    } else if (warp == 1) {
        grid_dependency_wait();
        // Behind the expansion comes the prefill attention, which reads its queries ahead of its own wait: it may start once the kernels
        // before this one, and with them the queries, are done.
        if constexpr (kPaged) grid_launch_dependents();
        if (rank == 0) {
            constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, 2 * BM, NT);
            bool ok = true;
            uint32_t nt = 0, par = 0;
            int s = 0;
            for (uint32_t u = u0; u < u1 && ok; nt++) {
                const uint32_t end = min(kCut && u < c1 ? c1 : u1, (u / a.kb + 1) * a.kb);
                ok = mbar_wait<kSleepCluster>(acc_empty(nt & 1), ((nt >> 1) & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                const uint32_t d = tmem + (nt & 1) * NT;
                for (bool first = true; u < end && ok; u++, first = false) {
                    ok = mbar_wait<kSleepCluster>(full(s), par, abort_flag, status);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t da = desc_lo(base + s * STAGE), db = desc_lo(base + s * STAGE + A_BYTES);
#pragma unroll
                        for (int k = 0; k < BK / 16; k++)
                            tc_mma_pair(d, da + ((k * 32) >> 4), desc_hi(1024), db + ((k * 32) >> 4), desc_hi(1024), IDESC, (first && k == 0) ? 0u : 1u);
                        tc_commit_pair(empty(s));
                        if (u + 1 == end) tc_commit_pair(acc_full(nt & 1));
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; par ^= 1; }
                }
                if (kCut && u == c1) u = cut_end;
            }
        }
    } else {
        // Epilogue: warp w reads TMEM lanes 32*(w%4) .. +31; thread = one row of this block's 128, columns = outputs, half of the
        // tile's for each four warps.  A warp's outputs leave through a box of its own, without a barrier with the others.  (Four
        // warps with boxes of 128 rows in common: the expansion of a 4096 chunk at 8192 404 us, 374 now; 200 rows x 7168 x 16384 78.7,
        // 69.0; 27 blocks over a 777-token prompt 1840, 1817.)
        grid_dependency_wait();
        const uint32_t e = warp - 2, q4 = warp % 4, r = q4 * 32 + lane;
        const uint32_t leader_empty = map_to_rank(acc_empty(0), 0);
        constexpr int CH = 32, CHUNKS = NT / 2 / CH;
        const int c_first = int(e / 4) * CHUNKS;
        const uint32_t box = OFF_STORE + e * STORE_BYTES;
        bool ok = true;
        uint32_t nt = 0;
        for (uint32_t u = u0; u < u1; nt++) {
            const uint32_t vt = u / a.kb, t_end = (vt + 1) * a.kb, end = min(kCut && u < c1 ? c1 : u1, t_end), tile = tile_id(vt);
            const bool cut = kCut && (u != vt * a.kb || end != t_end);
            const Tile tl = tile_of(a, tile);
            const uint32_t N = tl.w ? a.N[1] : a.N[0], m0 = (2 * tl.m + rank) * BM + q4 * 32, m = m0 + lane;
            T* out = tl.w ? out1 : out0;
            // what the outputs are added to is requested two steps of 32 columns ahead, the first two while the tile is
            // computed: a thread's pieces lie a row apart, and each step would wait for its own round trip to memory (27 blocks
            // over a prompt of 777 tokens: 2067 -> 2025 us; the same in gemm_rows_kernel, where it is one trip, costs 1.5 %).
            // A worker of a cut tile asks before it hands its part over, so nobody has stored yet.
            auto residual = [&](int c, uint4 (&rs)[4]) {
                const uint32_t n0 = tl.n * NT + c * CH;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (kResidual && (kTma || a.residual) && m < a.M && c < c_first + CHUNKS && n0 + 8 * i < N) rs[i] = load8(out + size_t(m) * N + n0 + 8 * i, kTma || a.vec_io);
            };
            uint4 rs0[4], rs1[4];
            residual(c_first, rs0);
            residual(c_first + 1, rs1);
            ok = ok && mbar_wait(acc_full(nt & 1), (nt >> 1) & 1, abort_flag, status);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const uint32_t acc = tmem + ((q4 * 32u) << 16) + (nt & 1) * NT;
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_empty + 8u * (nt & 1));
            };
            // columns c*CH.. of the tile, complete: round and store.  All lanes of a warp pass here together.
            auto finish = [&](int c, const float (&v)[CH], uint4 (&rs)[4]) {
                const uint32_t n0 = tl.n * NT + c * CH;
                T* p = out + size_t(m) * N + n0;
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; i++) pk[i] = Elem<T>::pack2(v[2 * i], v[2 * i + 1]);
                if (kResidual && (kTma || a.residual) && m < a.M) {
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (n0 + 8 * i >= N) break;
                        const uint32_t ow[4] = {rs[i].x, rs[i].y, rs[i].z, rs[i].w};
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const auto* xo = reinterpret_cast<const T*>(&ow[j]);
                            const T* xn = reinterpret_cast<const T*>(&pk[4 * i + j]);
                            pk[4 * i + j] = Elem<T>::pack2(Elem<T>::to_f32(xo[0]) + Elem<T>::to_f32(xn[0]), Elem<T>::to_f32(xo[1]) + Elem<T>::to_f32(xn[1]));
                        }
                    }
                }
                residual(c + 2, rs);
                if constexpr (!kTma) {
                    if (m >= a.M || !ok) return;
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (n0 + 8 * i < N) store8(p + 8 * i, make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]), a.vec_io);
                    return;
                }
                // 64 outputs x 32 rows go to shared memory in the 128-byte swizzle and TMA writes whole rows of the box; a thread
                // storing its own 64 bytes per row piece reaches a third of that rate on 400 MB of output.
                if (c % 2 == 0) {                                  // the box before must have been read
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    __syncwarp();
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<uint4*>(sm + box + lane * 128 + ((((c % 2) * 4 + i) ^ (lane & 7)) << 4)) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                if (c % 2 == 1) {
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if (ok && n0 - CH < N && m0 < a.M) tma_store_2d(tl.w ? &map_c1 : &map_c0, base + box, int(n0 - CH), int(m0));
                        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                    }
                }
            };
            static_assert(CHUNKS % 2 == 0, "boxes of two chunks");
            if (!kCut || !cut) {
#pragma unroll 1
                for (int c = c_first; c < c_first + CHUNKS; c += 2) {
                    float v[CH];
                    load_acc(acc + c * CH, v);
                    finish(c, v, rs0);
                    load_acc(acc + (c + 1) * CH, v);
                    if (c + 2 == c_first + CHUNKS) release();
                    finish(c + 1, v, rs1);
                }
            }
            if constexpr (kCut) if (cut && hand_over<NT, CH, 32 * EPI_WARPS>(a, worker, 2, rank, tile, [&](int c, float (&v)[CH]) { load_acc(acc + c * CH, v); }, r, c_first, c_first + CHUNKS, tid == 64, ok, last_slot, release)) {
#pragma unroll 1
                for (int c = c_first; c < c_first + CHUNKS; c += 2) {
                    float v[CH];
                    sum_partials<NT, CH>(a, 2, rank, tile, r, c, v);
                    finish(c, v, rs0);
                    sum_partials<NT, CH>(a, 2, rank, tile, r, c + 1, v);
                    finish(c + 1, v, rs1);
                }
            }
            u = kCut && end == c1 ? cut_end : end;
        }
        if (kTma && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
        __syncwarp();
    }
    // neither block may leave while its twin can still signal its barriers or feed a pair MMA from its shared memory
    tc_fence_before();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc_pair<TMEM_COLS>(tmem);
    }
}

// y = T(float(x) * rsqrt(mean(x^2) + eps) * float(w)) per row (the reference's rms_norm kernel, src/metal/kernel_sources.h:
// 264-312; step A of the driver, and q_a_norm from the ROUNDED projection).  Bound by one round trip to memory: a thread
// keeps its values in registers between the two passes, in 16-byte pieces.  x and y may be the same buffer.
// As many rows per SM at a time as there can be, because the next kernel's blocks start when the last row has: rows of 2,048 values in
// blocks of 256 threads with a piece each are eight to an SM, with 512 threads and room for four pieces each they were two, 777 rows of a
// prompt three waves, and the projection behind them began 3 us later (27 blocks, hidden 2048: 1725 -> 1656 us).
// NORM_MAX: pieces of 8 values per thread held in registers.
template <typename T, int NORM_THREADS, int NORM_MAX>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_rows_kernel(const T* x, const T* __restrict__ w, T* y, uint32_t N, float eps, bool vec)
{
    __shared__ float red[NORM_THREADS / 32];
    grid_launch_dependents();
    const uint32_t row = blockIdx.x, tid = threadIdx.x, pieces = N / 8;
    const T* xr = x + size_t(row) * N;
    T* yr = y + size_t(row) * N;
    uint4 wv[NORM_MAX], xv[NORM_MAX];
#pragma unroll
    for (int k = 0; k < NORM_MAX; k++) if (tid + k * NORM_THREADS < pieces) wv[k] = load8(w + 8 * (tid + k * NORM_THREADS), true);
    grid_dependency_wait();
    auto sum8 = [](const uint4& v) {
        const T* e = reinterpret_cast<const T*>(&v);
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) { const float f = Elem<T>::to_f32(e[j]); s += f * f; }
        return s;
    };
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < NORM_MAX; k++)
        if (tid + k * NORM_THREADS < pieces) { xv[k] = load8(xr + 8 * (tid + k * NORM_THREADS), vec); ss += sum8(xv[k]); }
    for (uint32_t p = tid + NORM_MAX * NORM_THREADS; p < pieces; p += NORM_THREADS) ss += sum8(load8(xr + 8 * p, vec));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (tid % 32 == 0) red[tid / 32] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < NORM_THREADS / 32; i++) tot += red[i];
    const float inv = rsqrtf(tot / float(N) + eps);
    auto scale8 = [&](const uint4& v, const uint4& g) {
        const T *e = reinterpret_cast<const T*>(&v), *f = reinterpret_cast<const T*>(&g);
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            o[j] = Elem<T>::pack2(Elem<T>::to_f32(e[2 * j]) * inv * Elem<T>::to_f32(f[2 * j]), Elem<T>::to_f32(e[2 * j + 1]) * inv * Elem<T>::to_f32(f[2 * j + 1]));
        return make_uint4(o[0], o[1], o[2], o[3]);
    };
#pragma unroll
    for (int k = 0; k < NORM_MAX; k++)
        if (tid + k * NORM_THREADS < pieces) store8(yr + 8 * (tid + k * NORM_THREADS), scale8(xv[k], wv[k]), true);
    for (uint32_t p = tid + NORM_MAX * NORM_THREADS; p < pieces; p += NORM_THREADS)
        store8(yr + 8 * p, scale8(load8(xr + 8 * p, vec), load8(w + 8 * p, true)), true);
}

template <typename T>
cudaError_t configure_type()
{
    auto set = [](auto kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
    cudaError_t e = set(gemm_rows_kernel<T, 16>, rows_smem(16));
    if (e == cudaSuccess) e = set(gemm_rows_kernel<T, 32>, rows_smem(32));
    if (e == cudaSuccess) e = set(gemm_rows_kernel<T, 64>, rows_smem(64));
    if (e == cudaSuccess) e = set(gemm_rows_kernel<T, 128>, rows_smem(128));
    auto pair = [&]<bool kPaged, bool kCut, bool kResidual, bool kTma>() {
        if (e == cudaSuccess) e = set(gemm_pair_kernel<T, 128, kPaged, kCut, kResidual, kTma>, pair_smem(128));
        if (e == cudaSuccess) e = set(gemm_pair_kernel<T, 256, kPaged, kCut, kResidual, kTma>, pair_smem(256));
    };
    pair.template operator()<false, false, false, true>();
    pair.template operator()<false, false, true, true>();
    pair.template operator()<false, true, false, true>();
    pair.template operator()<false, true, true, true>();
    pair.template operator()<false, true, true, false>();
    pair.template operator()<true, false, false, true>();
    pair.template operator()<true, true, false, true>();
    return e;
}

// Tile width, cut tiles and run length of a launch: the shortest estimate of
//   whole tiles         a round of full tiles of all pairs costs 400 ns per k-block with 256 outputs, 275 with 128; the last round, with
//                       fewer pairs at work, 273 to 399, or 207 to 289;
//   all tiles cut       equal runs of k-blocks, and the hand-over (partial out, counter, partials in): 15 and 9 us more.  A k-block costs 417
//                       or 272 ns, and more with many rows of A: the pairs stand at different places along K, so that what they ask of
//                       L2 is not merged (7168 x 16384, 2300 rows: 0.63 us per k-block, 0.40 with whole tiles; a tenth of that where
//                       every pair has one tile or less);
//   the rest cut        the tiles beyond full rounds (or those and one round's) are cut and come first, whole tiles follow.
// Fitted to whole and cut runs of both widths over 20 weights x 9 row counts, 160 to 4096 (whole tiles: within 3.5 % standard deviation).
// Against one cost per k-block for both, and no rest, us:  7168 x 16384, 1300 / 2600 / 3500 rows 339 / 730 / 918 -> 262 / 526 / 647;
// 6144 x 8192, 900: 103 -> 78; 25152 x 7168, 600 / 1300: 228 / 484 -> 192 / 378; 1536 x 12288, 3500: 120 -> 102; 198 shapes of 129 to
// 3500 rows 0.97 in the mean.  gemm_rows_kernel: cycles, about 400 per k-block (the HBM rate), hand-over about 4000 and 50 per column.
struct Shape { uint32_t nt, m_tiles, n_tiles[2], run, cut_tiles; };
Shape pick_shape(const GemmCall& g, bool rows_kernel, uint32_t kb, const GemmWorkspace& ws)
{
    Shape best{};
    uint64_t best_cost = ~0ull;
    const uint32_t workers = rows_kernel ? ws.blocks : ws.blocks / 2;
    auto consider = [&](uint32_t nt, uint32_t m_side, uint32_t n_side, auto whole_cost, auto cut_cost) {
        Shape s{nt, (g.M + m_side - 1) / m_side, {0, 0}, 0, 0};
        for (int i = 0; i < g.n_weights; i++) s.n_tiles[i] = (g.w[i].N + n_side - 1) / n_side;
        const uint32_t tiles = s.m_tiles * (s.n_tiles[0] + s.n_tiles[1]), rounds = tiles / workers, rest = tiles % workers;
        auto take = [&](uint64_t cost, uint64_t run, uint32_t cut_tiles) {
            if (cost >= best_cost) return;
            best_cost = cost;
            best = s;
            best.run = uint32_t(run);
            best.cut_tiles = cut_tiles;
        };
        take(whole_cost(rounds, double(rest) / workers), uint64_t(rounds + (rest > 0)) * kb, 0);
        for (uint32_t whole = 0; whole <= rounds; whole++) {             // rounds of whole tiles behind the cut ones
            if (whole && (rows_kernel || whole + 1 < rounds)) continue;
            const uint32_t cut = tiles - whole * workers;
            const uint64_t run = std::max<uint64_t>({(uint64_t(cut) * kb + workers - 1) / workers, 2, whole ? kb / 4 : 0});
            if (cut && cut * (rows_kernel ? 1 : 2) <= ws.max_tiles) take(cut_cost(run, whole, s.m_tiles), run, cut);
        }
    };
    if (rows_kernel) {                                       // cycles
        const uint32_t nt = g.M <= 16 ? 16 : g.M <= 32 ? 32 : g.M <= 64 ? 64 : 128;
        consider(nt, nt, BM, [&](uint64_t rounds, double rest) { return (rounds + (rest > 0)) * kb * 400; },
                 [&](uint64_t run, uint64_t, uint64_t) { return run * 400 + 4000 + 50 * nt; });
    } else {                                                 // nanoseconds
        auto pairs = [&](uint32_t nt, double start, double tile, double full, double few, double more, double cut_start, double cut, double far) {
            consider(nt, 2 * BM, nt,
                     [=](uint64_t rounds, double rest) { return uint64_t(start + (rounds + (rest > 0)) * tile + kb * (rounds * full + (rest > 0 ? few + more * rest : 0))); },
                     [=](uint64_t run, uint64_t rounds, uint64_t m_tiles) {
                         const double rows = std::clamp<double>(double(m_tiles) * kb, 400, 2500) - 400;
                         return uint64_t(cut_start + rounds * (tile + kb * full) + run * (cut + (run > kb ? 1.0 : 0.1) * far * rows));
                     });
        };
        pairs(256, 6000, 0, 400, 273, 126, 20700, 417, 0.0716);
        pairs(128, 4500, 420, 275, 207, 82, 13600, 272, 0.033);
    }
    return best;
}

template <typename T>
int launch_type(const GemmCall& g, const GemmWorkspace& ws, int dtype, uint32_t* status, const LaunchStream& st)
{
    const bool rows_kernel = !g.paged_map && g.M <= 128;
    GemmArgs a{};
    a.M = g.M;
    a.kb = (g.K + BK - 1) / BK;
    const Shape sh = pick_shape(g, rows_kernel, a.kb, ws);
    const uint32_t nt = sh.nt;
    a.m_tiles = sh.m_tiles;
    a.n_tiles[0] = sh.n_tiles[0];
    a.n_tiles[1] = sh.n_tiles[1];
    a.units = a.m_tiles * (a.n_tiles[0] + a.n_tiles[1]) * a.kb;
    a.run = sh.run;
    const uint32_t whole_tiles = a.units / a.kb;
    const uint32_t outputs = g.w[0].N + (g.n_weights > 1 ? g.w[1].N : 0u);
    a.group_m = rows_kernel ? a.m_tiles : group_of(g.K, outputs, a.m_tiles);
    a.cut_tiles = sh.cut_tiles;
    a.stride = std::max(1u, std::min(whole_tiles - sh.cut_tiles, ws.blocks / 2));          // all pairs where tiles are cut and others are whole
    const uint32_t workers = rows_kernel || sh.cut_tiles == whole_tiles ? (a.units + a.run - 1) / a.run : a.stride;
    a.residual = g.residual ? 1u : 0u;
    bool tile_store = !rows_kernel;                          // pairs: outputs leave by TMA
    a.vec_io = 1u;
    a.packed = g.packed ? 1u : 0u;
    a.partial = ws.partial;
    a.counters = ws.counters;
    alignas(64) CUtensorMap ma, mc[2];
    T* out[2] = {nullptr, nullptr};
    for (int i = 0; i < g.n_weights; i++) {
        const GemmWeight& w = g.w[i];
        if (w.N % 8) return -1;
        a.N[i] = w.N;
        a.w_row0[i] = w.row0;
        out[i] = static_cast<T*>(w.out);
        if (reinterpret_cast<uintptr_t>(w.out) & 15u) {
            a.vec_io = 0u;
            tile_store = false;
        }
        // storage-type output with rows that TMA can address: the epilogue stores tiles (see the kernel)
        if (tile_store && !make_matrix_map(&mc[i], dtype, w.out, g.M, w.N, 32)) tile_store = false;
    }
    if (g.paged_map) {
        a.table = g.table;
        a.layer = g.layer;
        a.n_pages = g.n_pages;
    } else if (!make_matrix_map(&ma, dtype, g.A, g.M, g.K, rows_kernel ? nt : BM)) return -1;
    const int last = g.n_weights - 1;
    auto map_of = [&](int i) -> const CUtensorMap& { return rows_kernel || nt == 256 ? *g.w[i].map : *g.w[i].map64; };   // boxes of 128 or 64 weight rows
    const CUtensorMap &m0 = map_of(0), &m1 = map_of(last), &pa = g.paged_map ? *g.paged_map : ma;
    if (rows_kernel) {
        auto go = [&](auto kernel) {
            return int(launch_pdl(kernel, dim3(workers), dim3(rows_threads(int(nt))), size_t(rows_smem(int(nt))), st, pa, m0, m1, out[0], out[1], a, status));
        };
        return nt == 16 ? go(gemm_rows_kernel<T, 16>) : nt == 32 ? go(gemm_rows_kernel<T, 32>)
             : nt == 64 ? go(gemm_rows_kernel<T, 64>) : go(gemm_rows_kernel<T, 128>);
    }
    const CUtensorMap &c0 = tile_store ? mc[0] : m0, &c1 = tile_store ? mc[last] : m0;
    auto go = [&](auto kernel) {
        return int(launch_pdl(kernel, dim3(2 * workers), dim3(PAIR_THREADS), size_t(pair_smem(int(nt))), st, pa, m0, m1, c0, c1, out[0], out[1], a, status));
    };
    auto width = [&]<bool kPaged, bool kCut, bool kResidual, bool kTma>() {
        return nt == 256 ? go(gemm_pair_kernel<T, 256, kPaged, kCut, kResidual, kTma>) : go(gemm_pair_kernel<T, 128, kPaged, kCut, kResidual, kTma>);
    };
    const bool cut = sh.cut_tiles != 0;
    if (g.paged_map) {                                   // outputs in the library's own buffers
        if (!tile_store) return -1;
        return cut ? width.template operator()<true, true, false, true>() : width.template operator()<true, false, false, true>();
    }
    if (!tile_store) return width.template operator()<false, true, true, false>();
    if (g.residual) return cut ? width.template operator()<false, true, true, true>() : width.template operator()<false, false, true, true>();
    return cut ? width.template operator()<false, true, false, true>() : width.template operator()<false, false, false, true>();
}

}  // namespace

// The kernels of one element type: setting the attribute loads a kernel (first context of a process: 21.3 ms with both types, 20.1).
int gemm_tc5_configure(int dtype)
{
    if (const int e = gemm_few_tc5_configure(dtype)) return e;
    return int(dtype == 0 ? configure_type<__half>() : configure_type<__nv_bfloat16>());
}

// two slots of 128 x 256 floats per block (a worker of a pair launch is two blocks)
size_t gemm_tc5_partial_bytes(uint32_t blocks) { return size_t(2) * blocks * 128 * 256 * sizeof(float); }

// src [N][K] row-major -> dst [ceil(N / 128)][ceil(K / 64)][128][64], zero-filled: one warp per 128-byte piece row
static __global__ void __launch_bounds__(256)
gemm_pack_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, uint32_t N, uint32_t K)
{
    const uint32_t kb = (K + BK - 1) / BK, tile = blockIdx.y, k = blockIdx.x;
    for (uint32_t i = threadIdx.x; i < BM * 8; i += 256) {
        const uint32_t row = tile * BM + i / 8, col = k * BK + (i % 8) * 8;
        dst[(size_t(tile) * kb + k) * (BM * 8) + i] = row < N && col < K ? src[(size_t(row) * K + col) / 8] : make_uint4(0, 0, 0, 0);
    }
}

size_t gemm_tc5_packed_values(uint64_t N, uint64_t K) { return (N + BM - 1) / BM * BM * ((K + BK - 1) / BK) * BK; }

bool gemm_tc5_packed_maps(GemmWeightMaps* maps, int dtype, const void* packed, uint64_t N, uint64_t K)
{
    const uint64_t rows = gemm_tc5_packed_values(N, K) / BK;
    return make_matrix_map(&maps->box128, dtype, packed, rows, BK, 128) && make_matrix_map(&maps->box64, dtype, packed, rows, BK, 64);
}

// K a multiple of 8; both DEVICE
int launch_gemm_pack(const void* src, void* dst, uint32_t N, uint32_t K, cudaStream_t st)
{
    gemm_pack_kernel<<<dim3((K + BK - 1) / BK, (N + BM - 1) / BM), 256, 0, st>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), N, K);
    return int(cudaGetLastError());
}

bool gemm_tc5_weight_maps(GemmWeightMaps* maps, int dtype, const void* W, uint64_t rows, uint64_t K)
{
    return make_matrix_map(&maps->box128, dtype, W, rows, K, 128) && make_matrix_map(&maps->box64, dtype, W, rows, K, 64);
}

// Returns a cudaError_t value, or -1 when the operands cannot be addressed (pointers must be 16-byte aligned, row lengths
// multiples of 8).
int launch_gemm_tc5(int dtype, const GemmCall& call, const GemmWorkspace& ws, uint32_t* status, const LaunchStream& st, uint64_t& launched, bool* exchanged)
{
    if (exchanged) *exchanged = false;
    if (call.M == 0 || call.n_weights == 0) return 0;
    GemmCall g = call;
    const bool aligned = (reinterpret_cast<uintptr_t>(g.A) & 15u) == 0;
    // an output over the rows themselves: the kernel that normalises on the way would read what its other blocks wrote
    bool apart = true;
    for (int i = 0; i < g.n_weights; i++) {
        const char *o = static_cast<const char*>(g.w[i].out), *x = static_cast<const char*>(g.A);
        if (g.A && o < x + size_t(g.M) * g.K * 2 && x < o + size_t(g.M) * g.w[i].N * 2) apart = false;
        if (g.w[i].N % 8) return -1;
    }
    if (g.A && g.K % 8 == 0 && aligned && apart)
        if (const uint32_t cs = gemm_few_tc5_cluster(g, ws.clusters)) {
            launched++;
            if (exchanged) *exchanged = gemm_few_tc5_exchanges(g);
            return launch_gemm_few_tc5(dtype, g, cs, status, st);
        }
    if (g.norm_w) {
        if (const int e = launch_rmsnorm_rows(dtype, g.A, g.norm_w, g.norm_out, g.M, g.K, g.eps, st)) return e;
        launched++;
        g.A = g.norm_out;
    }
    launched++;
    const LaunchStream s(st.st, st.plain && !g.norm_w);          // the norm went first
    return dtype == 0 ? launch_type<__half>(g, ws, dtype, status, s) : launch_type<__nv_bfloat16>(g, ws, dtype, status, s);
}

int launch_rmsnorm_rows(int dtype, const void* x, const void* w, void* y, uint32_t rows, uint32_t N, float eps, const LaunchStream& st)
{
    if (rows == 0) return 0;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;      // w and y are the library's own buffers
    auto go = [&](auto* out) {
        using T = std::remove_pointer_t<decltype(out)>;
        const auto kernel = N <= 2048 ? rmsnorm_rows_kernel<T, 256, 1> : N <= 8192 ? rmsnorm_rows_kernel<T, 256, 4> : rmsnorm_rows_kernel<T, 512, 4>;
        return int(launch_pdl(kernel, dim3(rows), dim3(N <= 8192 ? 256 : 512), 0, st, static_cast<const T*>(x), static_cast<const T*>(w), out, N, eps, vec));
    };
    return dtype == 0 ? go(static_cast<__half*>(y)) : go(static_cast<__nv_bfloat16*>(y));
}

}  // namespace mla
