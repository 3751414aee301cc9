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
// Work = (output tile, k-block of 64) units in one line; every SM gets an equal run of them (one persistent block per SM),
// so a launch is balanced whatever its tile count.  A tile cut by a run boundary is finished by the block that arrives
// last at the tile's counter: every contributor leaves its float partial in global memory (L2), the last one adds them in
// the order of the runs (bit-reproducible) and stores.  Where there are many tiles per SM, runs end on tile boundaries.
// Two orientations of one kernel:
//   kSwap   up to 128 rows: 128 weight rows are the M side of the MMA, the rows of A its N side (16, 32, 64 or 128
//           columns): the bytes in flight are weight bytes, and a step of 4 rows does not pay for 128.
//   !kSwap  more rows: 128 rows of A x 256 outputs per tile; tiles of the storage type leave through shared memory and TMA.
// Warps: 0 TMA producer (the first stages' weight tiles are constant and requested before the grid dependency is
// waited for), 1 MMA issuer (tcgen05.mma M128 N=NT K16), 2-5 epilogue, two accumulators in turn.
#include <cuda.h>

#include <algorithm>

#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int BM = 128, BK = 64;                         // M side of the MMA, k-block
constexpr int A_BYTES = BM * BK * 2;                     // 16,384
constexpr int STORE_BYTES = BM * 128;                    // one box of 64 outputs x 128 rows on its way out
constexpr int NUM_THREADS = 32 * 6;
constexpr int stage_bytes(int nt) { return A_BYTES + nt * BK * 2; }
constexpr int n_stages(int nt) { return nt == 256 ? 4 : nt == 128 ? 6 : nt == 64 ? 8 : nt == 32 ? 10 : 11; }
constexpr int off_store(int nt) { return n_stages(nt) * stage_bytes(nt); }
constexpr int off_misc(int nt) { return off_store(nt) + (nt == 256 ? 2 * STORE_BYTES : 0); }
constexpr int MISC_BYTES = 256;
constexpr int smem_bytes(int nt) { return off_misc(nt) + MISC_BYTES + 1024; }      // + slack for 1 KB alignment
static_assert(smem_bytes(256) <= 232448 && smem_bytes(16) <= 232448 && smem_bytes(128) <= 232448, "shared memory of one block");

struct GemmArgs {
    uint32_t M, kb;                     // rows of A, k-blocks
    uint32_t m_tiles, n_tiles[2];       // tiles along the rows of A, and along the outputs of each weight
    uint32_t N[2], w_row0[2];           // outputs of each weight; first row of the weight inside its map
    uint32_t whole_tiles;               // runs end on tile boundaries
    uint32_t residual;                  // out = T(float(out) + float(T(x))) instead of T(x)
    uint32_t tile_store;                // !kSwap: outputs leave by TMA
    uint32_t vec_io;                    // outputs start on a 16-byte boundary
    const uint32_t* table;              // paged A: block table of the sequence (64 rows per page), else nullptr
    uint32_t layer, n_pages;
    float* partial;                     // [2 x blocks][NT/4][128] float4
    uint32_t* counters;                 // [tiles], zero between launches
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

template <typename T, int NT, bool kSwap, bool kPaged>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                const __grid_constant__ CUtensorMap map_c0, const __grid_constant__ CUtensorMap map_c1, T* __restrict__ out0, T* __restrict__ out1,
                const GemmArgs a, uint32_t* __restrict__ status)
{
    constexpr int STAGES = n_stages(NT), STAGE = stage_bytes(NT);
    constexpr uint32_t TMEM_COLS = 2 * NT < 32 ? 32 : 2 * NT;
    extern __shared__ unsigned char gemm_smem[];
    const uint32_t raw = smem_u32(gemm_smem);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = gemm_smem + (base - raw);
    const uint32_t bar0 = base + off_misc(NT);                   // full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    auto full = [&](int s) { return bar0 + 8u * uint32_t(s); };
    auto empty = [&](int s) { return bar0 + 8u * uint32_t(STAGES + s); };
    auto acc_full = [&](int b) { return bar0 + 8u * uint32_t(2 * STAGES + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * uint32_t(2 * STAGES + 2 + b); };
    static_assert((2 * STAGES + 4) * 8 <= 224, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + off_misc(NT) + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + off_misc(NT) + 228);
    volatile uint32_t* last_slot = reinterpret_cast<volatile uint32_t*>(sm + off_misc(NT) + 232);
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;

    // this block's run of units
    const uint32_t tiles = a.m_tiles * (a.n_tiles[0] + a.n_tiles[1]), blocks = gridDim.x;
    auto run_begin = [&](uint32_t b) -> uint32_t {
        return a.whole_tiles ? uint32_t(uint64_t(tiles) * b / blocks) * a.kb : uint32_t(uint64_t(tiles) * a.kb * b / blocks);
    };
    const uint32_t u0 = run_begin(blockIdx.x), u1 = run_begin(blockIdx.x + 1);
    struct Tile { uint32_t w, m, n; };                            // which weight, tile along A's rows, tile along its outputs
    auto tile_of = [&](uint32_t t) -> Tile {
        Tile r;
        const uint32_t nt = t / a.m_tiles;
        r.m = t % a.m_tiles;
        r.w = nt >= a.n_tiles[0] ? 1u : 0u;
        r.n = nt - (r.w ? a.n_tiles[0] : 0u);
        return r;
    };

    grid_launch_dependents();
    if (tid == 0) {
        *abort_flag = 0;
        for (int s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 128); }
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // operand addresses of a stage: [M side 128 rows][N side NT rows]; the weight is the M side when kSwap
            auto load_w = [&](uint32_t u, int s) {
                const Tile t = tile_of(u / a.kb);
                const int k = int(u % a.kb) * BK;
                const CUtensorMap* mw = t.w ? &map_w1 : &map_w0;
                const uint32_t dst = base + s * STAGE + (kSwap ? 0 : A_BYTES);
                const int row = int(a.w_row0[t.w] + t.n * (kSwap ? BM : NT));
                tma_load_2d(dst, mw, full(s), k, row);
                if (!kSwap) tma_load_2d(dst + A_BYTES, mw, full(s), k, row + BM);       // boxes of 128 weight rows
            };
            uint32_t cur_m = ~0u, next_m = ~0u, page[2] = {0, 0}, next_page[2] = {0, 0};
            auto page_of = [&](uint32_t i) { return __ldg(a.table + min(i, (a.M + kPage - 1) / kPage - 1)); };   // past the end: the last page again
            auto load_a = [&](uint32_t u, int s) {
                const Tile t = tile_of(u / a.kb);
                const int k = int(u % a.kb) * BK;
                const uint32_t dst = base + s * STAGE + (kSwap ? A_BYTES : 0);
                if constexpr (kPaged) {
                    if (t.m != cur_m) {                            // the page ids of the next tile are requested a tile ahead
                        if (t.m == next_m) { page[0] = next_page[0]; page[1] = next_page[1]; }
                        else { page[0] = page_of(2 * t.m); page[1] = page_of(2 * t.m + 1); }
                        cur_m = t.m;
                        next_m = t.m + 1 < a.m_tiles ? t.m + 1 : 0;
                        next_page[0] = page_of(2 * next_m);
                        next_page[1] = page_of(2 * next_m + 1);
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++) {             // two pages of 64 rows
                        uint32_t pg = page[h];
                        if (pg >= a.n_pages) { atomicOr(status, ST_BAD_PAGE); pg = 0; }
                        tma_load_3d(dst + h * (A_BYTES / 2), &map_a, full(s), k, int(pg * kPage), int(a.layer));
                    }
                } else {
                    tma_load_2d(dst, &map_a, full(s), k, int(t.m * (kSwap ? NT : BM)));
                }
            };
            const uint32_t n = u1 - u0, ahead = min(n, uint32_t(STAGES));
            for (uint32_t i = 0; i < ahead; i++) {
                mbar_expect_tx(full(int(i)), STAGE);
                load_w(u0 + i, int(i));
            }
            grid_dependency_wait();      // the activations come from an earlier kernel of the stream
            for (uint32_t i = 0; i < ahead; i++) load_a(u0 + i, int(i));
            bool ok = true;
            for (uint32_t i = ahead; i < n && ok; i++) {
                const int s = int(i % STAGES);
                ok = mbar_wait(empty(s), ((i / STAGES) & 1) ^ 1, abort_flag, status);
                if (!ok) break;
                mbar_expect_tx(full(s), STAGE);
                load_w(u0 + i, s);
                load_a(u0 + i, s);
            }
        }
    } else if (warp == 1) {
        grid_dependency_wait();
        constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, BM, NT);
        bool ok = true;
        uint32_t nt = 0;
        for (uint32_t u = u0, i = 0; u < u1 && ok; nt++) {
            const uint32_t end = min(u1, (u / a.kb + 1) * a.kb);
            ok = mbar_wait(acc_empty(int(nt & 1)), ((nt >> 1) & 1) ^ 1, abort_flag, status);
            if (!ok) break;
            const uint32_t d = tmem + (nt & 1) * NT;
            for (bool first = true; u < end && ok; u++, i++, first = false) {
                const int s = int(i % STAGES);
                ok = mbar_wait(full(s), (i / STAGES) & 1, abort_flag, status);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t da = desc_lo(base + s * STAGE), db = desc_lo(base + s * STAGE + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; k++)
                        tc_mma(d, da + ((k * 32) >> 4), desc_hi(1024), db + ((k * 32) >> 4), desc_hi(1024), IDESC, (first && k == 0) ? 0u : 1u);
                    tc_commit(empty(s));
                    if (u + 1 == end) tc_commit(acc_full(int(nt & 1)));
                }
                __syncwarp();
            }
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32*(w%4) .. +31; thread = one row of the tile's M side
        grid_dependency_wait();
        const uint32_t q4 = warp % 4, r = q4 * 32 + lane;
        auto group_sync = [&]() { asm volatile("barrier.cta.sync 1, 128;\n" ::: "memory"); };
        bool ok = true;
        uint32_t nt = 0, boxes = 0;
        for (uint32_t u = u0; u < u1; nt++) {
            const uint32_t tile = u / a.kb, t_end = (tile + 1) * a.kb, end = min(u1, t_end);
            const bool split = u != tile * a.kb || end != t_end;
            ok = ok && mbar_wait(acc_full(int(nt & 1)), (nt >> 1) & 1, abort_flag, status);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const uint32_t acc = tmem + ((q4 * 32u) << 16) + (nt & 1) * NT;
            constexpr int CH = NT < 32 ? NT : 32;                 // columns per step
            auto load_acc = [&](int c, float (&v)[CH]) {
                uint32_t x[CH];
                if constexpr (CH == 16) tc_ld16(acc + c * CH, x);
                else tc_ld32(acc + c * CH, x);
                tc_wait_ld();
#pragma unroll
                for (int i = 0; i < CH; i++) v[i] = __uint_as_float(x[i]);
            };
            const Tile tl = tile_of(tile);
            const uint32_t N = a.N[tl.w];
            T* out = tl.w ? out1 : out0;
            // columns c*CH.. of the tile, complete: round and store
            auto finish = [&](int c, const float (&v)[CH]) {
                if constexpr (kSwap) {
                    const uint32_t o = tl.n * BM + r;
                    if (o >= N) return;
                    const uint32_t m0 = tl.m * NT + c * CH, live = min(uint32_t(CH), a.M > m0 ? a.M - m0 : 0u);
                    T* p = out + size_t(m0) * N + o;
                    T res[CH];                                     // all of them on their way before the first store
                    if (a.residual) {
#pragma unroll
                        for (int i = 0; i < CH; i++) if (uint32_t(i) < live) res[i] = p[size_t(i) * N];
                    }
#pragma unroll
                    for (int i = 0; i < CH; i++) {
                        if (uint32_t(i) >= live) continue;
                        T x = Elem<T>::from_f32(v[i]);
                        if (a.residual) x = Elem<T>::from_f32(Elem<T>::to_f32(res[i]) + Elem<T>::to_f32(x));
                        p[size_t(i) * N] = x;
                    }
                } else {
                    const uint32_t m = tl.m * BM + r, n0 = tl.n * NT + c * CH;
                    T* p = out + size_t(m) * N + n0;
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; i++) pk[i] = Elem<T>::pack2(v[2 * i], v[2 * i + 1]);
                    if (a.residual && m < a.M) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (n0 + 8 * i >= N) break;
                            const uint4 o4 = load8(p + 8 * i, a.vec_io);
                            const uint32_t ow[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                const auto* xo = reinterpret_cast<const T*>(&ow[j]);
                                const T* xn = reinterpret_cast<const T*>(&pk[4 * i + j]);
                                pk[4 * i + j] = Elem<T>::pack2(Elem<T>::to_f32(xo[0]) + Elem<T>::to_f32(xn[0]), Elem<T>::to_f32(xo[1]) + Elem<T>::to_f32(xn[1]));
                            }
                        }
                    }
                    if (a.tile_store) {
                        // 64 outputs x 128 rows go to shared memory in the 128-byte swizzle and TMA writes whole rows of the box; a
                        // thread storing its own 64 bytes per row piece reaches a third of that rate on 400 MB of output.
                        unsigned char* box = sm + off_store(NT) + (boxes & 1) * STORE_BYTES + r * 128;
                        if (c % 2 == 0) {                          // the box that used this buffer before must have been read
                            if (warp == 2 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
                            group_sync();
                        }
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            *reinterpret_cast<uint4*>(box + ((((c % 2) * 4 + i) ^ (r & 7)) << 4)) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                        if (c % 2 == 1) {
                            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                            group_sync();
                            if (warp == 2 && lane == 0) {
                                if (*abort_flag == 0 && tl.n * NT + (c - 1) * CH < N)
                                    tma_store_2d(tl.w ? &map_c1 : &map_c0, base + off_store(NT) + (boxes & 1) * STORE_BYTES, int(tl.n * NT + (c - 1) * CH), int(tl.m * BM));
                                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                            }
                            boxes++;
                        }
                        return;
                    }
                    if (m >= a.M) return;
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (n0 + 8 * i < N) store8(p + 8 * i, make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]), a.vec_io);
                }
            };
            if (!split) {
#pragma unroll 1
                for (int c = 0; c < NT / CH; c++) {
                    float v[CH];
                    load_acc(c, v);
                    if (c + 1 == NT / CH) { tc_fence_before(); mbar_arrive(acc_empty(int(nt & 1))); }
                    finish(c, v);
                }
            } else {
                // slot 0 of a block: the tile its run begins in, slot 1: the tile its run ends in
                float4* slot = reinterpret_cast<float4*>(a.partial) + size_t(2 * blockIdx.x + (nt == 0 ? 0 : 1)) * (NT / 4) * 128;
#pragma unroll 1
                for (int c = 0; c < NT / CH; c++) {
                    float v[CH];
                    load_acc(c, v);
                    if (c + 1 == NT / CH) { tc_fence_before(); mbar_arrive(acc_empty(int(nt & 1))); }
#pragma unroll
                    for (int i = 0; i < CH / 4; i++) __stcg(slot + (c * (CH / 4) + i) * 128 + r, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
                }
                // contributors: the blocks whose runs meet [tile * kb, (tile + 1) * kb)
                uint32_t b0 = blockIdx.x, b1 = blockIdx.x;
                while (b0 > 0 && run_begin(b0) > tile * a.kb) b0--;
                while (b1 + 1 < blocks && run_begin(b1 + 1) < t_end) b1++;
                __threadfence();
                group_sync();
                if (warp == 2 && lane == 0) {
                    const uint32_t before = ok ? atomicAdd(a.counters + tile, 1u) : 0u;
                    const uint32_t is_last = ok && before == b1 - b0 ? 1u : 0u;
                    if (is_last) a.counters[tile] = 0;             // as the next launch expects it
                    *last_slot = is_last;
                }
                group_sync();
                if (*last_slot) {
                    __threadfence();
#pragma unroll 1
                    for (int c = 0; c < NT / CH; c++) {
                        float v[CH];
#pragma unroll
                        for (int i = 0; i < CH; i++) v[i] = 0.0f;
                        for (uint32_t b = b0; b <= b1; b++) {
                            const float4* sl = reinterpret_cast<const float4*>(a.partial) +
                                               size_t(2 * b + (run_begin(b) / a.kb == tile ? 0 : 1)) * (NT / 4) * 128;
#pragma unroll
                            for (int i = 0; i < CH / 4; i++) {
                                const float4 p = __ldcg(sl + (c * (CH / 4) + i) * 128 + r);
                                v[4 * i] += p.x; v[4 * i + 1] += p.y; v[4 * i + 2] += p.z; v[4 * i + 3] += p.w;
                            }
                        }
                        finish(c, v);
                    }
                }
                group_sync();                                      // last_slot is read by everyone before the next tile's writer
            }
            u = end;
        }
        if constexpr (!kSwap)
            if (a.tile_store && warp == 2 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

// y = T(float(x) * rsqrt(mean(x^2) + eps) * float(w)) per row (the reference's rms_norm kernel, src/metal/kernel_sources.h:
// 264-312; step A of the driver, and q_a_norm from the ROUNDED projection).  Bound by one round trip to memory: a thread
// keeps its values in registers between the two passes, in 16-byte pieces.  x and y may be the same buffer.
constexpr int NORM_THREADS = 512, NORM_MAX = 4;                    // pieces of 8 values per thread held in registers
template <typename T>
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

using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                       CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

TensorMapEncodeFn encoder()
{
    static TensorMapEncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(p);
    }();
    return fn;
}

// rows x K matrix of 16-bit values, K contiguous, row pitch ld elements: box 64 values x box_rows rows, 128-byte swizzle
bool make_map(CUtensorMap* map, int dtype, const void* ptr, uint64_t rows, uint64_t K, uint64_t ld, uint32_t box_rows)
{
    TensorMapEncodeFn enc = encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {K, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {BK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, dtype == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr),
               dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T>
cudaError_t configure_type()
{
    auto set = [](auto kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
    cudaError_t e = set(gemm_tc5_kernel<T, 16, true, false>, smem_bytes(16));
    if (e == cudaSuccess) e = set(gemm_tc5_kernel<T, 32, true, false>, smem_bytes(32));
    if (e == cudaSuccess) e = set(gemm_tc5_kernel<T, 64, true, false>, smem_bytes(64));
    if (e == cudaSuccess) e = set(gemm_tc5_kernel<T, 128, true, false>, smem_bytes(128));
    if (e == cudaSuccess) e = set(gemm_tc5_kernel<T, 256, false, false>, smem_bytes(256));
    if (e == cudaSuccess) e = set(gemm_tc5_kernel<T, 256, false, true>, smem_bytes(256));
    return e;
}

template <typename T>
int launch_type(const GemmCall& g, const GemmWorkspace& ws, int dtype, uint32_t* status, cudaStream_t st)
{
    const bool swap = !g.paged_map && g.M <= 128;
    const uint32_t nt = !swap ? 256 : g.M <= 16 ? 16 : g.M <= 32 ? 32 : g.M <= 64 ? 64 : 128;
    GemmArgs a{};
    a.M = g.M;
    a.kb = (g.K + BK - 1) / BK;
    a.m_tiles = (g.M + (swap ? nt : BM) - 1) / (swap ? nt : BM);
    a.residual = g.residual ? 1u : 0u;
    const uint32_t n_side = swap ? BM : nt;
    alignas(64) CUtensorMap ma, mc[2];
    T* out[2] = {nullptr, nullptr};
    a.tile_store = swap ? 0u : 1u;
    a.vec_io = 1u;
    for (int i = 0; i < g.n_weights; i++) {
        const GemmWeight& w = g.w[i];
        a.N[i] = w.N;
        a.w_row0[i] = w.row0;
        a.n_tiles[i] = (w.N + n_side - 1) / n_side;
        out[i] = static_cast<T*>(w.out);
        if (w.N % 8) return -1;
        if (reinterpret_cast<uintptr_t>(w.out) & 15u) a.vec_io = a.tile_store = 0u;
        // storage-type output with rows that TMA can address: the epilogue stores tiles (see the kernel)
        if (a.tile_store && !make_map(&mc[i], dtype, w.out, g.M, w.N, w.N, BM)) a.tile_store = 0u;
    }
    if (g.paged_map) {
        a.table = g.table;
        a.layer = g.layer;
        a.n_pages = g.n_pages;
    } else if (!make_map(&ma, dtype, g.A, g.M, g.K, g.K, swap ? nt : BM)) return -1;
    if (g.n_weights == 1 || !a.tile_store) mc[1] = a.tile_store ? mc[0] : *g.w[0].map;
    if (!a.tile_store) mc[0] = *g.w[0].map;
    const uint32_t tiles = a.m_tiles * (a.n_tiles[0] + a.n_tiles[1]);
    // whole tiles where the imbalance of the last one is below a sixteenth, or where a cut tile would cost more than it
    // saves (fewer than two k-blocks per block); otherwise equal runs of k-blocks
    a.whole_tiles = tiles >= 16 * ws.blocks || uint64_t(tiles) * a.kb < 2ull * ws.blocks ? 1u : 0u;
    const uint32_t blocks = std::min(ws.blocks, a.whole_tiles ? tiles : tiles * a.kb);
    if (!a.whole_tiles && tiles > ws.max_tiles) a.whole_tiles = 1u;
    a.partial = ws.partial;
    a.counters = ws.counters;
    const CUtensorMap& m0 = *g.w[0].map;
    const CUtensorMap& m1 = g.n_weights > 1 ? *g.w[1].map : m0;
    auto go = [&](auto kernel) {
        return int(launch_pdl(kernel, dim3(blocks), dim3(NUM_THREADS), size_t(smem_bytes(int(nt))), st, g.paged_map ? *g.paged_map : ma, m0, m1,
                              mc[0], mc[1], out[0], out[1], a, status));
    };
    if (g.paged_map) return go(gemm_tc5_kernel<T, 256, false, true>);
    if (!swap) return go(gemm_tc5_kernel<T, 256, false, false>);
    return nt == 16 ? go(gemm_tc5_kernel<T, 16, true, false>) : nt == 32 ? go(gemm_tc5_kernel<T, 32, true, false>)
         : nt == 64 ? go(gemm_tc5_kernel<T, 64, true, false>) : go(gemm_tc5_kernel<T, 128, true, false>);
}

}  // namespace

int gemm_tc5_configure()
{
    cudaError_t e = configure_type<__half>();
    if (e == cudaSuccess) e = configure_type<__nv_bfloat16>();
    return int(e);
}

// two slots of 128 x 256 floats per block
size_t gemm_tc5_partial_bytes(uint32_t blocks) { return size_t(2) * blocks * 128 * 256 * sizeof(float); }

bool gemm_tc5_weight_map(CUtensorMap* map, int dtype, const void* W, uint64_t rows, uint64_t K) { return make_map(map, dtype, W, rows, K, K, BM); }

// Returns a cudaError_t value, or -1 when the operands cannot be addressed (pointers must be 16-byte aligned, row lengths
// multiples of 8).
int launch_gemm_tc5(int dtype, const GemmCall& g, const GemmWorkspace& ws, uint32_t* status, cudaStream_t st)
{
    if (g.M == 0 || g.n_weights == 0) return 0;
    return dtype == 0 ? launch_type<__half>(g, ws, dtype, status, st) : launch_type<__nv_bfloat16>(g, ws, dtype, status, st);
}

int launch_rmsnorm_rows(int dtype, const void* x, const void* w, void* y, uint32_t rows, uint32_t N, float eps, cudaStream_t st)
{
    if (rows == 0) return 0;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;      // w and y are the library's own buffers
    if (dtype == 0)
        return int(launch_pdl(rmsnorm_rows_kernel<__half>, dim3(rows), dim3(NORM_THREADS), 0, st, static_cast<const __half*>(x),
                              static_cast<const __half*>(w), static_cast<__half*>(y), N, eps, vec));
    return int(launch_pdl(rmsnorm_rows_kernel<__nv_bfloat16>, dim3(rows), dim3(NORM_THREADS), 0, st, static_cast<const __nv_bfloat16*>(x),
                          static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y), N, eps, vec));
}

}  // namespace mla
