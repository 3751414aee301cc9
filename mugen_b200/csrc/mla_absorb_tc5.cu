// q absorption (+ optionally the cache append of the same layer-step) on the 5th-generation tensor
// cores, sm_100a.
//
//   q_abs[r][h][d] = sum_{i<128} q[r][h][i] * W_UK[h*128+i][d],  d < 512;  q_abs[r][h][512..575] = q_rope
//   (reference: transformer.cpp:2563-2573; a query row gets the layout of a cache row)
//
// What bounds it is W_UK (131 KB per layer and head, read once), so the kernel is a weight stream: persistent blocks, one
// per SM, each with an equal run of (layer, head) units.  W_UK_h^T ([512 d][128 i], contraction index contiguous, made
// once at registration) arrives by TMA in pieces of 128 d x 64 i (16 KB) through a ring of twelve or eight, across unit
// boundaries, and is the M side of the MMA (tcgen05.mma M128 N=NT K16, four d-tiles of NT = 16, 32 or 64 columns, two
// accumulator sets in turn); the query rows are its N side, so a step of one row does not pay for 64.  Four warps copy
// q_nope into swizzled operand rows (two buffers) and q_rope behind the absorbed dims; four drain the accumulators.
// Where there are fewer units than SMs (16 heads, one layer) a unit is a part of a head: one to four d-tiles, and a part of
// the row tiles.  (One block per head with everything in sequence: 27 layers x 16 heads x 1 row took 24 us for 57 MB.)
//
// Append (when the caller fuses the two steps): one new row per warp, the bit-exact RMSNorm + RoPE + scatter of
// mla_append.cuh.  It shares the launch because it is a chain of dependent float additions that takes as long as the absorb
// itself: four further warps of every block take up to two rows each, blocks behind the absorb blocks what is left.
#include <algorithm>

#include "mla_absorb_ring.h"
#include "mla_append.cuh"
#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int PIECE = 128 * 128;                // 16,384: [128 d][64 i]
// An issuer per d-tile: one warp could issue a head's 32 MMAs as fast as the tensor core takes them, but its waits for eight pieces of W
// stand one behind the other (with the merge's issuers: 8 layers x 128 heads x 8 sequences, layer by layer, 514.6 -> 508.4 us).
constexpr int ISSUERS = 4, FIRST_EPI = 1 + ISSUERS, FIRST_QUERY = FIRST_EPI + 4;
constexpr int APPEND_WARPS = 4, FIRST_APPEND = FIRST_QUERY + 4;
constexpr int NUM_WARPS = FIRST_APPEND + APPEND_WARPS, NUM_THREADS = 32 * NUM_WARPS;   // W producer, MMA issuers, 4 epilogue, 4 query, 4 append warps
constexpr uint32_t APPEND_PER_WARP = 2;         // rows an absorb block's append warp takes at most
constexpr int a_bytes(int nt) { return nt * 256; }                              // q_nope of a row tile: two sub-tiles [NT][64 i]
constexpr int stages(int nt) { return ISSUERS * (nt == 64 ? 2 : 3); }             // as many per issuer as fit (mla_absorb_ring.h)
constexpr int off_a(int nt) { return stages(nt) * PIECE; }
constexpr int off_append(int nt) { return off_a(nt) + 2 * a_bytes(nt); }
constexpr int off_misc(int nt) { return off_append(nt) + APPEND_WARPS * kAppendRowSmem; }
constexpr int MISC_BYTES = 320;
constexpr int smem_bytes(int nt) { return off_misc(nt) + MISC_BYTES + 1024; }   // + slack to round the base up to 1 KB
static_assert(smem_bytes(16) <= 232448 && smem_bytes(32) <= 232448 && smem_bytes(64) <= 232448, "shared memory of one block");
static_assert(NUM_WARPS * kAppendRowSmem <= smem_bytes(16), "the append blocks live in the absorb blocks' shared memory");

struct AbsorbArgs {
    uint32_t rows, H, layer0;
    uint32_t d_parts, r_parts;          // a head's d-tiles (4 / d_parts per unit) and row tiles are cut into so many units
    uint32_t units, run, blocks;        // all layers' units; units per block; absorb blocks of the grid
    const float* cos_sin;               // not null: rotate the last 64 dims of every head with the row's position
    const uint32_t *q_pos, *att_row;
    uint32_t cs_rows, app_layers;
    // The kernel just ahead uploads this launch's metadata, that of a group of layers (att_row is null).  Nothing of it is read, and no
    // kernel behind is let start, before the wait: the kernels behind read metadata ahead of theirs.  W does not depend on it (16 heads x
    // 27 layers, one sequence: 43.7 -> 40.6 us a step against a launch that starts when the upload is over; 128 heads x 8 layers, one
    // sequence 80.3 -> 75.6).
    uint32_t behind_upload;
};

template <typename T, int NT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
absorb_tc5_kernel(const __grid_constant__ CUtensorMap map_w, const T* __restrict__ q, T* __restrict__ q_abs, const AbsorbArgs a,
                  const AppendArgs app, uint32_t* __restrict__ status)
{
    constexpr int STAGES = stages(NT), OFF_A = off_a(NT), OFF_MISC = off_misc(NT);
    constexpr AbsorbRing RING{STAGES / ISSUERS};
    constexpr uint32_t TMEM_COLS = 8 * NT;                      // two sets of four d-tiles x NT columns
    extern __shared__ unsigned char absorb_tc5_smem[];
    if (!a.behind_upload) grid_launch_dependents();
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    // Apart from kv_a the append touches nothing that an earlier kernel of the stream still reads or writes: constant
    // tables, the step metadata (in place when this kernel starts, or behind_upload), and slots of this layer's pool, last read by
    // this layer's attention in the PREVIOUS step.  Where the host knows that kv_a was complete before the kernel ahead of
    // this one started (the later layers of a multi-layer call, whose kv_a the caller handed over with the first layer's),
    // the append works first and waits last; the wait then only keeps "this kernel completes after its predecessors", which
    // the kernels behind it rely on.
    const uint32_t app_total = app.rows * a.app_layers, app_inside = min(app_total, a.blocks * APPEND_WARPS * APPEND_PER_WARP);
    auto append = [&](uint32_t i0, uint32_t step, uint32_t end, unsigned char* smem) {
        bool waited = !app.wait_first;
        if (a.behind_upload) {
            grid_dependency_wait();
            grid_launch_dependents();
            waited = true;
        }
        for (uint32_t i = i0; i < end; i += step) {
            AppendRow<T> row;
            row.prepare(app, i / app.rows, i % app.rows, status);
            if (!waited) { grid_dependency_wait(); waited = true; }
            row.run(app, smem);
        }
        if (!app.wait_first || !waited) grid_dependency_wait();
    };
    if (blockIdx.x >= a.blocks) {
        append(app_inside + (blockIdx.x - a.blocks) * NUM_WARPS + warp, ~0u / 2, app_total, absorb_tc5_smem + warp * kAppendRowSmem);
        return;
    }
    const uint32_t raw = smem_u32(absorb_tc5_smem);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = absorb_tc5_smem + (base - raw);
    const uint32_t bar0 = base + OFF_MISC;        // full[STAGES], empty[STAGES], a_full[2], a_empty[2], acc_full[2], acc_empty[2]
    auto full = [&](uint32_t s) { return bar0 + 8u * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8u * (STAGES + s); };
    auto a_full = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + b); };
    auto a_empty = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
    auto acc_full = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + 4 + b); };
    auto acc_empty = [&](uint32_t b) { return bar0 + 8u * (2 * STAGES + 6 + b); };
    static_assert((2 * STAGES + 8) * 8 <= 304, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 304);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + 308);

    const uint32_t row_tiles = (a.rows + NT - 1) / NT, n_d = 4 / a.d_parts;
    const uint32_t u0 = blockIdx.x * a.run, u1 = min(a.units, u0 + a.run);
    struct Unit { uint32_t li, h, d0, rt0, rt1; };
    auto unit_of = [&](uint32_t u) -> Unit {
        Unit x;
        const uint32_t parts = a.d_parts * a.r_parts, hu = u / parts, p = u % parts, rp = p % a.r_parts;
        x.h = hu % a.H;
        x.li = hu / a.H;
        x.d0 = (p / a.r_parts) * n_d;
        x.rt0 = row_tiles * rp / a.r_parts;
        x.rt1 = row_tiles * (rp + 1) / a.r_parts;
        return x;
    };

    if (tid == 0) {
        *abort_flag = 0;
        for (uint32_t s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (uint32_t b = 0; b < 2; b++) { mbar_init(a_full(b), 128); mbar_init(a_empty(b), ISSUERS); mbar_init(acc_full(b), ISSUERS); mbar_init(acc_empty(b), 128); }
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
            for (uint32_t u = u0; u < u1 && ok; u++) {
                const Unit x = unit_of(u);
                const int row = int(((a.layer0 + x.li) * a.H + x.h) * kRank);
                for (uint32_t p = 0; p < 2 * n_d && ok; p++) {
                    const uint32_t s = RING.stage(p / 2, u - u0, p & 1);
                    ok = mbar_wait<kPoll, true>(empty(s), RING.parity(u - u0, p & 1) ^ 1, abort_flag, status);
                    if (!ok) break;
                    mbar_expect_tx(full(s), PIECE);
                    tma_load_2d(base + s * PIECE, &map_w, full(s), 64 * int(p & 1), row + 128 * int(x.d0 + p / 2));
                }
            }
            grid_dependency_wait();
        }
    } else if (warp < FIRST_EPI) {
        const uint32_t d = warp - 1;               // this issuer's d-tile of every unit
        constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, 128, NT), HI = desc_hi(1024);
        bool ok = true;
        uint32_t n = 0;                            // row tiles so far
        for (uint32_t u = u0; u < u1 && ok; u++) {
            const Unit x = unit_of(u);
            for (uint32_t rt = x.rt0; rt < x.rt1 && ok; rt++, n++) {
                const uint32_t b = n & 1, par = (n >> 1) & 1;
                ok = mbar_wait<kPoll, true>(a_full(b), par, abort_flag, status) && mbar_wait(acc_empty(b), par ^ 1, abort_flag, status);
                if (d >= n_d) {                    // a part of a head has fewer
                    if (ok && lane == 0) { mbar_arrive(a_empty(b)); mbar_arrive(acc_full(b)); }
                    __syncwarp();
                    continue;
                }
                for (uint32_t half = 0; half < 2 && ok; half++) {
                    const uint32_t s = RING.stage(d, u - u0, half);
                    ok = mbar_wait(full(s), RING.parity(u - u0, half), abort_flag, status);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t da = desc_lo(base + s * PIECE), db = desc_lo(base + OFF_A + b * a_bytes(NT) + half * (NT * 128));
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            tc_mma(tmem + b * 4 * NT + d * NT, da + ((k * 32) >> 4), HI, db + ((k * 32) >> 4), HI, IDESC, (half == 0 && k == 0) ? 0u : 1u);
                        if (rt + 1 == x.rt1) tc_commit(empty(s));          // the unit's last row tile frees the weights
                        if (half) { tc_commit(a_empty(b)); tc_commit(acc_full(b)); }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < FIRST_QUERY) {
        // ---- epilogue: lane = d, columns = query rows
        grid_dependency_wait();                    // q_abs is still read by the attention kernel before
        const uint32_t q4 = warp % 4;
        bool ok = true;
        uint32_t n = 0;
        for (uint32_t u = u0; u < u1; u++) {
            const Unit x = unit_of(u);
            for (uint32_t rt = x.rt0; rt < x.rt1; rt++, n++) {
                const uint32_t b = n & 1;
                ok = ok && mbar_wait(acc_full(b), (n >> 1) & 1, abort_flag, status);
                ok = __all_sync(0xffffffffu, ok);
                tc_fence_after();
                // Two neighbouring lanes trade a value of every other column, so that a store carries two dims of a row: even lanes write
                // column k, odd lanes column k + 1, 64 bytes of either per warp.  (A 16-bit store per value: 3.8 us for the 4 x 128 x 64
                // values of a tile, 2.7 now.)
                constexpr int CH = NT < 32 ? 16 : 32;
                const uint32_t live = min(uint32_t(NT), a.rows - rt * NT), odd = lane & 1;
                const size_t pitch = size_t(a.H) * kRow;
                T* dst0 = q_abs + ((size_t(x.li) * a.rows + rt * NT + odd) * a.H + x.h) * kRow + x.d0 * 128 + q4 * 32 + (lane - odd);
#pragma unroll 1
                for (uint32_t d = 0; d < n_d; d++) {
#pragma unroll 1
                    for (uint32_t c = 0; c < NT; c += CH) {
                        if (c >= live) break;
                        uint32_t o[CH];
                        tc_ldn(tmem + ((q4 * 32u) << 16) + b * 4 * NT + d * NT + c, o);
                        tc_wait_ld();
                        T* dst = dst0 + d * 128 + c * pitch;
#pragma unroll
                        for (int k = 0; k < CH; k += 2) {
                            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? o[k] : o[k + 1], 1);
                            const uint32_t w = odd ? Elem<T>::pack2(__uint_as_float(got), __uint_as_float(o[k + 1]))
                                                   : Elem<T>::pack2(__uint_as_float(o[k]), __uint_as_float(got));
                            if (ok && c + k + odd < live) *reinterpret_cast<uint32_t*>(dst) = w;
                            dst += 2 * pitch;
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(acc_empty(b));
            }
        }
    } else {
        // ---- query rows: q_nope -> operand rows, q_rope -> behind the absorbed dims (by the unit that has d-tile 0).  A block with several
        // row tiles leaves the rope part to the append warps: it took the query warps 2,000 to 3,000 cycles per tile, and everything
        // waited for the operand rows of the next one.  From the wait to the last output of 27 layers x 16 heads x 80 rows 51,500 ->
        // 31,600 cycles; 16 sequences x 5 verify rows 322 -> 317 us, 64 x 8 985 -> 907, 4 layers of 128 heads x 100 sequences of 300 tokens 190 -> 172.
        // With a single tile the rope part is not in the way, and the append warps may be busy for longer.
        const uint32_t t = (tid - FIRST_QUERY * 32) % 128;
        Unit x = unit_of(u0);                      // the divisions not behind the wait
        const bool several = u1 - u0 > 1 || x.rt1 - x.rt0 > 1;
        if (warp >= FIRST_APPEND) {
            append(blockIdx.x * APPEND_WARPS + warp - FIRST_APPEND, a.blocks * APPEND_WARPS, app_inside, sm + off_append(NT) + (warp - FIRST_APPEND) * kAppendRowSmem);
        } else {
            // Rows of many steps lie far apart and have not been touched for a pass over the cache: the first load of a tile took 5 us from the
            // wait on, W_UK was there after 2 (16 sequences x 5 rows to verify, with the epilogue's wider stores 324.6 -> 320.2 us; 32
            // sequences through three blocks of 128 heads 375 -> 372).  L2 is the point of coherence, so asking ahead of the wait is safe.  (Not with one tile of up to
            // 16 rows, which the kernel before may just be writing: 27 blocks of 4 sequences 757 -> 761 us.)
            if constexpr (NT > 16) {
                for (uint32_t u = u0; u < u1; u++) {
                    const Unit y = unit_of(u);
                    const uint32_t ra = y.rt0 * NT, n = min(a.rows, y.rt1 * NT) - ra;
                    for (uint32_t i = t; i < 3 * n; i += 128) {
                        const uint32_t r = ra + i / 3;
                        const T* p = q + ((size_t(y.li) * a.rows + (a.att_row ? a.att_row[r] : r)) * a.H + y.h) * kQDim + (i % 3) * 64;
                        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
                    }
                }
            }
            grid_dependency_wait();
            if (a.behind_upload) grid_launch_dependents();
            bool ok = true;
            uint32_t n = 0;
            for (uint32_t u = u0; u < u1; u++, x = unit_of(u)) {
                const T* ql = q + size_t(x.li) * a.rows * a.H * kQDim;
                for (uint32_t rt = x.rt0; rt < x.rt1; rt++, n++) {
                    const uint32_t b = n & 1, r0 = rt * NT;
                    ok = ok && mbar_wait(a_empty(b), ((n >> 1) & 1) ^ 1, abort_flag, status);
                    unsigned char* dst = sm + OFF_A + b * a_bytes(NT);
                    auto q_row = [&](uint32_t r) -> const T* { return ql + (size_t(a.att_row ? a.att_row[r] : r) * a.H + x.h) * kQDim; };
                    uint4 v[NT / 8];                                          // 16 chunks of 16 bytes per row
#pragma unroll
                    for (int k = 0; k < NT / 8; k++) {
                        const uint32_t c = t + 128 * k, rr = c / 16;
                        v[k] = r0 + rr < a.rows ? reinterpret_cast<const uint4*>(q_row(r0 + rr))[c % 16] : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int k = 0; k < NT / 8; k++) {
                        const uint32_t c = t + 128 * k, rr = c / 16, ch = c % 16;
                        *reinterpret_cast<uint4*>(dst + (ch / 8) * (NT * 128) + rr * 128 + (((ch % 8) ^ (rr & 7)) << 4)) = v[k];
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    mbar_arrive(a_full(b));
                }
            }
        }
        if ((warp >= FIRST_APPEND) == several) {
            for (uint32_t u = u0; u < u1; u++) {
                x = unit_of(u);
                if (x.d0 != 0) continue;
                const T* ql = q + size_t(x.li) * a.rows * a.H * kQDim;
                auto q_row = [&](uint32_t r) -> const T* { return ql + (size_t(a.att_row ? a.att_row[r] : r) * a.H + x.h) * kQDim; };
                const uint32_t ra = x.rt0 * NT, n_rows = min(a.rows, x.rt1 * NT) - ra;
                T* qa = q_abs + (size_t(x.li) * a.rows * a.H + x.h) * kRow + kRank;
                if (a.cos_sin == nullptr) {
                    for (uint32_t c = t; c < n_rows * 8; c += 128) {      // already rotated: 8 chunks per row
                        const uint32_t r = ra + c / 8;
                        reinterpret_cast<uint4*>(qa + size_t(r) * a.H * kRow)[c % 8] = reinterpret_cast<const uint4*>(q_row(r) + kNope)[c % 8];
                    }
                } else {
                    // q-side RoPE (reference: transformer.cpp:3882-3921, NeoX pairs (i, i+32), YaRN frequencies): the same
                    // table and the same separately rounded products as the k_rope rotation of the append; eight pairs at a time
                    for (uint32_t c = t; c < n_rows * 4; c += 128) {
                        const uint32_t r = ra + c / 4, i = (c % 4) * 8;
                        const uint32_t pos = a.q_pos[r];
                        const uint4* src = reinterpret_cast<const uint4*>(q_row(r) + kNope + i);
                        const uint4 v0 = src[0], v1 = src[4];
                        if (pos >= a.cs_rows) {
                            if (i == 0) atomicOr(status, ST_BAD_SLOT);
                            continue;
                        }
                        const float4* tb = reinterpret_cast<const float4*>(a.cos_sin + size_t(pos) * kRope + i);
                        const float4 c0 = __ldg(tb), c1 = __ldg(tb + 1), s0 = __ldg(tb + 8), s1 = __ldg(tb + 9);
                        const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                        const T *x0 = reinterpret_cast<const T*>(&v0), *x1 = reinterpret_cast<const T*>(&v1);
                        float y0[8], y1[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const float f0 = Elem<T>::to_f32(x0[j]), f1 = Elem<T>::to_f32(x1[j]);
                            y0[j] = __fsub_rn(__fmul_rn(f0, cs[j]), __fmul_rn(f1, sn[j]));
                            y1[j] = __fadd_rn(__fmul_rn(f1, cs[j]), __fmul_rn(f0, sn[j]));
                        }
                        uint4* o = reinterpret_cast<uint4*>(qa + size_t(r) * a.H * kRow + i);
                        o[0] = make_uint4(Elem<T>::pack2(y0[0], y0[1]), Elem<T>::pack2(y0[2], y0[3]), Elem<T>::pack2(y0[4], y0[5]), Elem<T>::pack2(y0[6], y0[7]));
                        o[4] = make_uint4(Elem<T>::pack2(y1[0], y1[1]), Elem<T>::pack2(y1[2], y1[3]), Elem<T>::pack2(y1[4], y1[5]), Elem<T>::pack2(y1[6], y1[7]));
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

template <typename T>
cudaError_t configure_type()
{
    auto set = [](auto kernel, int bytes) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        // every kernel of a layer-step asks for the same (maximal) shared-memory carve-out, so the SMs are not
        // re-partitioned between consecutive launches
        return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    };
    cudaError_t e = set(absorb_tc5_kernel<T, 16>, smem_bytes(16));
    if (e == cudaSuccess) e = set(absorb_tc5_kernel<T, 32>, smem_bytes(32));
    if (e == cudaSuccess) e = set(absorb_tc5_kernel<T, 64>, smem_bytes(64));
    return e;
}

}  // namespace

int absorb_tc5_configure()
{
    const cudaError_t e = configure_type<__half>();
    return int(e != cudaSuccess ? e : configure_type<__nv_bfloat16>());
}

// w_map: host CUtensorMap over W_UK^T of all layers ([layers*H*512 d][128 i], box 64 i x 128 d, 128-byte swizzle).  q, q_abs
// and (with kv_a != nullptr: the launch also appends) kv_a hold m.layers consecutive layers from layer0; layer_pool and
// norm_w point at layer0's slices.  With rotate_q the last 64 dims of every query head are rotated with the row's
// position (m.row_pos) before they are stored.  behind_upload: see AbsorbArgs; the launch is then not plain.
int launch_absorb_tc5(int dtype, const void* q, const void* w_map, void* q_abs, uint32_t H, uint32_t layer0, const void* kv_a,
                      void* layer_pool, uint64_t pool_slots, const void* norm_w, const float* cos_sin, uint32_t cs_rows,
                      float eps, const StepMeta& m, bool rotate_q, bool append_waits, bool behind_upload, uint32_t sm_count, uint32_t* status, const LaunchStream& st)
{
    if (m.rows == 0) return 0;
    const CUtensorMap* map = static_cast<const CUtensorMap*>(w_map);
    AppendArgs app{};
    if (kv_a) app = AppendArgs{kv_a, layer_pool, pool_slots, norm_w, cos_sin, cs_rows, eps, m.app_pos, m.app_slot, m.app_rows, append_waits ? 1u : 0u};
    const uint32_t nt = m.rows <= 16 ? 16 : m.rows <= 32 ? 32 : 64, row_tiles = (m.rows + nt - 1) / nt, heads = m.layers * H;
    AbsorbArgs a{m.rows, H, layer0, 1, 1, 0, 0, 0, rotate_q ? cos_sin : nullptr, m.row_pos, m.att_row, cs_rows, m.layers, behind_upload ? 1u : 0u};
    // a head is cut while its parts still leave SMs idle: along d first (the weights are then still read once)
    while (a.d_parts < 4 && heads * a.d_parts * 2 <= sm_count) a.d_parts *= 2;
    a.r_parts = std::max(1u, std::min(row_tiles, sm_count / (heads * a.d_parts)));
    a.units = heads * a.d_parts * a.r_parts;
    a.run = (a.units + sm_count - 1) / sm_count;
    a.blocks = (a.units + a.run - 1) / a.run;
    const uint32_t app_total = app.rows * m.layers, app_inside = std::min(app_total, a.blocks * APPEND_WARPS * APPEND_PER_WARP);
    dim3 grid(a.blocks + (app_total - app_inside + NUM_WARPS - 1) / NUM_WARPS);        // append blocks carry the trailing indices
    auto go = [&](auto kernel, auto* qp, auto* qa) {
        return int(launch_pdl(kernel, grid, dim3(NUM_THREADS), size_t(smem_bytes(int(nt))), st, *map, qp, qa, a, app, status));
    };
    if (dtype == 0) {
        const auto* qp = static_cast<const __half*>(q);
        auto* qa = static_cast<__half*>(q_abs);
        return nt == 16 ? go(absorb_tc5_kernel<__half, 16>, qp, qa) : nt == 32 ? go(absorb_tc5_kernel<__half, 32>, qp, qa) : go(absorb_tc5_kernel<__half, 64>, qp, qa);
    }
    const auto* qp = static_cast<const __nv_bfloat16*>(q);
    auto* qa = static_cast<__nv_bfloat16*>(q_abs);
    return nt == 16 ? go(absorb_tc5_kernel<__nv_bfloat16, 16>, qp, qa) : nt == 32 ? go(absorb_tc5_kernel<__nv_bfloat16, 32>, qp, qa) : go(absorb_tc5_kernel<__nv_bfloat16, 64>, qp, qa);
}

}  // namespace mla
