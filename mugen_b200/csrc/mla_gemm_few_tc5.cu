// Projections of up to 32 rows whose weight matrix fits the SMs in one go, with the RMSNorm of the rows in front, sm_100a.
//
//   out[M][N] = norm(x)[M][K] . W[N][K]^T   (or x as it is; optionally added to what out holds)
//
// The same contraction as gemm_rows_kernel (mla_gemm_tc5.cu: weight rows are the M side of the MMA, packed weights) for the
// steps of a few sequences, where no launch of the block has more than a few microseconds of work and what counts is the chain
// from one dependency to the next.  What that chain was made of there (27 blocks of 16 heads x 4 rows, timed inside the kernels):
// the normalisation as a launch of its own 0.8 us and the hand-over to the next launch 1.1; one issuing warp for all MMAs 1.6; a
// tile cut over workers finished through global memory (partials, fence, counter, partials back) 3.5 to 5.  Here
//   * a cluster of 1, 2, 4 or 8 blocks takes one tile of 128 outputs, every block an equal share of K: the sums meet in the
//     blocks' shared memory (each block finishes the rows c = rank, rank + cluster size, ..), in the order of the ranks;
//   * four warps issue the MMAs, into accumulators of their own that the epilogue adds in a fixed order;
//   * the rows come by ordinary loads, so that their normalisation needs no pass of its own: every warp sums the squares of its rows,
//     or, where they are long, those of its block's share of K, and the cluster exchanges the sums; the rounded values go to the
//     operand tile.
// 27 blocks of 16 heads x 4 rows: 937 -> 808 us per step, 752 -> 701 with whole rows summed by their warp (the exchange had taken 1.25 of
// a projection's seven microseconds) and with kernels of less code.  The parts of what is left: rows loaded 0.6, squares 0.4, normalised
// 0.8, MMAs 1.1, sums to their blocks 0.9, stored and left 0.6.
#include <cuda.h>

#include <algorithm>

#include "mla_few_ring.h"
#include "mla_launch.h"
#include "mla_tc5.cuh"

namespace mla {

namespace {

using namespace tc5;

constexpr int BM = 128, BK = 64;
constexpr int W_BYTES = BM * BK * 2;                        // 16,384: one packed tile of 128 outputs x 64 inputs
constexpr int STAGES = FewRing::stages, ISSUERS = FewRing::issuers;
constexpr int ROW_WARPS = 8;                                // the row warps load and normalise the rows, and finish the tile
constexpr int FIRST_ROW_WARP = 1 + ISSUERS, NUM_THREADS = 32 * (FIRST_ROW_WARP + ROW_WARPS);
constexpr int MAX_CLUSTER = 8;
constexpr int A_BYTES = 32768;                              // operand tiles [k-block][NT rows][64 inputs]
constexpr int max_kblocks(int nt) { return A_BYTES / (nt * BK * 2); }       // of one block: 16 (16 rows) or 8 (32 rows)
constexpr int OFF_A = STAGES * W_BYTES;
constexpr int OFF_RED = OFF_A + A_BYTES;                    // [source rank][rows of this rank][128 outputs] floats: NT * 512 bytes
constexpr int OFF_SS = OFF_RED + 32 * BM * 4;               // [source rank][32 rows] floats
constexpr int OFF_MISC = OFF_SS + MAX_CLUSTER * 32 * 4;
constexpr int SMEM_BYTES = OFF_MISC + 256 + 1024;           // + slack for 1 KB alignment
static_assert(SMEM_BYTES <= 232448, "shared memory of one block");

// 16 bytes by a load that stays where it is written: rows behind grid_dependency_wait (from memory that the compiler takes for
// constant it may move ahead), norm weights ahead of it (it may move them behind)
__device__ __forceinline__ uint4 load_here(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }

struct FewArgs {
    uint32_t M, K, kb;                  // rows, inputs, k-blocks
    uint32_t cs, cs_log2;               // blocks of a cluster
    uint32_t split, split_log2;         // row warps that share a row (up to four rows)
    uint32_t n_tiles0, N[2];            // tiles of the first weight; outputs of each
    uint32_t residual, whole;
    float eps;
};

// Sums of squares of a warp's rows (pitch 8 rows) in pieces of 8 values, in every lane; eight loads of a lane in flight.
template <typename T, int ROWS>
__device__ __forceinline__ void row_squares(const T* row0, size_t pitch, uint32_t rows, uint32_t pieces, uint32_t lane, float (&sum)[ROWS]) {
    constexpr int PER = 8 / ROWS;
    float s[ROWS][4] = {};
    for (uint32_t c0 = lane; c0 < pieces; c0 += 32 * PER) {
        uint4 v[ROWS][PER];
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int i = 0; i < PER; i++)
                v[r][i] = uint32_t(r) < rows && c0 + 32 * i < pieces ? load_here(row0 + r * pitch + size_t(c0 + 32 * i) * 8) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const T* f = reinterpret_cast<const T*>(&v[r][i]);
#pragma unroll
                for (int j = 0; j < 8; j++) { const float y = Elem<T>::to_f32(f[j]); s[r][j % 4] += y * y; }
            }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        float t = (s[r][0] + s[r][1]) + (s[r][2] + s[r][3]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        sum[r] = t;
    }
}
// ROWS: rows of a row warp, at most.  Norm: none, the cluster's blocks exchange their shares of a row's squares, every warp sums its whole
// rows itself, or any of them.  A kernel of its own for each is the faster one, by what it does not have to fetch of its own code: all
// of them and all numbers of rows in one, 16 heads x 9 to 32 rows, hidden 2048, 5 to 20 % slower.  With up to 8 rows, where that is least,
// one kernel for both projections of a block is the better choice yet (27 blocks of 4 sequences 709 us with two, 699 with one).
enum NormKind { kNoNorm = 0, kExchange = 1, kWhole = 2, kAny = 3 };
template <typename T, int NT, int ROWS, int Norm>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1, const T* x,
                const T* norm_w, T* out0, T* out1, const FewArgs a, uint32_t* __restrict__ status)
{
    constexpr uint32_t TMEM_COLS = ISSUERS * NT;
    constexpr int PER = max_kblocks(NT) * 8 / 32;      // pieces of 8 values per lane and row, at most
    extern __shared__ unsigned char few_smem[];
    const uint32_t raw = smem_u32(few_smem);                    // every block of a cluster sees the same offset
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = few_smem + (base - raw);
    const uint32_t bar0 = base + OFF_MISC;                      // full[STAGES], empty[STAGES], rows, acc, squares, sums
    auto full = [&](uint32_t s) { return bar0 + 8u * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8u * (STAGES + s); };
    const uint32_t a_full = bar0 + 8u * (2 * STAGES), acc_full = a_full + 8, ss_full = a_full + 16, red_full = a_full + 24;
    static_assert((2 * STAGES + 4) * 8 <= 224, "barriers overflow their area");
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC + 228);
    const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const uint32_t rank = cluster_rank(), tile = blockIdx.x / a.cs;
    const uint32_t kb0 = a.kb * rank / a.cs, kbs = a.kb * (rank + 1) / a.cs - kb0;         // this block's k-blocks (at least one)
    const uint32_t second = tile >= a.n_tiles0 ? 1u : 0u, tn = tile - (second ? a.n_tiles0 : 0u);

    grid_launch_dependents();
    if (tid == 0) {
        *abort_flag = 0;
        for (uint32_t s = 0; s < STAGES; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(a_full, ROW_WARPS);
        mbar_init(acc_full, min(uint32_t(ISSUERS), kbs));
        mbar_init(ss_full, a.cs * min(uint32_t(ROW_WARPS), a.M * a.split));
        mbar_init(red_full, a.cs * ROW_WARPS);
        mbar_init_fence();
    }
    if (warp == 1) tc_alloc<TMEM_COLS>(tmem_slot);
    tc_fence_before();
    // every block's barriers must exist before another one writes to it
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---- the weights are constant: their loads do not wait for earlier kernels
        if (lane == 0) {
            bool ok = true;
            const CUtensorMap* map = second ? &map_w1 : &map_w0;
            const int row0 = int((tn * a.kb + kb0) * BM);
            for (uint32_t i = 0; i < kbs; i++) {
                const uint32_t s = FewRing::stage(i);
                ok = mbar_wait<kPoll, true>(empty(s), FewRing::parity(i) ^ 1, abort_flag, status);
                if (!ok) break;
                mbar_expect_tx(full(s), W_BYTES);
                tma_load_2d(base + s * W_BYTES, map, full(s), 0, row0 + int(i * BM));
            }
            grid_dependency_wait();
        }
    } else if (warp < FIRST_ROW_WARP) {
        // ---- issuer p takes the k-blocks of its own stages (mla_few_ring.h), in order
        constexpr uint32_t IDESC = instr_desc(Fmt<T>::v, BM, NT), HI = desc_hi(1024);
        const uint32_t p = warp - 1;
        bool ok = p < kbs && mbar_wait<kPoll, true>(a_full, 0, abort_flag, status);
        for (uint32_t i = p, next; i < kbs && ok; i = next) {
            const uint32_t s = FewRing::stage(i);
            next = FewRing::next(i);
            ok = mbar_wait(full(s), FewRing::parity(i), abort_flag, status);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t da = desc_lo(base + s * W_BYTES), db = desc_lo(base + OFF_A + i * (NT * 128));
#pragma unroll
                for (int k = 0; k < BK / 16; k++)
                    tc_mma(tmem + p * NT, da + ((k * 32) >> 4), HI, db + ((k * 32) >> 4), HI, IDESC, (i == p && k == 0) ? 0u : 1u);
                tc_commit(empty(s));
                if (next >= kbs) tc_commit(acc_full);
            }
            __syncwarp();
        }
    } else {
        const uint32_t e = warp - FIRST_ROW_WARP, t = tid - FIRST_ROW_WARP * 32;
        T* out = second ? out1 : out0;
        const uint32_t N = second ? a.N[1] : a.N[0], o = tn * BM + t % BM;       // (indexed, the arguments are copied to the stack)
        const uint32_t pieces = kbs * 8, p0 = kb0 * 8, n_pieces = a.K / 8;
        // this warp's rows: e, e + 8, .., or with few of them a share of one row
        const uint32_t part = e & (a.split - 1), my_rows = e < a.M * a.split ? (a.split > 1 ? 1 : (a.M - e + ROW_WARPS - 1) / ROW_WARPS) : 0;
        auto row_of = [&](int r) -> uint32_t { return (e >> a.split_log2) + ROW_WARPS * r; };
        auto piece = [&](int k) -> uint32_t { return lane + 32 * (part + a.split * k); };
        uint4 g[PER];
        if (Norm != kNoNorm && (Norm != kAny || norm_w)) {
#pragma unroll
            for (int k = 0; k < PER; k++) {
                const uint32_t c = piece(k);
                g[k] = c < pieces && p0 + c < n_pieces ? load_here(norm_w + size_t(p0 + c) * 8) : make_uint4(0, 0, 0, 0);
            }
        }
        grid_dependency_wait();                    // x and out belong to earlier kernels
        // this thread finishes output o of the rows rank + cs * i, i = t / 128, t / 128 + 2, ..
        T res[NT / 2];
        if (a.residual) {
#pragma unroll
            for (int i = 0; i < NT / 2; i++) {
                const uint32_t row = rank + a.cs * (t / BM + 2 * i);
                if (o < N && row < a.M) res[i] = out[size_t(row) * N + o];
            }
        }
        bool ok = true;
        // ---- the rows into the operand tiles
        uint4 v[ROWS][PER];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            if (uint32_t(r) >= my_rows) break;
            const uint32_t row = row_of(r);
#pragma unroll
            for (int k = 0; k < PER; k++) {
                const uint32_t c = piece(k);
                v[r][k] = make_uint4(0, 0, 0, 0);
                if (c < pieces && p0 + c < n_pieces) v[r][k] = load_here(x + size_t(row) * a.K + size_t(p0 + c) * 8);
            }
        }
        // row r of this warp as the projection takes it
        auto normalise = [&](int r, float inv) {
#pragma unroll
            for (int k = 0; k < PER; k++) {
                if (32 * a.split * k >= pieces) break;
                const T *f = reinterpret_cast<const T*>(&v[r][k]), *w = reinterpret_cast<const T*>(&g[k]);
                uint32_t y[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    y[j] = Elem<T>::pack2(Elem<T>::to_f32(f[2 * j]) * inv * Elem<T>::to_f32(w[2 * j]), Elem<T>::to_f32(f[2 * j + 1]) * inv * Elem<T>::to_f32(w[2 * j + 1]));
                v[r][k] = make_uint4(y[0], y[1], y[2], y[3]);
            }
        };
        if (Norm == kWhole || (Norm == kAny && a.whole)) {
            if (my_rows) {
                float sum[ROWS];
                row_squares<T, ROWS>(x + size_t(row_of(0)) * a.K, size_t(ROW_WARPS) * a.K, my_rows, n_pieces, lane, sum);
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                    if (uint32_t(r) < my_rows) normalise(r, rsqrtf(sum[r] / float(a.K) + a.eps));
            }
        } else if ((Norm == kExchange || (Norm == kAny && norm_w)) && my_rows) {
            float* ss = reinterpret_cast<float*>(sm + OFF_SS);
            float sq[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                sq[r] = 0.0f;
                if (uint32_t(r) >= my_rows) break;
#pragma unroll
                for (int k = 0; k < PER; k++) {
                    if (32 * a.split * k >= pieces) break;
                    const T* f = reinterpret_cast<const T*>(&v[r][k]);
#pragma unroll
                    for (int j = 0; j < 8; j++) { const float y = Elem<T>::to_f32(f[j]); sq[r] += y * y; }
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) sq[r] += __shfl_xor_sync(0xffffffffu, sq[r], off);
            }
            if (lane < a.cs) {                     // lane l tells block l
                const uint32_t dst = map_to_rank(base + OFF_SS, lane) + (rank * 32 + e) * 4;
#pragma unroll
                for (int r = 0; r < ROWS; r++)
                    if (uint32_t(r) < my_rows) asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;\n" ::"r"(dst + ROW_WARPS * r * 4), "f"(sq[r]) : "memory");
                mbar_arrive_cluster(map_to_rank(ss_full, lane));
            }
            __syncwarp();
            ok = mbar_wait<kSleepCluster>(ss_full, 0, abort_flag, status);
            ok = __all_sync(0xffffffffu, ok);
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                if (uint32_t(r) >= my_rows) break;
                float tot = 0.0f;
                const uint32_t at = (e & ~(a.split - 1)) + ROW_WARPS * r;        // the row's first entry
                for (uint32_t s = 0; s < a.cs; s++)
#pragma unroll
                    for (uint32_t p = 0; p < ROW_WARPS; p++) if (p < a.split) tot += ss[s * 32 + at + p];
                normalise(r, rsqrtf(tot / float(a.K) + a.eps));
            }
        }
        // rows behind the last one keep what the memory held: a row reaches no column but its own
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            if (uint32_t(r) >= my_rows) break;
            const uint32_t row = row_of(r);
#pragma unroll
            for (int k = 0; k < PER; k++) {
                const uint32_t c = piece(k);
                if (c < pieces) *reinterpret_cast<uint4*>(sm + OFF_A + (c / 8) * (NT * 128) + row * 128 + (((c % 8) ^ (row & 7)) << 4)) = v[r][k];
            }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full);

        // ---- this block's sums to the blocks that finish them: warp e reads lanes 32 * (warp % 4).. of columns NT / 2 * (e / 4)..
        constexpr int HALF = NT / 2;
        const uint32_t q4 = warp % 4, c0 = (e / 4) * HALF, slots = NT >> a.cs_log2;
        ok = mbar_wait(acc_full, 0, abort_flag, status) && ok;
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        if (c0 < a.M && ok) {
            const uint32_t acc = tmem + ((q4 * 32u) << 16) + c0, n_acc = min(uint32_t(ISSUERS), kbs);
            uint32_t w[ISSUERS][HALF];
#pragma unroll
            for (int p = 0; p < ISSUERS; p++) if (uint32_t(p) < n_acc) tc_ldn(acc + p * NT, w[p]);
            tc_wait_ld();
            const uint32_t dst = base + OFF_RED + (rank * slots * BM + q4 * 32 + lane) * 4;
#pragma unroll
            for (int i = 0; i < HALF; i++) {
                const uint32_t c = c0 + i;
                if (c >= a.M) break;
                float s = __uint_as_float(w[0][i]);
#pragma unroll
                for (int p = 1; p < ISSUERS; p++) if (uint32_t(p) < n_acc) s += __uint_as_float(w[p][i]);
                asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;\n" ::"r"(map_to_rank(dst + (c >> a.cs_log2) * (BM * 4), c & (a.cs - 1))), "f"(s) : "memory");
            }
        }
        __syncwarp();
        if (lane < a.cs) announce_share(map_to_rank(red_full, lane), ok);
        __syncwarp();
        cluster_arrive();
        const bool all = mbar_wait<kSleepCluster>(red_full, 0, abort_flag, status);
        ok = __all_sync(0xffffffffu, all && ok);
        const float* red = reinterpret_cast<const float*>(sm + OFF_RED);
#pragma unroll
        for (int i = 0; i < NT / 2; i++) {
            const uint32_t slot = t / BM + 2 * i, row = rank + a.cs * slot;
            if (row >= a.M || o >= N || !ok) break;
            float s = 0.0f;
#pragma unroll
            for (uint32_t r = 0; r < MAX_CLUSTER; r++) if (r < a.cs) s += red[(r * slots + slot) * BM + t % BM];
            T y = Elem<T>::from_f32(s);
            if (a.residual) y = Elem<T>::from_f32(Elem<T>::to_f32(res[i]) + Elem<T>::to_f32(y));
            out[size_t(row) * N + o] = y;
        }
        tc_fence_before();
    }
    // no block may leave while another one may still write to it: the row warps arrived when they had sent their last word
    tc_fence_before();
    __syncwarp();
    if (warp < FIRST_ROW_WARP) cluster_arrive();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc<TMEM_COLS>(tmem);
    }
}

cudaLaunchConfig_t launch_config(cudaLaunchAttribute (&at)[2], uint32_t blocks, uint32_t cs, const LaunchStream& st)
{
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = st.plain ? 0 : 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cs;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = st.st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

template <typename T, typename F>
void for_each_kernel(F f)
{
    f(gemm_few_kernel<T, 16, 1, kAny>);
    f(gemm_few_kernel<T, 16, 2, kNoNorm>); f(gemm_few_kernel<T, 16, 2, kExchange>); f(gemm_few_kernel<T, 16, 2, kWhole>);
    f(gemm_few_kernel<T, 32, 4, kNoNorm>); f(gemm_few_kernel<T, 32, 4, kExchange>); f(gemm_few_kernel<T, 32, 4, kWhole>);
}

template <typename T>
cudaError_t configure_type()
{
    auto set = [](auto kernel) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    };
    cudaError_t e = cudaSuccess;
    for_each_kernel<T>([&](auto kernel) { if (e == cudaSuccess) e = set(kernel); });
    return e;
}

template <typename T>
int launch_type(const GemmCall& g, uint32_t cs, uint32_t* status, const LaunchStream& st)
{
    FewArgs a{};
    a.M = g.M;
    a.K = g.K;
    a.kb = (g.K + BK - 1) / BK;
    a.cs = cs;
    a.cs_log2 = cs == 8 ? 3 : cs / 2;
    a.split_log2 = g.M <= 1 ? 3 : g.M <= 2 ? 2 : g.M <= 4 ? 1 : 0;
    a.split = 1u << a.split_log2;
    a.eps = g.eps;
    a.residual = g.residual ? 1u : 0u;
    uint32_t tiles = 0;
    for (int i = 0; i < g.n_weights; i++) {
        a.N[i] = g.w[i].N;
        tiles += (g.w[i].N + BM - 1) / BM;
        if (i == 0) a.n_tiles0 = tiles;
    }
    const int last = g.n_weights - 1;
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = launch_config(at, tiles * cs, cs, st);
    auto go = [&](auto kernel) {
        return int(cudaLaunchKernelEx(&cfg, kernel, *g.w[0].map, *g.w[last].map, static_cast<const T*>(g.A), static_cast<const T*>(g.norm_w),
                                      static_cast<T*>(g.w[0].out), static_cast<T*>(g.w[last].out), a, status));
    };
    const int norm = !g.norm_w ? kNoNorm : gemm_few_tc5_exchanges(g) ? kExchange : kWhole;
    a.whole = norm == kWhole;
    auto pick = [&](auto none, auto exchange, auto whole) { return norm == kNoNorm ? go(none) : norm == kWhole ? go(whole) : go(exchange); };
    if (g.M <= 8) return go(gemm_few_kernel<T, 16, 1, kAny>);
    if (g.M <= 16) return pick(gemm_few_kernel<T, 16, 2, kNoNorm>, gemm_few_kernel<T, 16, 2, kExchange>, gemm_few_kernel<T, 16, 2, kWhole>);
    return pick(gemm_few_kernel<T, 32, 4, kNoNorm>, gemm_few_kernel<T, 32, 4, kExchange>, gemm_few_kernel<T, 32, 4, kWhole>);
}

}  // namespace

int gemm_few_tc5_configure(int dtype) { return int(dtype == 0 ? configure_type<__half>() : configure_type<__nv_bfloat16>()); }

// clusters of 1, 2, 4 and 8 blocks that the current device holds at a time
int gemm_few_tc5_clusters(int dtype, uint32_t (&n)[4])
{
    for (int i = 0; i < 4; i++) {
        cudaLaunchAttribute at[2];
        const cudaLaunchConfig_t cfg = launch_config(at, 1u << i, 1u << i, cudaStream_t(nullptr));
        int c = 0;
        const cudaError_t e = dtype == 0 ? cudaOccupancyMaxActiveClusters(&c, gemm_few_kernel<__half, 32, 4, kExchange>, &cfg)
                                         : cudaOccupancyMaxActiveClusters(&c, gemm_few_kernel<__nv_bfloat16, 32, 4, kExchange>, &cfg);
        if (e != cudaSuccess) return int(e);
        n[i] = uint32_t(c);
    }
    return 0;
}

// Blocks of a cluster for this call, 0: not a call for this kernel, or one that the general kernel is faster at.  Its tiles must be
// resident at once: a second round of clusters would cost as much as the first, and the general kernel's equal runs have none.  The
// most blocks that fit, also where they leave fewer SMs to the launches before and behind (16 heads x 4 rows: clusters of 4 808 us,
// of 2 835).
// What a cluster gains over the general kernel are the k-blocks that a tile's block does not walk itself, and the hand-over of a cut
// tile; what it loses is the way of the sums from block to block, more with more blocks and with more rows that each must finish.
// One projection from packed weights in a chain of launches of the same kernel, general kernel -> this one (us; - / +: the rule
// refuses / takes):
//   k-blocks  tiles  cluster  blocks    4 rows         16 rows        32 rows
//      4       16       4       64     2.6 -> 2.9     2.8 -> 3.2     3.2 -> 3.8     -
//      8       32       4      128     3.1 -> 4.2     3.2 -> 4.5     3.8 -> 5.0     -
//     10       16       8      128     3.2 -> 3.1     3.4 -> 3.5     4.1 -> 4.1     +
//     10       24       4       96     3.5 -> 4.0     3.8 -> 4.2     4.5 -> 4.8     + up to 8 rows
//     10       72       2      144     4.5 -> 5.1     4.7 -> 5.6     5.4 -> 6.1     -
//     16       48       2       96     5.1 -> 4.7     5.3 -> 5.2     6.0 -> 5.9     +
//     16       72       2      144     5.9 -> 6.3     6.0 -> 6.7     6.6 -> 7.3     + up to 16 rows
//     16       96       1       96     6.8 -> 7.6     7.0 -> 8.5                    -
//     32       24       4       96     7.0 -> 5.0     7.4 -> 5.3     8.6 -> 5.8     +
//     32       56       2      112     9.3 -> 8.0     9.6 -> 8.5                    +
// In a block the rule takes it a little earlier than this chain says, because there the instructions of the one kernel are near, and
// those of the other are fetched.  With limits as the chain has them (8 k-blocks spared in clusters of 8, 9 to 12 in those of 4, 8 and at most 112
// blocks in those of 2) blocks of 4 to 8 heads, hidden 1024 to 7168, take 0.93 to 1.07 of their time, 1.005 in the mean, and more
// where it is a user's common case: 5 heads, hidden 2048, 2 / 8 / 17 rows 24.7 / 24.4 / 28.0 us per layer, 25.5 / 25.8 / 29.7.
// With the norm in front the general kernel has a launch more, and only single blocks with more than 8 rows lose: 64 heads, hidden
// 4096, q_lora 512, all by the general kernel / both projections here / as the rule has it: 8 rows 13.0 / 10.6 / 10.6, 16 rows 13.2 /
// 14.3 / 12.7, 32 rows 15.5 / 19.0 / 15.7.  16 heads x 4 rows: hidden 4096 10.8 -> 9.3, hidden 7168 with q_lora 1536 18.4 -> 15.1.
// q_b alone by the general kernel where q_a exchanges (hidden 3072 and 4096, q_lora 512 and 768, 9 to 32 rows): slower in 31 of 36 blocks,
// 0.97 to 1.05.
uint32_t gemm_few_tc5_cluster(const GemmCall& g, const uint32_t (&resident)[4])
{
    if (!g.packed || g.M > 32 || g.M == 0) return 0;
    const uint32_t kb = (g.K + BK - 1) / BK, kmax = uint32_t(max_kblocks(g.M <= 16 ? 16 : 32));
    uint32_t tiles = 0;
    for (int i = 0; i < g.n_weights; i++) tiles += (g.w[i].N + BM - 1) / BM;
    for (int i = 3; i >= 0; i--) {              // the most blocks that fit
        const uint32_t cs = 1u << i;
        if (cs > kb || tiles > resident[i]) continue;
        const uint32_t kbs = (kb + cs - 1) / cs;
        if (kbs > kmax) return 0;
        if (g.norm_w) return cs > 1 || g.M <= 8 ? cs : 0;
        const uint32_t blocks = tiles * cs, spared = g.M <= 8 && blocks <= 112 ? 5 : blocks <= 64 ? 6 : 8;
        return cs > 1 && kb - kbs >= spared && (cs > 2 || g.M <= 16 || blocks <= 96) ? cs : 0;
    }
    return 0;
}

// Whether the cluster's blocks exchange their shares of a row's squares; otherwise every warp sums its whole rows itself.
// A warp's whole rows are a trip to L2 for every 256 pieces of 8 values of them, the exchange is one trip and one through the cluster:
// (16 heads, hidden 2048, input projections of 1 / 8 / 16 / 32 rows: 7.0 / 7.1 / 7.9 / 9.9 us by exchange, 5.7 / 5.8 / 7.0 / 8.6
// whole.)  For short rows of more than 8, where it matters least, the kernel is the better one whose instructions the projection just
// before has fetched.  Blocks, us per layer, q_b by exchange / whole, 12 and 32 rows: 16 heads, hidden 2048, q_lora 512 (whole rows before)
// 33.9 / 32.3 and 41.8 / 37.8; 32 heads, hidden 4096, q_lora 512 (exchange before) 41.7 / 41.6 and 52.9 / 53.9; 16 heads, hidden 7168, q_lora 768,
// 32 rows (the general kernel before) 53.9 / 51.7.
bool gemm_few_tc5_exchanges(const GemmCall& g)
{
    if (!g.norm_w) return false;
    return g.M <= 8 ? g.K > 4096 : g.K > 2048 || (g.K < 1024 && g.exchange_near);
}

int launch_gemm_few_tc5(int dtype, const GemmCall& g, uint32_t cs, uint32_t* status, const LaunchStream& st)
{
    return dtype == 0 ? launch_type<__half>(g, cs, status, st) : launch_type<__nv_bfloat16>(g, cs, status, st);
}

}  // namespace mla
