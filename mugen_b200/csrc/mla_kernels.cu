// Small kernels around the attention core: latent-row append, partial merge + W_UV projection, bulk row copy.  sm_100a.
#include "mla_append.cuh"
#include "mla_launch.h"

namespace mla {

// ------------------------------------------------------------------------------------------
// Append on its own (mla_append.cuh): eight rows per block, one warp each.
// ------------------------------------------------------------------------------------------
constexpr int kAppendWarps = 8;
template <typename T>
__global__ void __launch_bounds__(32 * kAppendWarps)
append_kernel(const AppendArgs a, uint32_t* __restrict__ status)
{
    __shared__ __align__(16) unsigned char smem[kAppendWarps * kAppendRowSmem];
    grid_launch_dependents();
    AppendRow<T> row;
    row.prepare(a, 0, blockIdx.x * kAppendWarps + threadIdx.x / 32, status);
    grid_dependency_wait();              // kv_a comes from an earlier kernel of the stream
    row.run(a, smem + (threadIdx.x / 32) * kAppendRowSmem);
}

int launch_append(int dtype, const void* kv_a, void* layer_pool, uint64_t pool_slots, const void* norm_w, const float* cos_sin,
                  uint32_t cs_rows, float eps, const StepMeta& m, uint32_t* status, const LaunchStream& st)
{
    if (m.app_rows == 0) return 0;
    const AppendArgs a{kv_a, layer_pool, pool_slots, norm_w, cos_sin, cs_rows, eps, m.app_pos, m.app_slot, m.app_rows, 1};
    const dim3 grid((m.app_rows + kAppendWarps - 1) / kAppendWarps), block(32 * kAppendWarps);
    return dtype == 0 ? int(launch_pdl(append_kernel<__half>, grid, block, 0, st, a, status))
                      : int(launch_pdl(append_kernel<__nv_bfloat16>, grid, block, 0, st, a, status));
}

// ------------------------------------------------------------------------------------------
// The step's metadata from page-locked host memory into the device buffer, read by the SMs.  A few KB: what bounds it is one round
// trip over the host link (about 1.5 us), so every thread asks for all its pieces at once, and ahead of the wait for the kernels
// before it, which may still read what the buffer held.  A copy-engine transfer takes 3.5 to 4 us at this size, starts only when those
// kernels have ended, and sits between them and the step's first kernel with a gap of 2 us on either side.  Copies against this kernel, us per
// pass, SM clock 1,965 MHz: one user, 16 heads x 27 layers, two uploads 56.9 -> 45.4; 27 blocks of 16 heads x 4 sequences 707 -> 703; 8 sequences by
// calls, eight layers of 128 heads 503 -> 499; one sequence of 131,072 tokens, four layers, unchanged.
// ------------------------------------------------------------------------------------------
constexpr int kFetchThreads = 256, kFetchPieces = 4;         // pieces of 16 bytes per thread, all in flight together
__global__ void __launch_bounds__(kFetchThreads)
fetch_kernel(const uint4* host, uint4* device, uint32_t pieces)
{
    grid_launch_dependents();
    uint4 v[kFetchPieces];
    const uint32_t i0 = blockIdx.x * (kFetchThreads * kFetchPieces) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kFetchPieces; k++) if (i0 + k * kFetchThreads < pieces) v[k] = __ldcv(host + i0 + k * kFetchThreads);
    grid_dependency_wait();
#pragma unroll
    for (int k = 0; k < kFetchPieces; k++) if (i0 + k * kFetchThreads < pieces) device[i0 + k * kFetchThreads] = v[k];
}

int launch_fetch(const void* host, void* device, uint32_t pieces, cudaStream_t st)
{
    constexpr uint32_t per = kFetchThreads * kFetchPieces;
    if (pieces == 0) return 0;
    return int(launch_pdl(fetch_kernel, dim3((pieces + per - 1) / per), dim3(kFetchThreads), 0, st, static_cast<const uint4*>(host),
                          static_cast<uint4*>(device), pieces));
}

// ------------------------------------------------------------------------------------------
// Bulk copy of ready-made latent rows into a sequence's pages (cache fill / restore).
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
write_rows_kernel(const uint4* __restrict__ src, uint4* __restrict__ pool, uint64_t pool_slots,
                  const uint32_t* __restrict__ table, uint32_t row_begin, uint32_t n,
                  uint32_t* __restrict__ status)
{
    constexpr int kChunks = kRow * 2 / 16;
    const uint32_t r = blockIdx.x * 4 + threadIdx.x / 32;   // one warp per row
    if (r >= n) return;
    const uint32_t row = row_begin + r;
    const uint64_t slot = uint64_t(table[row / kPage]) * kPage + row % kPage;
    if (slot >= pool_slots) {
        if ((threadIdx.x & 31) == 0) atomicOr(status, ST_BAD_SLOT);
        return;
    }
    for (int c = threadIdx.x & 31; c < kChunks; c += 32)
        pool[slot * kChunks + c] = src[size_t(r) * kChunks + c];
}

void launch_write_rows(const void* src, void* layer_pool, uint64_t pool_slots, const uint32_t* table,
                       uint32_t row_begin, uint32_t n, uint32_t* status, cudaStream_t st)
{
    if (n == 0) return;
    write_rows_kernel<<<(n + 3) / 4, 128, 0, st>>>(static_cast<const uint4*>(src),
                                                    static_cast<uint4*>(layer_pool), pool_slots,
                                                    table, row_begin, n, status);
}

template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------------------------------
// Merge of partial softmax states + W_UV projection (reference: transformer.cpp:2610-2620).
// A partial record is 514 floats per (part, head): m (log2 domain), l, acc[512].
//   M = max m_p ;  w_p = 2^(m_p - M) ;  o_c = sum w_p*acc_p / sum w_p*l_p
//   out[r][h][j] = T( sum_d o_c[d] * W_UV[h*128+j][d] )
// Parts of row r are the row's split-KV segments, as its RowParts says.
// ------------------------------------------------------------------------------------------

// The merged, still un-normalised state of every (row, head) written out (the per-GPU partial of a KV-range-sharded
// sequence): one block per (head, row); the 16 warps take a slice of the row's parts each (a lane owns dims
// 64*k + 2*lane (+1), k = 0..7, so a warp load covers whole lines of a record), their sums meet in shared memory and
// every thread folds one dim.  One sequence cut into 74 segments costs two round trips to memory.
__global__ void __launch_bounds__(512)
export_partial_kernel(const float* __restrict__ recs, const RowParts* __restrict__ parts, uint32_t rec_stride,
                      float* __restrict__ exported, uint32_t H)
{
    __shared__ __align__(8) float scratch[16][kRank], ml_s[16][2];
    grid_launch_dependents();
    const uint32_t h = blockIdx.x, r = blockIdx.y, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const RowParts rp = parts[r];
    uint32_t pb = rp.begin, pe = rp.end;
    auto rec_of = [&](uint32_t p) -> const float* { return recs + (size_t(p) * rec_stride + rp.rec_off + h) * kPart; };
    const uint32_t chunk = (pe - pb + 15) / 16;
    pb = min(pe, pb + warp * chunk);
    pe = min(pe, pb + chunk);
    float M = -INFINITY, L = 0.0f, acc[16];
#pragma unroll
    for (int k = 0; k < 16; k++) acc[k] = 0.0f;
    grid_dependency_wait();              // the states belong to the attention kernel; the plan was there before
    for (uint32_t p = pb; p < pe; p += 4) {
        float2 ml[4], v[4][8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool on = p + i < pe;
            const float* rc = rec_of(on ? p + i : pb);
            ml[i] = on ? *reinterpret_cast<const float2*>(rc) : make_float2(-INFINITY, 0.0f);
#pragma unroll
            for (int k = 0; k < 8; k++)
                v[i][k] = on ? *reinterpret_cast<const float2*>(rc + 2 + 64 * k + 2 * lane) : make_float2(0.0f, 0.0f);
        }
        const float Mn = fmaxf(fmaxf(M, ml[0].x), fmaxf(fmaxf(ml[1].x, ml[2].x), ml[3].x));
        if (Mn > -INFINITY) {
            const float sc = exp2f(M - Mn);
            L *= sc;
#pragma unroll
            for (int k = 0; k < 16; k++) acc[k] *= sc;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float w = exp2f(ml[i].x - Mn);
                L = fmaf(w, ml[i].y, L);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    acc[2 * k] = fmaf(w, v[i][k].x, acc[2 * k]);
                    acc[2 * k + 1] = fmaf(w, v[i][k].y, acc[2 * k + 1]);
                }
            }
            M = Mn;
        }
    }
    // thread t folds dim t over the sixteen slices
#pragma unroll
    for (int k = 0; k < 8; k++) *reinterpret_cast<float2*>(scratch[warp] + 64 * k + 2 * lane) = make_float2(acc[2 * k], acc[2 * k + 1]);
    if (lane == 0) { ml_s[warp][0] = M; ml_s[warp][1] = L; }
    __syncthreads();
    float big = -INFINITY;
#pragma unroll
    for (int j = 0; j < 16; j++) big = fmaxf(big, ml_s[j][0]);
    float sum = 0.0f, lsum = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const float w = big == -INFINITY ? 0.0f : exp2f(ml_s[j][0] - big);
        sum = fmaf(w, scratch[j][threadIdx.x], sum);
        lsum = fmaf(w, ml_s[j][1], lsum);
    }
    float* ex = exported + (size_t(r) * H + h) * kPart;
    ex[2 + threadIdx.x] = sum;
    if (threadIdx.x == 0) { ex[0] = big; ex[1] = lsum; }
}

// Same merge, projection on the warp-level tensor path.  Block = (head, group of up to 4 row tiles
// of 16 query rows), 16 warps.  W_UV_h (128 x 512, 128 KB) is staged ONCE per block in shared
// memory with 16-byte loads and serves every row tile of the block.  Per row tile:
//   1. warp r finds row r's M and 1/L: its lanes take the row's parts in parallel;
//   2. the merged, normalised o_c[16 x 512] is built in shared memory as TWO 16-bit matrices,
//      hi = T(o) and lo = T(o - hi): together they carry ~16 (bf16) / 22 (fp16) mantissa bits, so
//      the float state is not rounded to the storage type before W_UV; thread -> (row, 16 dims);
//   3. out[16 x 128] = (hi + lo)[16 x 512] . W_UV_h^T, m16n8k16 with f32 accumulate; warp w owns
//      outputs [8w, 8w+8), all fragments come from shared memory through ldmatrix.
constexpr int kMergeTilesPerBlock = 4;
constexpr int kMergePitch = kRank + 8;               // elements; keeps ldmatrix rows on distinct banks
constexpr size_t kMergeSmem = size_t(kVDim + 32) * kMergePitch * 2 + 16 * 4 * 4;
template <typename T>
__global__ void __launch_bounds__(512)
merge_outproj_mma_kernel(const float* __restrict__ recs, const RowParts* __restrict__ parts, uint32_t rec_stride,
                         const T* __restrict__ w_uv, T* __restrict__ out, uint32_t rows, uint32_t H)
{
    constexpr int PITCH = kMergePitch;
    extern __shared__ __align__(16) unsigned char merge_smem[];
    T* w_s = reinterpret_cast<T*>(merge_smem);                       // [128][PITCH]
    T* a_hi = w_s + size_t(kVDim) * PITCH;                           // [16][PITCH]
    T* a_lo = a_hi + 16 * PITCH;                                     // [16][PITCH]
    float* row_m = reinterpret_cast<float*>(a_lo + 16 * PITCH);
    float* row_inv = row_m + 16;
    uint32_t* row_pb = reinterpret_cast<uint32_t*>(row_inv + 16);
    uint32_t* row_pe = row_pb + 16;
    const uint32_t h = blockIdx.x, tid = threadIdx.x;
    const uint32_t warp = tid / 32, lane = tid % 32, g = lane / 4, t4 = lane % 4;
    const uint32_t rt_begin = blockIdx.y * kMergeTilesPerBlock;
    const uint32_t rt_end = min(rt_begin + kMergeTilesPerBlock, (rows + 15) / 16);
    auto rec_of = [&](uint32_t r, uint32_t p) -> const float* {
        return recs + (size_t(p) * rec_stride + parts[r].rec_off + h) * kPart;
    };
    {   // stage W_UV_h: 128 rows x 64 chunks of 16 bytes, 16 chunks per thread, all in flight at once
        const uint4* src = reinterpret_cast<const uint4*>(w_uv + size_t(h) * kVDim * kRank);
        uint4 v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = src[tid + 512 * i];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int c = tid + 512 * i, row = c / 64, ch = c % 64;
            *reinterpret_cast<uint4*>(w_s + size_t(row) * PITCH + ch * 8) = v[i];
        }
    }
    const int mi = lane / 8, lr = lane % 8;
    const uint32_t hi_addr = static_cast<uint32_t>(__cvta_generic_to_shared(a_hi + ((mi % 2) * 8 + lr) * PITCH + (mi / 2) * 8));
    const uint32_t lo_addr = static_cast<uint32_t>(__cvta_generic_to_shared(a_lo + ((mi % 2) * 8 + lr) * PITCH + (mi / 2) * 8));
    // B fragments of outputs [8w, 8w+8) for two k-steps per ldmatrix.x4: matrices (k0-7, k8-15) of step s, then of step s+1
    const uint32_t w_addr = static_cast<uint32_t>(__cvta_generic_to_shared(w_s + size_t(warp * 8 + lr) * PITCH + mi * 8));
    for (uint32_t rt = rt_begin; rt < rt_end; rt++) {
        const uint32_t r0 = rt * 16;
        {
            const uint32_t r = r0 + warp;                // warp <-> row
            uint32_t pb = 0, pe = 0;
            if (r < rows) { pb = parts[r].begin; pe = parts[r].end; }
            float M = -INFINITY;
            for (uint32_t p = pb + lane; p < pe; p += 32) M = fmaxf(M, rec_of(r, p)[0]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
            float L = 0.0f;
            if (M > -INFINITY)
                for (uint32_t p = pb + lane; p < pe; p += 32) {
                    const float* rc = rec_of(r, p);
                    L = fmaf(exp2f(rc[0] - M), rc[1], L);
                }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
            if (lane == 0) {
                row_m[warp] = M;
                row_inv[warp] = L > 0.0f ? 1.0f / L : 0.0f;
                row_pb[warp] = pb;
                row_pe[warp] = pe;
            }
        }
        __syncthreads();                                 // also: W_UV staged (first tile), previous tile's MMAs done
        {   // thread -> row tid/32, dims (tid%32)*16 .. +15
            const uint32_t rr = tid / 32, r = r0 + rr, d0 = (tid % 32) * 16;
            const float M = row_m[rr], inv = row_inv[rr];
            const uint32_t pb = row_pb[rr], pe = row_pe[rr];
            float acc[16];
#pragma unroll
            for (int i = 0; i < 16; i++) acc[i] = 0.0f;
            if (inv > 0.0f)
                for (uint32_t p = pb; p < pe; p++) {
                    const float* rc = rec_of(r, p);
                    const float w = exp2f(rc[0] - M);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float2 v = *reinterpret_cast<const float2*>(rc + 2 + d0 + 2 * i);
                        acc[2 * i] = fmaf(w, v.x, acc[2 * i]);
                        acc[2 * i + 1] = fmaf(w, v.y, acc[2 * i + 1]);
                    }
                }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float o0 = acc[2 * i] * inv, o1 = acc[2 * i + 1] * inv;
                const T h0 = Elem<T>::from_f32(o0), h1 = Elem<T>::from_f32(o1);
                *reinterpret_cast<uint32_t*>(a_hi + rr * PITCH + d0 + 2 * i) = Elem<T>::pack2(o0, o1);
                *reinterpret_cast<uint32_t*>(a_lo + rr * PITCH + d0 + 2 * i) =
                    Elem<T>::pack2(o0 - Elem<T>::to_f32(h0), o1 - Elem<T>::to_f32(h1));
            }
        }
        __syncthreads();
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
        for (int ks = 0; ks < kRank / 16; ks += 2) {
            uint32_t bw[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                         : "=r"(bw[0]), "=r"(bw[1]), "=r"(bw[2]), "=r"(bw[3]) : "r"(w_addr + ks * 32));
#pragma unroll
            for (int u = 0; u < 2; u++) {
                uint32_t ah[4], al[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                             : "=r"(ah[0]), "=r"(ah[1]), "=r"(ah[2]), "=r"(ah[3]) : "r"(hi_addr + (ks + u) * 32));
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                             : "=r"(al[0]), "=r"(al[1]), "=r"(al[2]), "=r"(al[3]) : "r"(lo_addr + (ks + u) * 32));
                mma16816<T>(c, ah, bw[2 * u], bw[2 * u + 1]);
                mma16816<T>(c, al, bw[2 * u], bw[2 * u + 1]);
            }
        }
        const int col = warp * 8 + t4 * 2;
        if (r0 + g < rows)
            *reinterpret_cast<uint32_t*>(out + (size_t(r0 + g) * H + h) * kVDim + col) = Elem<T>::pack2(c[0], c[1]);
        if (r0 + g + 8 < rows)
            *reinterpret_cast<uint32_t*>(out + (size_t(r0 + g + 8) * H + h) * kVDim + col) = Elem<T>::pack2(c[2], c[3]);
        __syncthreads();                                 // a_hi / a_lo / row_* are rewritten by the next tile
    }
}

// Once per device, with that device current (function attributes are per device).
int merge_mma_configure()
{
    cudaError_t e = cudaFuncSetAttribute(merge_outproj_mma_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMergeSmem));
    if (e != cudaSuccess) return int(e);
    e = cudaFuncSetAttribute(merge_outproj_mma_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMergeSmem));
    return int(e);
}

void launch_merge(int dtype, const float* recs, const StepMeta& m, const void* w_uv, void* out, uint32_t H, cudaStream_t st)
{
    const uint32_t rows = m.rows * m.layers;
    if (rows == 0) return;
    const uint32_t row_tiles = (rows + 15) / 16;
    dim3 grid16(H, (row_tiles + kMergeTilesPerBlock - 1) / kMergeTilesPerBlock);
    if (dtype == 0)
        merge_outproj_mma_kernel<__half><<<grid16, 512, kMergeSmem, st>>>(
            recs, m.parts, m.rec_stride, static_cast<const __half*>(w_uv), static_cast<__half*>(out), rows, H);
    else
        merge_outproj_mma_kernel<__nv_bfloat16><<<grid16, 512, kMergeSmem, st>>>(
            recs, m.parts, m.rec_stride, static_cast<const __nv_bfloat16*>(w_uv), static_cast<__nv_bfloat16*>(out), rows, H);
}

int launch_export_partial(const float* recs, const StepMeta& m, float* exported, uint32_t H, cudaStream_t st)
{
    if (m.rows == 0) return 0;
    return int(launch_pdl(export_partial_kernel, dim3(H, m.rows), dim3(512), 0, st, recs, m.parts, m.rec_stride, exported, H));
}

}  // namespace mla
