// The cache append: RMSNorm(c_kv)*w, NeoX RoPE(k_rope) and the scatter of a 576-value row into its page slot.
// Follows the reference's statements one by one so that the stored bits equal the CPU path's
// (src/core/model/transformer.cpp:3935-3948 and :3964-3975):
//   ss = sum_i x_i*x_i            sequential, float, multiply and add rounded separately
//   r  = 1 / sqrt(ss/512 + eps)
//   c_kv[i] = T( (x_i*r) * w_i )  two multiplies, one final rounding
//   k[i]    = T( x0*cos - x1*sin ),  k[i+32] = T( x1*cos + x0*sin )   from the original x0, x1
// cos/sin come from a host-built table (the host evaluates them with the same libm calls as the CPU path; device
// cosf/sinf are not bit-identical to glibc's).  The squares are formed in parallel (each product is rounded on its own, as
// in the reference), then ONE lane adds them in index order: the sum's rounding sequence is the reference's.
#pragma once

#include "mla_common.cuh"

namespace mla {

struct AppendArgs {          // rows == 0: no append blocks in this launch
    const void* kv_a;        // [layers][rows][576]
    void* pool;              // the first layer's slice of the cache pool
    uint64_t pool_slots;     // token slots per layer
    const void* norm_w;      // [layers][512]
    const float* cos_sin;
    uint32_t cs_rows;
    float eps;
    const uint32_t* row_pos;
    const uint64_t* row_slot;
    uint32_t rows;
    uint32_t wait_first;     // kv_a may be the output of the kernel just before this one in the stream
};

constexpr int kAppendRowSmem = kRow * 2 + kRank * 4;      // 3,200 bytes of shared memory per row (16-byte aligned)

// One new cache row by one warp, in two steps.  `prepare` reads what the step's metadata and the constant tables hold (slot,
// position, cos / sin, norm weights) and may run ahead of the grid dependency wait; `run` needs kv_a.  Left where they are
// used these loads form a chain of dependent round trips to memory (~1 us each) in a kernel whose whole budget is a few
// microseconds.  The row is normalised and rotated in place in shared memory: every element (pair) has one lane.  What
// bounds it then is the sum of squares, a chain of 512 dependent additions (~1.1 us).
template <typename T>
struct AppendRow {
    bool live = false;
    uint64_t slot = 0;
    uint32_t layer = 0, row = 0;
    float cs = 0.0f, sn = 0.0f;
    T nw[kRank / 32];

    __device__ __forceinline__ void prepare(const AppendArgs& a, uint32_t layer_, uint32_t r, uint32_t* status) {
        const uint32_t lane = threadIdx.x % 32;
        layer = layer_;
        row = r;
        live = r < a.rows;
        if (!live) return;
        slot = a.row_slot[r];
        const uint32_t pos = a.row_pos[r];
        if (slot == ~uint64_t(0)) { live = false; return; }                    // a query-only row: nothing to append
        if (slot >= a.pool_slots || pos >= a.cs_rows) {
            if (lane == 0) atomicOr(status, ST_BAD_SLOT);
            live = false;
            return;
        }
        cs = a.cos_sin[size_t(pos) * kRope + lane];
        sn = a.cos_sin[size_t(pos) * kRope + 32 + lane];
        const T* norm_w = static_cast<const T*>(a.norm_w) + size_t(layer) * kRank;
#pragma unroll
        for (int k = 0; k < kRank / 32; k++) nw[k] = norm_w[lane + 32 * k];
    }

    __device__ __forceinline__ void run(const AppendArgs& a, unsigned char* smem) const {
        if (!live) return;
        const uint32_t lane = threadIdx.x % 32;
        float* sq = reinterpret_cast<float*>(smem);
        T* x = reinterpret_cast<T*>(smem + kRank * 4);
        constexpr uint32_t kChunks = kRow * 2 / 16;   // 72 x 16 bytes
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const T*>(a.kv_a) + (size_t(layer) * a.rows + row) * kRow);
        uint4 chunk[3];
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) if (lane + 32 * k < kChunks) chunk[k] = src[lane + 32 * k];
        __syncwarp();                                  // the row before has left the buffer
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) if (lane + 32 * k < kChunks) reinterpret_cast<uint4*>(x)[lane + 32 * k] = chunk[k];
        __syncwarp();
        float v[kRank / 32];
#pragma unroll
        for (int k = 0; k < kRank / 32; k++) {
            v[k] = Elem<T>::to_f32(x[lane + 32 * k]);
            sq[lane + 32 * k] = __fmul_rn(v[k], v[k]);
        }
        {
            const float x0 = Elem<T>::to_f32(x[kRank + lane]), x1 = Elem<T>::to_f32(x[kRank + 32 + lane]);
            x[kRank + lane]      = Elem<T>::from_f32(__fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn)));
            x[kRank + 32 + lane] = Elem<T>::from_f32(__fadd_rn(__fmul_rn(x1, cs), __fmul_rn(x0, sn)));
        }
        __syncwarp();
        float rinv = 0.0f;
        if (lane == 0) {
            float ss = 0.0f;
#pragma unroll 16
            for (int i = 0; i < kRank; i += 4) {
                const float4 s4 = *reinterpret_cast<const float4*>(sq + i);
                ss = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(ss, s4.x), s4.y), s4.z), s4.w);
            }
            rinv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, float(kRank)), a.eps)));
        }
        rinv = __shfl_sync(0xffffffffu, rinv, 0);
#pragma unroll
        for (int k = 0; k < kRank / 32; k++) x[lane + 32 * k] = Elem<T>::from_f32(__fmul_rn(__fmul_rn(v[k], rinv), Elem<T>::to_f32(nw[k])));
        __syncwarp();
        uint4* dst = reinterpret_cast<uint4*>(static_cast<T*>(a.pool) + (size_t(layer) * a.pool_slots + slot) * kRow);
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) if (lane + 32 * k < kChunks) dst[lane + 32 * k] = reinterpret_cast<const uint4*>(x)[lane + 32 * k];
    }
};

}  // namespace mla
