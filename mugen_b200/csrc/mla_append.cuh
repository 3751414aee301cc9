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

constexpr int kAppendRowSmem = kRank * 4;      // the row's squares: 2,048 bytes of shared memory per row (16-byte aligned)

// One new cache row by one warp, in two steps.  `prepare` reads what the step's metadata and the constant tables hold (slot,
// position, cos / sin, norm weights) and may run ahead of the grid dependency wait; `run` needs kv_a.  Left where they are
// used these loads form a chain of dependent round trips to memory (~1 us each) in a kernel whose whole budget is a few
// microseconds.  The row stays in registers, 16-byte pieces lane + 32 * k of it (pieces 64..71 are the rope dims, in lanes 0..7; the
// pairs (i, i + 32) meet by a shuffle): only its squares go through shared memory, to the lane that adds them.
// What bounds it is that sum, a chain of 512 dependent additions: 1.1 us, 1.3 to 2.5 measured.  (The whole row through shared memory in
// 16-bit values, then its squares, a value at a time, and the sum without the loads ahead of it: 4.1 us for the sum, 5.5 in all; 27
// blocks over a 777-token prompt 1806 -> 1725 us.)
template <typename T>
struct AppendRow {
    bool live = false;
    uint64_t slot = 0;
    uint32_t layer = 0, row = 0;
    uint4 nw[2];                       // norm weights of this lane's two pieces of c_kv
    float4 cs[2], sn[2];               // lanes 0..7: cos / sin of pairs 8 * (lane % 4) .. + 7

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
        const float4* tb = reinterpret_cast<const float4*>(a.cos_sin + size_t(pos) * kRope) + 2 * (lane % 4);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (lane < 8) { cs[k] = tb[k]; sn[k] = tb[8 + k]; }
            nw[k] = reinterpret_cast<const uint4*>(static_cast<const T*>(a.norm_w) + size_t(layer) * kRank)[lane + 32 * k];
        }
    }

    __device__ __forceinline__ void run(const AppendArgs& a, unsigned char* smem) const {
        if (!live) return;
        const uint32_t lane = threadIdx.x % 32;
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const T*>(a.kv_a) + (size_t(layer) * a.rows + row) * kRow);
        uint4* dst = reinterpret_cast<uint4*>(static_cast<T*>(a.pool) + (size_t(layer) * a.pool_slots + slot) * kRow);
        uint4 x[2], rope = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 2; k++) x[k] = src[lane + 32 * k];
        if (lane < 8) rope = src[64 + lane];
        __syncwarp();                                  // the row before has been summed
        float4* sq = reinterpret_cast<float4*>(smem);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const T* e = reinterpret_cast<const T*>(&x[k]);
            float s[8];
#pragma unroll
            for (int j = 0; j < 8; j++) { const float f = Elem<T>::to_f32(e[j]); s[j] = __fmul_rn(f, f); }
            sq[2 * (lane + 32 * k)] = make_float4(s[0], s[1], s[2], s[3]);
            sq[2 * (lane + 32 * k) + 1] = make_float4(s[4], s[5], s[6], s[7]);
        }
        __syncwarp();
        float rinv = 0.0f;
        if (lane == 0) {
            // the next eight pieces are on their way while these are added: the additions alone make the chain
            constexpr int AHEAD = 8;
            float ss = 0.0f;
            float4 now[AHEAD], next[AHEAD];
#pragma unroll
            for (int j = 0; j < AHEAD; j++) now[j] = sq[j];
#pragma unroll 2
            for (int i = 0; i < kRank / 4; i += AHEAD) {
#pragma unroll
                for (int j = 0; j < AHEAD; j++) next[j] = sq[(i + AHEAD + j) % (kRank / 4)];
#pragma unroll
                for (int j = 0; j < AHEAD; j++) {
                    ss = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(ss, now[j].x), now[j].y), now[j].z), now[j].w);
                    now[j] = next[j];
                }
            }
            rinv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, float(kRank)), a.eps)));
        }
        {   // NeoX pairs (i, i + 32): piece 64 + j holds x0 of pairs 8 j .., piece 68 + j their x1
            uint32_t mine[4] = {rope.x, rope.y, rope.z, rope.w}, other[4], y[4];
#pragma unroll
            for (int j = 0; j < 4; j++) other[j] = __shfl_xor_sync(0xffffffffu, mine[j], 4);
            if (lane < 8) {
                const float c[8] = {cs[0].x, cs[0].y, cs[0].z, cs[0].w, cs[1].x, cs[1].y, cs[1].z, cs[1].w};
                const float s[8] = {sn[0].x, sn[0].y, sn[0].z, sn[0].w, sn[1].x, sn[1].y, sn[1].z, sn[1].w};
                const T *em = reinterpret_cast<const T*>(mine), *eo = reinterpret_cast<const T*>(other);
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float fm = Elem<T>::to_f32(em[j]), fo = Elem<T>::to_f32(eo[j]);
                    v[j] = lane < 4 ? __fsub_rn(__fmul_rn(fm, c[j]), __fmul_rn(fo, s[j])) : __fadd_rn(__fmul_rn(fm, c[j]), __fmul_rn(fo, s[j]));
                }
#pragma unroll
                for (int j = 0; j < 4; j++) y[j] = Elem<T>::pack2(v[2 * j], v[2 * j + 1]);
                dst[64 + lane] = make_uint4(y[0], y[1], y[2], y[3]);
            }
        }
        rinv = __shfl_sync(0xffffffffu, rinv, 0);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const T *e = reinterpret_cast<const T*>(&x[k]), *w = reinterpret_cast<const T*>(&nw[k]);
            uint32_t y[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                y[j] = Elem<T>::pack2(__fmul_rn(__fmul_rn(Elem<T>::to_f32(e[2 * j]), rinv), Elem<T>::to_f32(w[2 * j])),
                                      __fmul_rn(__fmul_rn(Elem<T>::to_f32(e[2 * j + 1]), rinv), Elem<T>::to_f32(w[2 * j + 1])));
            dst[lane + 32 * k] = make_uint4(y[0], y[1], y[2], y[3]);
        }
    }
};

}  // namespace mla
