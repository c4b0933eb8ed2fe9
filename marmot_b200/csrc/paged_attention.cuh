// Attention over a paged KV pool: parameters and the tensor-core pieces that its kernels share (decoder.cu, attention.cu).
#pragma once

#include "common.cuh"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace mcu {

struct PagedParams {
    const uint32_t *meta;   // [T][4]: seq_slot, pos, kv_slot, flags
    const uint32_t *table;  // [seqs][max_blocks]
    const float *q, *k_new, *v_new;
    void *kv_k, *kv_v;      // [blocks][layers][kv_heads][block_size][head_dim]
    float *out;
    int n_q_heads, n_kv_heads, max_blocks, n_layers, layer, block_shift;
    float scale;
    int n_tokens;
    int *odd_v;  // prompts: set by the append when a V value of the call is not finite, cleared by the merge
};

constexpr int PM_WARPS = 4;
constexpr int PM_TILE = 32;
constexpr int PM_CHUNK = PM_WARPS * PM_TILE;

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
// D += A B, all sixteen rows of A: rows 0..7 carry the f16 heads of the eight query heads' values, rows 8..15 their
// f16 tails, so one instruction yields both partial products (c[0..1] = head row g, c[2..3] = tail row g).
__device__ __forceinline__ void mma_hi_lo(float (&c)[4], uint32_t a_hi0, uint32_t a_lo0, uint32_t a_hi1, uint32_t a_lo1, uint32_t b0,
                                          uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a_hi0), "r"(a_lo0), "r"(a_hi1), "r"(a_lo1), "r"(b0), "r"(b1));
}
// (x, y) as an f16 pair plus the f16 pair of what that rounding lost.
__device__ __forceinline__ void split_half2(float x, float y, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 t = __floats2half2_rn(x - f.x, y - f.y);
    hi = *(const uint32_t *)&h;
    lo = *(const uint32_t *)&t;
}

struct FusedDecode {
    const float2 *rope;  // [T][HD / 2] {cos, sin} of position * frequency, from rope_table_kernel
    int *tickets;        // [T][kv_heads], zero between launches; null: the chunk states are merged by a kernel of its own
    int neox;
};

// One warp per (token, KV head, chunk), tiles by TMA (attention.cu): decode steps, RoPE and KV append included, and tokens whose K and
// V rows are in the pool already.  Both leave chunk states for paged_attention_merge_kernel, except for tokens with a single
// chunk, whose results they write.
bool attention_decode_supported(int n_tokens, int head_dim);
cudaError_t launch_attention_decode(const PagedParams &p, int n_chunks, float *partial, const FusedDecode &fd, int *err,
                                    cudaStream_t s);
cudaError_t launch_attention_prompt(const PagedParams &p, int head_dim, int n_chunks, float *partial, int *err, cudaStream_t s);

}  // namespace mcu
