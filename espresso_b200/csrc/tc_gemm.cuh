// tcgen05 / TMA building blocks of the products (stream_gemm.cuh, pair_gemm.cuh): copies, shared-memory and instruction
// descriptors, bounded barrier waits, MMA issue, and the activations of their epilogues.
#pragma once
#include <cuda.h>

#include "mega_kernel.cuh"  // mbarrier helpers

namespace esp {

constexpr int kTcBlockK = 64;   // 64 x 16-bit = one 128-byte swizzle row
constexpr unsigned kTcSpinLimit = 1u << 22;

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
                 "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 x 16-bit) with the 128-byte
// swizzle: 8-row groups are 1024 bytes apart (stride byte offset), the leading byte offset is unused (1).
__device__ __forceinline__ uint64_t umma_smem_desc_sw128(const void* smem_tile) {
    const uint32_t addr = smem_u32(smem_tile);
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);   // start address, bits [0,14)
    d |= (uint64_t)1 << 16;                    // leading byte offset (ignored for swizzled K-major), bits [16,30)
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset, bits [32,46)
    d |= (uint64_t)1 << 46;                    // descriptor version of this architecture, bits [46,48)
    d |= (uint64_t)2 << 61;                    // layout type: 128-byte swizzle, bits [61,64)
    return d;
}

// Instruction descriptor of tcgen05.mma.kind::f16: fp32 accumulator, fp16 or bf16 operands, both K-major, M = m, N = n.
__device__ __forceinline__ uint32_t umma_idesc_f16(int m, int n, int bf16) {
    uint32_t d = 0;
    d |= 1u << 4;                        // accumulator format: f32
    d |= (uint32_t)(bf16 ? 1 : 0) << 7;  // A format
    d |= (uint32_t)(bf16 ? 1 : 0) << 10; // B format
    d |= (uint32_t)(n >> 3) << 17;       // N / 8
    d |= (uint32_t)(m >> 4) << 24;       // M / 16
    return d;
}

// True in one lane of a converged warp.  The loops that issue TMA copies and MMAs are run by the whole warp and elect a lane
// only around the instructions: the same loop under `if (lane == 0)` took 1041 cycles per 64-wide K block (four MMAs and one
// barrier wait) whatever the MMA's shape, against 509 (N = 256, the tensor pipe's own time) and ~320 (N <= 64) this way.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ bool tc_wait(uint64_t* bar, unsigned parity, int* error) {
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++spins > kTcSpinLimit || ((spins & 0xfffu) == 0 && __ldcg(error) != 0)) {
            atomicCAS(error, 0, 7);
            return false;
        }
    }
    return true;
}

// The same with one answer for a whole warp, for loops whose next instructions are warp-wide (elect, tcgen05.ld, warp barriers):
// lanes that poll on their own can end apart when a wait runs out, and those still in the loop would wait for the others for good.
__device__ __forceinline__ bool tc_wait_warp(uint64_t* bar, unsigned parity, int* error) { return __all_sync(0xffffffffu, tc_wait(bar, parity, error)); }

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Activations of epilogues whose results are rounded to one 16-bit part right away (2^-12 or 2^-9): the hardware
// approximations of exponential and division may stand in for tanhf.  Error against 64 bits over [-3, 3], 2-norm relative:
// silu 4.8e-8 and gelu 5.3e-8, with tanhf (silu_f, gelu_f) 3.8e-8 and 3.6e-8.  Rows of several parts take the latter.
__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
__device__ __forceinline__ float gelu_fast(float x) {
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    const float t = 1.0f - __fdividef(2.0f, 1.0f + __expf(2.0f * u));  // tanh(u)
    return 0.5f * x * (1.0f + t);
}

__device__ __forceinline__ uint32_t pack16x2(float a, float b, int bf16) {
    const uint32_t lo = bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(a)) : __half_as_ushort(__float2half_rn(a));
    const uint32_t hi = bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(b)) : __half_as_ushort(__float2half_rn(b));
    return lo | (hi << 16);
}

}  // namespace esp
