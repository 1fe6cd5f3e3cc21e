// Element-wise stages beside the products of many rows (stream_gemm.cuh, pair_gemm.cuh):
//   k_prep_rows    RMSNorm / LayerNorm / none -> fp16 or bf16 operand rows, in one or more 16-bit parts
//   k_rope_append  per-head q/k norm, half-split RoPE on q (in place) and k, KV-cache append of k and v: models whose q/k/v
//                  product cannot do this in its epilogue
//   k_head_done    turns the packed per-row maxima of the LM-head GEMM into tokens (head_finalize)
// Every kernel here is launched with programmatic stream serialization: it lets its successor start early and
// waits for its predecessor before it touches global memory.
// Reference arithmetic: see decode_kernels.cuh.
#pragma once
#include "decode_kernels.cuh"

namespace esp {

__device__ __forceinline__ uint16_t to_16bit(float v, int bf16) {
    return bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

// 16-bit parts of two values: the rounded values packed into one word (fp16 parts saturate); x and y keep the remainders.
__device__ __forceinline__ uint32_t part16x2(float& x, float& y, bool bf16) {
    uint32_t d;
    if (bf16) {
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(y), "f"(x));
        x -= __uint_as_float(d << 16);
        y -= __uint_as_float(d & 0xffff0000u);
    } else {
        asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(y), "f"(x));
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&d));
        x -= f.x;
        y -= f.y;
    }
    return d;
}
// Four values of row r -> their parts at columns k..k+3 of operand rows r, r + 8, r + 16.
__device__ __forceinline__ void store_parts4(uint16_t* buf, int ld, int r, int k, float4 v, int parts, bool bf16) {
    uint16_t* dst = buf + (size_t)r * ld + k;
#pragma unroll 1
    for (int j = 0; j < parts; j++) {
        const uint32_t lo = part16x2(v.x, v.y, bf16), hi = part16x2(v.z, v.w, bf16);
        *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
        dst += (size_t)8 * ld;
    }
}

// Row of the rotation table (max_seq rows) for a batch row at position `pos`.  A sequence that has filled its context stays in
// the batch as an inactive row at pos = max_seq; the products read a row's rotation before they know whether it is active.
__host__ __device__ __forceinline__ int rope_row(int pos, int max_seq) { return pos < max_seq ? pos : max_seq - 1; }

struct PrepArgs {
    const int* active;
    const float* src;  // [rows][K] fp32
    int K;             // a multiple of 4
    int norm;          // NormKind
    float eps;
    const float* g;
    const float* b;
    uint16_t* dst;     // [rows][K] fp16/bf16
    int bf16;
    int parts;         // 16-bit parts per value (see stream_gemm.cuh): part j of row r goes to row r + 8 j
};

// One CTA per row, the row in registers: VEC float4 per thread (VEC = 0: rows of more than 8192 elements, re-read for every
// pass).  Bound by latency at few rows: one load round trip, one or two block reductions, one store; the code is kept short
// because instruction fetch is a visible part of a launch this small.
template <int VEC>
__global__ void __launch_bounds__(kThreads) k_prep_rows(const PrepArgs p) {
    __shared__ float red[kRedFloats];
    constexpr int N = VEC ? VEC : 1;
    const int r = blockIdx.x, K = p.K, nvec = K >> 2;
    float4 g[N], b[N];
    if (VEC && p.norm != NORM_NONE) {  // gains do not depend on the previous kernel
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int idx = threadIdx.x + i * kThreads;
            g[i] = b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < nvec) {
                g[i] = __ldg(reinterpret_cast<const float4*>(p.g) + idx);
                if (p.norm == NORM_LAYER) b[i] = __ldg(reinterpret_cast<const float4*>(p.b) + idx);
            }
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    const int active = __ldcg(p.active + r);
    const float4* src = reinterpret_cast<const float4*>(p.src + (size_t)r * K);
    if constexpr (VEC > 0) {
        float4 v[N];  // requested together with the row's state
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int idx = threadIdx.x + i * kThreads;
            v[i] = idx < nvec ? __ldcg(src + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (!active) return;
        float inv = 1.f, mean = 0.f;
        if (p.norm == NORM_LAYER) {
            float sm = 0.f;
#pragma unroll
            for (int i = 0; i < N; i++) sm += (v[i].x + v[i].y) + (v[i].z + v[i].w);
            mean = block_sum(sm, red) / (float)K;
        }
        if (p.norm != NORM_NONE) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < N; i++) {
                if (threadIdx.x + i * kThreads >= nvec) continue;
                v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
                ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
            }
            ss = block_sum(ss, red);
            inv = 1.0f / sqrtf(ss / (float)K + p.eps);
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int idx = threadIdx.x + i * kThreads;
            if (idx >= nvec) continue;
            if (p.norm != NORM_NONE)
                v[i] = make_float4(fmaf(v[i].x * inv, g[i].x, b[i].x), fmaf(v[i].y * inv, g[i].y, b[i].y), fmaf(v[i].z * inv, g[i].z, b[i].z), fmaf(v[i].w * inv, g[i].w, b[i].w));
            store_parts4(p.dst, K, r, 4 * idx, v[i], p.parts, p.bf16);
        }
    } else {
        if (!active) return;
        float inv = 1.f, mean = 0.f;
        if (p.norm == NORM_LAYER) {
            float sm = 0.f;
#pragma unroll 1
            for (int k = threadIdx.x; k < nvec; k += kThreads) { const float4 v = __ldcg(src + k); sm += (v.x + v.y) + (v.z + v.w); }
            mean = block_sum(sm, red) / (float)K;
        }
        if (p.norm != NORM_NONE) {
            float ss = 0.f;
#pragma unroll 1
            for (int k = threadIdx.x; k < nvec; k += kThreads) {
                const float4 v = __ldcg(src + k);
                const float x = v.x - mean, y = v.y - mean, z = v.z - mean, w = v.w - mean;
                ss = fmaf(x, x, fmaf(y, y, fmaf(z, z, fmaf(w, w, ss))));
            }
            ss = block_sum(ss, red);
            inv = 1.0f / sqrtf(ss / (float)K + p.eps);
        }
#pragma unroll 1
        for (int k = threadIdx.x; k < nvec; k += kThreads) {
            float4 v = __ldcg(src + k);
            if (p.norm != NORM_NONE) {
                const float4 gg = __ldg(reinterpret_cast<const float4*>(p.g) + k);
                const float4 bb = p.norm == NORM_LAYER ? __ldg(reinterpret_cast<const float4*>(p.b) + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                v = make_float4(fmaf((v.x - mean) * inv, gg.x, bb.x), fmaf((v.y - mean) * inv, gg.y, bb.y), fmaf((v.z - mean) * inv, gg.z, bb.z), fmaf((v.w - mean) * inv, gg.w, bb.w));
            }
            store_parts4(p.dst, K, r, 4 * k, v, p.parts, p.bf16);
        }
    }
}

struct RopeArgs {
    ModelDims m;
    RowState rs;
    KvLayout kv;
    float* q;            // [rows][q_dim], rotated in place
    const float* k_raw;  // [rows][kv_dim]
    const float* v_raw;  // [rows][kv_dim]
    const float2* rope;  // [max_seq][head_dim/2] (cos, sin); null for GPT-2
    int layer;
    float* debug;        // optional capture of row 0 (q, k, v as stored)
    const float* q_norm; // [head_dim] per-head RMSNorm weights applied to q and k before RoPE (Qwen3), or null
    const float* k_norm;
};

// grid = (rows, chunks): one thread per rotation pair of q, per rotation pair of k, or per pair of v elements.
// The head_dim / 2 threads of a head are neighbours inside one CTA (256 is a multiple of 16, 32 and 64), which is what
// the optional per-head norm (applyPerHeadRMSNormInPlace, Sources/RealModelInference/RealModelInferenceEngine.swift:
// 6648-6672: v * rsqrt(mean(v^2) + eps) * w, before RoPE) uses for its sum of squares.
__global__ void __launch_bounds__(kThreads) k_rope_append(const RopeArgs p) {
    __shared__ float head_ss[kThreads / 32];
    const int r = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const int row_active = p.rs.active[r], pos = p.rs.pos[r], seq = p.rs.seq[r];  // one round trip for the three
    if (!row_active) return;
    const ModelDims& m = p.m;
    const int half = m.head_dim / 2;
    const int q_pairs = m.q_dim / 2, k_pairs = m.kv_dim / 2;
    const int i = blockIdx.y * kThreads + threadIdx.x;
    const bool rot = i < q_pairs + k_pairs;
    const bool is_q = i < q_pairs;
    const int local = is_q ? i : i - q_pairs;
    const int head = rot ? local / half : 0, idx = rot ? local - head * half : 0;
    const int i0 = head * m.head_dim + idx, i1 = i0 + half;
    float* q = p.q + (size_t)r * m.q_dim;
    const float* kr = p.k_raw + (size_t)r * m.kv_dim;
    float v0 = 0.f, v1 = 0.f;
    if (rot) { v0 = is_q ? q[i0] : kr[i0]; v1 = is_q ? q[i1] : kr[i1]; }
    if (p.q_norm) {  // uniform over the grid: every thread of the CTA takes part in the barrier
        float ss = v0 * v0 + v1 * v1;
        for (int o = (half < 32 ? half : 32) >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (half == 64) {  // a head spans two warps
            if ((threadIdx.x & 31) == 0) head_ss[threadIdx.x >> 5] = ss;
            __syncthreads();
            ss = head_ss[(threadIdx.x >> 5) & ~1] + head_ss[(threadIdx.x >> 5) | 1];
        }
        if (rot) {
            const float inv = 1.0f / sqrtf(ss / (float)m.head_dim + m.eps);
            const float* w = is_q ? p.q_norm : p.k_norm;
            v0 *= inv * w[idx];
            v1 *= inv * w[idx + half];
        }
    }
    if (i >= q_pairs + 2 * k_pairs) return;
    if (rot) {
        if (p.rope) {
            const float2 cs = p.rope[(size_t)pos * half + idx];
            const float r0 = v0 * cs.x - v1 * cs.y, r1 = v0 * cs.y + v1 * cs.x;
            v0 = r0; v1 = r1;
        }
        if (is_q) {
            q[i0] = v0; q[i1] = v1;
            if (p.debug && r == 0) { p.debug[i0] = v0; p.debug[i1] = v1; }
        } else {
            const size_t off = p.kv.offset(m, p.layer, seq, head, pos);
            p.kv.k[off + idx] = __float2half_rn(v0);
            p.kv.k[off + idx + half] = __float2half_rn(v1);
            if (p.debug && r == 0) {
                p.debug[m.q_dim + i0] = __half2float(__float2half_rn(v0));
                p.debug[m.q_dim + i1] = __half2float(__float2half_rn(v1));
            }
        }
    } else {
        const int e = 2 * (i - q_pairs - k_pairs);  // head_dim is even: both elements belong to one head
        const int head = e / m.head_dim, idx = e - head * m.head_dim;
        const float2 vv = *reinterpret_cast<const float2*>(p.v_raw + (size_t)r * m.kv_dim + e);
        const __half2 hv = __floats2half2_rn(vv.x, vv.y);
        *reinterpret_cast<__half2*>(p.kv.v + p.kv.offset(m, p.layer, seq, head, pos) + idx) = hv;
        if (p.debug && r == 0) {
            p.debug[m.q_dim + m.kv_dim + e] = __low2float(hv);
            p.debug[m.q_dim + m.kv_dim + e + 1] = __high2float(hv);
        }
    }
}

__global__ void k_head_done(const GemvArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    head_finalize(p.m, p.rows, p.rs, p.finalize_mode);
}

__global__ void k_copy_debug(const float* src, float* dst, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
}

}  // namespace esp
