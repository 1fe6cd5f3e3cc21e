// Element-wise stages of the batched (tensor-core) decode path.  The matrix products run in k_gemm_tc; these
// kernels prepare its 16-bit operand rows and apply what the GEMV path fuses into its epilogues:
//   k_prep_rows    (embedding) -> RMSNorm / LayerNorm / none -> fp16 or bf16 operand rows
//   k_rope_append  half-split RoPE on q (in place) and k, KV-cache append of k and v
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

// 16-bit parts of a value: part 0 is the rounded value, the next ones the rounded remainders (fp16 parts saturate).
__device__ __forceinline__ uint16_t part16(float& v, int bf16) {
    if (bf16) {
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        v -= __bfloat162float(h);
        return __bfloat16_as_ushort(h);
    }
    unsigned short h;
    asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
    v -= __half2float(__ushort_as_half(h));
    return h;
}
// Four values of row r -> their parts at columns k..k+3 of operand rows r, r + 8, r + 16.
__device__ __forceinline__ void store_parts4(uint16_t* buf, int ld, int r, int k, float4 v, int parts, int bf16) {
    for (int j = 0; j < parts; j++) {
        const uint32_t lo = part16(v.x, bf16) | ((uint32_t)part16(v.y, bf16) << 16);
        const uint32_t hi = part16(v.z, bf16) | ((uint32_t)part16(v.w, bf16) << 16);
        *reinterpret_cast<uint2*>(buf + (size_t)(r + 8 * j) * ld + k) = make_uint2(lo, hi);
    }
}

struct PrepArgs {
    ModelDims m;
    RowState rs;
    const float* src;         // [rows][K] fp32, or null when from_embedding
    float* hidden_out;        // from_embedding: the residual stream [rows][d_model] is initialised here
    const uint16_t* tok_emb;  // from_embedding
    const uint16_t* pos_emb;
    int emb_type;
    int from_embedding;
    int K;
    int norm;                 // NormKind
    const float* g;
    const float* b;
    uint16_t* dst;            // [rows][K] fp16/bf16
    int bf16;
    int parts;                // 16-bit parts per value (see stream_gemm.cuh): part j of row r goes to row r + 8 j
};

// One CTA per row.  Rows of up to 8192 elements are held in registers (one global read, 16-byte accesses); longer
// rows are re-read for every pass.
__global__ void __launch_bounds__(kThreads) k_prep_rows(const PrepArgs p) {
    __shared__ float red[kRedFloats];
    const int r = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    // The row's state words and (when the row comes from the residual stream) its values are requested together;
    // the check for an inactive row comes after the requests, so the chain is one memory round trip shorter.
    const int row_active = p.rs.active[r];
    const int K = p.K;
    const float* src = p.src ? p.src + (size_t)r * K : nullptr;
    const uint16_t* te = nullptr;
    const uint16_t* pe = nullptr;
    if (p.from_embedding) {
        te = p.tok_emb + (size_t)p.rs.tok[r] * K;
        if (p.pos_emb) pe = p.pos_emb + (size_t)p.rs.pos[r] * K;
    }
    uint16_t* dst = p.dst + (size_t)r * K;
    constexpr int kVec = 8;  // float4 per thread held in registers
    const bool fast = K % 4 == 0 && K / 4 <= kVec * kThreads;
    float4 pre[kVec];
    if (fast && !p.from_embedding) {
#pragma unroll
        for (int i = 0; i < kVec; i++) {
            const int idx = threadIdx.x + i * kThreads;
            pre[i] = idx < K / 4 ? reinterpret_cast<const float4*>(src)[idx] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (!row_active) return;
    if (fast) {
        const int nvec = K / 4;
        float4 v[kVec];
#pragma unroll
        for (int i = 0; i < kVec; i++) {
            const int idx = threadIdx.x + i * kThreads;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < nvec) {
                if (!p.from_embedding) {
                    v[i] = pre[i];
                } else {
                    const uint2 t = reinterpret_cast<const uint2*>(te)[idx];
                    v[i] = make_float4(emb_to_float((uint16_t)(t.x & 0xffffu), p.emb_type), emb_to_float((uint16_t)(t.x >> 16), p.emb_type),
                                       emb_to_float((uint16_t)(t.y & 0xffffu), p.emb_type), emb_to_float((uint16_t)(t.y >> 16), p.emb_type));
                    if (pe) {
                        const uint2 u = reinterpret_cast<const uint2*>(pe)[idx];
                        v[i].x += emb_to_float((uint16_t)(u.x & 0xffffu), p.emb_type);
                        v[i].y += emb_to_float((uint16_t)(u.x >> 16), p.emb_type);
                        v[i].z += emb_to_float((uint16_t)(u.y & 0xffffu), p.emb_type);
                        v[i].w += emb_to_float((uint16_t)(u.y >> 16), p.emb_type);
                    }
                    reinterpret_cast<float4*>(p.hidden_out + (size_t)r * K)[idx] = v[i];
                }
            }
        }
        float inv = 1.f, mean = 0.f;
        if (p.norm == NORM_RMS) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < kVec; i++) ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
            ss = block_sum(ss, red);
            inv = 1.0f / sqrtf(ss / (float)K + p.m.eps);
        } else if (p.norm == NORM_LAYER) {
            float sm = 0.f;
#pragma unroll
            for (int i = 0; i < kVec; i++) sm += (v[i].x + v[i].y) + (v[i].z + v[i].w);
            mean = block_sum(sm, red) / (float)K;
            float vs = 0.f;
#pragma unroll
            for (int i = 0; i < kVec; i++) {
                if (threadIdx.x + i * kThreads < nvec) {
                    const float a = v[i].x - mean, b = v[i].y - mean, c = v[i].z - mean, d = v[i].w - mean;
                    vs = fmaf(a, a, fmaf(b, b, fmaf(c, c, fmaf(d, d, vs))));
                }
            }
            vs = block_sum(vs, red);
            inv = 1.0f / sqrtf(vs / (float)K + p.m.eps);
        }
#pragma unroll
        for (int i = 0; i < kVec; i++) {
            const int idx = threadIdx.x + i * kThreads;
            if (idx >= nvec) continue;
            float4 o = v[i];
            if (p.norm == NORM_RMS) {
                const float4 g = reinterpret_cast<const float4*>(p.g)[idx];
                o = make_float4((o.x * inv) * g.x, (o.y * inv) * g.y, (o.z * inv) * g.z, (o.w * inv) * g.w);
            } else if (p.norm == NORM_LAYER) {
                const float4 g = reinterpret_cast<const float4*>(p.g)[idx];
                const float4 b = reinterpret_cast<const float4*>(p.b)[idx];
                o = make_float4((o.x - mean) * inv * g.x + b.x, (o.y - mean) * inv * g.y + b.y, (o.z - mean) * inv * g.z + b.z,
                                (o.w - mean) * inv * g.w + b.w);
            }
            store_parts4(p.dst, K, r, 4 * idx, o, p.parts, p.bf16);
        }
        return;
    }
    auto raw = [&](int k) {
        if (!p.from_embedding) return src[k];
        float v = emb_to_float(te[k], p.emb_type);
        if (pe) v += emb_to_float(pe[k], p.emb_type);
        return v;
    };
    float inv = 1.f, mean = 0.f;
    if (p.norm == NORM_RMS) {
        float ss = 0.f;
        for (int k = threadIdx.x; k < K; k += kThreads) { const float v = raw(k); ss = fmaf(v, v, ss); }
        ss = block_sum(ss, red);
        inv = 1.0f / sqrtf(ss / (float)K + p.m.eps);
    } else if (p.norm == NORM_LAYER) {
        float s = 0.f;
        for (int k = threadIdx.x; k < K; k += kThreads) s += raw(k);
        mean = block_sum(s, red) / (float)K;
        float vs = 0.f;
        for (int k = threadIdx.x; k < K; k += kThreads) { const float c = raw(k) - mean; vs = fmaf(c, c, vs); }
        vs = block_sum(vs, red);
        inv = 1.0f / sqrtf(vs / (float)K + p.m.eps);
    }
    for (int k = threadIdx.x; k < K; k += kThreads) {
        const float x = raw(k);
        if (p.from_embedding) p.hidden_out[(size_t)r * K + k] = x;
        float v = x;
        if (p.norm == NORM_RMS) v = (x * inv) * p.g[k];
        else if (p.norm == NORM_LAYER) v = (x - mean) * inv * p.g[k] + p.b[k];
        for (int j = 0; j < p.parts; j++) dst[(size_t)8 * j * K + k] = part16(v, p.bf16);
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
