// Attention of one new position per row against its sequence's fp16 cache, for decode steps and short prompt passes.
//
// Bound: HBM (every cached key and value of the row's KV head once), at short contexts the latency of the chain
// row state -> first keys and values -> merge.
//
// A CTA takes one row and one KV head, so grouped query heads share every load; its NW warps (8, 4 or 2: as many as keep
// all pairs resident at once) take alternate blocks of sixteen positions.  Every warp keeps the next da_stages blocks in flight through
// a ring of its own in shared memory (cp.async): a short context is then requested all at once, and its time is one round trip to
// memory instead of one per block (operands loaded a block ahead into registers: 256 GPT-2 rows at contexts 64 to 96: 711 -> 650 us per step).  Both
// products run on mma.sync.m16n8k16:
//   * scores: the query heads are the A operand.  A row of the MMA is a head's fp16 part: rows 0..7 the rounded queries,
//     rows 8..15 the rounding remainders (22 bits together), whose results land in the same thread and are added there.  Keys
//     are the B operand; a lane's 16-byte piece of a key row supplies two MMA steps once the query's dimensions are taken in
//     the same order.
//   * context: the probabilities, again split into two fp16 parts, are the A operand (the accumulator layout of the scores
//     is the operand layout), values the B operand: a lane loads the same run of dimensions of four positions and interleaves
//     them with byte permutes; output dimension n * (HD / 8) + j is column n of tile j.
// Softmax is online, in fp32 (decodeContext, Sources/RealModelInference/RealModelInferenceEngine.swift:6560-6640).
// Long contexts with few (row, KV head) pairs: up to eight CTAs of a cluster share a pair; they meet in the first one's shared
// memory, and only when the context really reaches past the first CTA's positions.
#pragma once
#include "prefill_attention.cuh"
#include "stream_gemm.cuh"

namespace esp {

constexpr int kDaBlock = 16;  // positions of one warp step
constexpr int kDaHeads = 8;                     // query heads of one CTA (an MMA's rows, twice)

struct DecodeAttArgs {
    ModelDims m;
    RowState rs;
    KvLayout kv;
    const float* q;    // [rows][q_dim] fp32, RoPE applied
    uint16_t* ctx16;   // operand rows of the output projection, 16-bit parts as in stream_gemm.cuh
    int bf16;
    int parts;
    int layer;
    float* debug;      // optional fp32 capture of row 0's context (already offset), or null
    L2Ahead ahead;
};

// Blocks in flight per warp.  Eight warps share a pair only where pairs are few: they (and the cluster) cover 128 to 1024 positions at
// once, and more shared memory would keep the next product's CTAs off the SM (5 rows of the 22-layer model: 713 us per step with
// one block, 716 with two, 750 with three).
__host__ __device__ constexpr int da_stages(int HD, int nw) { return nw == 8 ? 1 : HD == 128 ? 2 : 3; }
__host__ __device__ constexpr int da_ring_floats(int HD, int nw) { return da_stages(HD, nw) * kDaBlock * HD; }  // of one warp: keys and values, fp16
__host__ __device__ constexpr int da_smem_floats(int HD, int nw, int ranks) { return nw * (da_ring_floats(HD, nw) + kDaHeads * 2) + (ranks > 1 ? ranks * kDaHeads * (HD + 4) : 0); }

// Where 16-byte chunk c of row r of a 16-row tile lies (in bytes), so that the lanes of an operand load meet in different banks.
template <int HD>
__device__ __forceinline__ int da_key_at(int r, int c) { return r * (HD * 2) + ((HD == 32 ? c : c ^ ((r & 1) << 2)) << 4); }
template <int HD>
__device__ __forceinline__ int da_value_at(int r, int c) {
    return r * (HD * 2) + ((HD == 32 ? c : HD == 64 ? c ^ (r & 7) : c ^ (((r >> 1) & 1) | (((r >> 2) & 1) << 2))) << 4);
}

// grid = (KV heads x head groups, rows, cluster size); cluster = (1, 1, cluster size)
template <int HD, int NW>
__global__ void __launch_bounds__(NW * 32, (HD == 128 ? 8 : 16) / NW) k_attention_decode(const DecodeAttArgs p) {
    constexpr int kRound = NW * kDaBlock;  // positions of one CTA step
    constexpr int KB = HD / 32;   // 32-dimension blocks of a key row
    constexpr int NT = HD / 8;    // output tiles = dimensions per lane of a value row
    constexpr int kVw = NT / 2;   // 32-bit words of them
    constexpr int kStages = da_stages(HD, NW), kTileBytes = kDaBlock * HD * 2, kRingFloats = da_ring_floats(HD, NW);
    static_assert(kRingFloats >= kDaHeads * HD, "a warp parks its contexts in its ring");
    extern __shared__ __align__(128) float da_smem[];
    float* const s_o = da_smem;                                  // [warp]: the ring, then [head][HD]
    float* const s_ml = s_o + NW * kRingFloats;                  // [warp][head][max, sum]
    float* const s_rank = s_ml + NW * kDaHeads * 2;              // rank 0 of a cluster: [rank][head][HD + 2]
    const ModelDims& m = p.m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int qpk = m.n_head / m.n_kv_head, groups = (qpk + kDaHeads - 1) / kDaHeads;
    const int kvh = (int)blockIdx.x / groups, h0 = ((int)blockIdx.x - kvh * groups) * kDaHeads;
    const int nh = min(kDaHeads, qpk - h0), head0 = kvh * qpk + h0;
    const int row = (int)blockIdx.y, rank = (int)blockIdx.z, ranks = (int)gridDim.z;
    pdl_launch_dependents();
    if (warp == 0) l2_request(p.ahead, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x, gridDim.x * gridDim.y * gridDim.z, lane);
    pdl_wait();
    const int active = __ldcg(p.rs.active + row), pos = __ldcg(p.rs.pos + row), seq = __ldcg(p.rs.seq + row);
    float4 qv[KB][2];
#pragma unroll
    for (int kb = 0; kb < KB; kb++) {
        qv[kb][0] = qv[kb][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g < nh) {
            const float4* src = reinterpret_cast<const float4*>(p.q + (size_t)row * m.q_dim + (size_t)(head0 + g) * HD + kb * 32 + t * 8);
            qv[kb][0] = __ldcg(src);
            qv[kb][1] = __ldcg(src + 1);
        }
    }
    if (!active) return;  // (the same for every CTA of a cluster)
    const int visible = pos + 1;
    const int used = min(ranks, (visible + kRound - 1) / kRound);  // CTAs that have positions
    if (used == 1 && rank > 0) return;                                   // nothing to share: no barrier below
    if (used > 1) cluster_arrive();  // every CTA of the cluster has started: waited for before the first remote store
    const __half* K = p.kv.k + p.kv.offset(m, p.layer, seq, kvh, 0);
    const __half* V = p.kv.v + p.kv.offset(m, p.layer, seq, kvh, 0);

    // Positions base .. base + 15 into ring stage st; those past the context read as zeros.  (Coherent copies: the product before
    // this kernel appends to the cache while the kernel is already resident.)
    uint8_t* const ring = reinterpret_cast<uint8_t*>(s_o + warp * kRingFloats);
    const uint32_t ring_at = smem_u32(ring);
    auto request = [&](int base, int st) {
        if (base < visible) {
            constexpr int kChunks = HD / 8;
            const uint32_t at = ring_at + (uint32_t)(st * 2 * kTileBytes);
#pragma unroll
            for (int i = 0; i < kDaBlock * kChunks / 32; i++) {
                const int r = (lane + 32 * i) / kChunks, c = (lane + 32 * i) % kChunks, key = base + r;
                const size_t src = (size_t)min(key, visible - 1) * HD + c * 8;
                const int bytes = key < visible ? 16 : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + da_key_at<HD>(r, c)), "l"(K + src), "r"(bytes) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + kTileBytes + da_value_at<HD>(r, c)), "l"(V + src), "r"(bytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int step = used * kRound, first = rank < used ? rank * kRound + warp * kDaBlock : visible;
#pragma unroll
    for (int st = 0; st < kStages; st++) request(first + st * step, st);
    // queries, scaled, as (rounded, remainder) fp16 pairs: A registers of the two MMA steps of every 32 dimensions
    uint32_t qa[KB][2][4];
    {
        const float scale = 1.0f / sqrtf((float)HD);
#pragma unroll
        for (int kb = 0; kb < KB; kb++) {
            const float f[8] = {qv[kb][0].x, qv[kb][0].y, qv[kb][0].z, qv[kb][0].w, qv[kb][1].x, qv[kb][1].y, qv[kb][1].z, qv[kb][1].w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float x = f[2 * i] * scale, y = f[2 * i + 1] * scale;
                const uint32_t hi = pf_pack(x, y);
                const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&hi));
                qa[kb][i >> 1][(i & 1) * 2] = hi;
                qa[kb][i >> 1][(i & 1) * 2 + 1] = pf_pack(x - r.x, y - r.y);
            }
        }
    }
    float o[NT][4], mx = -INFINITY, sum = 0.f;  // head g: o[j][0] + o[j][2] is dimension 2t * NT + j, o[j][1] + o[j][3] (2t + 1) * NT + j
#pragma unroll
    for (int j = 0; j < NT; j++) { o[j][0] = 0.f; o[j][1] = 0.f; o[j][2] = 0.f; o[j][3] = 0.f; }
    int st = 0;
#pragma unroll 1
    for (int base = first; base < visible; base += step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        __syncwarp();
        const uint8_t* const tile = ring + st * 2 * kTileBytes;
        uint4 kr[2][KB];  // keys base + g and base + g + 8: this lane's 16-byte piece of every 32 dimensions
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int kb = 0; kb < KB; kb++) kr[i][kb] = *reinterpret_cast<const uint4*>(tile + da_key_at<HD>(8 * i + g, kb * 4 + t));
        uint32_t vr[4][kVw];  // values of positions base + 2t, 2t + 1, 2t + 8, 2t + 9: dimensions g * NT .. g * NT + NT - 1
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = 2 * t + (i & 1) + 8 * (i >> 1);
            if constexpr (kVw == 2) {
                const uint2 x = *reinterpret_cast<const uint2*>(tile + kTileBytes + da_value_at<HD>(r, g >> 1) + (g & 1) * 8);
                vr[i][0] = x.x; vr[i][1] = x.y;
            } else {
#pragma unroll
                for (int w = 0; w < kVw; w += 4) {
                    const uint4 x = *reinterpret_cast<const uint4*>(tile + kTileBytes + da_value_at<HD>(r, g * (NT / 8) + w / 4));
                    vr[i][w] = x.x; vr[i][w + 1] = x.y; vr[i][w + 2] = x.z; vr[i][w + 3] = x.w;
                }
            }
        }
        __syncwarp();
        request(base + kStages * step, st);
        st = st + 1 == kStages ? 0 : st + 1;
        float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kb = 0; kb < KB; kb++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                pf_mma(sc[i], qa[kb][0][0], qa[kb][0][1], qa[kb][0][2], qa[kb][0][3], kr[i][kb].x, kr[i][kb].y);
                pf_mma(sc[i], qa[kb][1][0], qa[kb][1][1], qa[kb][1][2], qa[kb][1][3], kr[i][kb].z, kr[i][kb].w);
            }
        float s[2][2], top = -INFINITY;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                s[i][e] = base + 8 * i + 2 * t + e < visible ? sc[i][e] + sc[i][e + 2] : -INFINITY;
                top = fmaxf(top, s[i][e]);
            }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float mn = fmaxf(mx, top);  // finite: position `base` is visible
        const float corr = expf(mx - mn);
        mx = mn;
        uint32_t pa[4];
        float add = 0.f;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float p0 = expf(s[i][0] - mn), p1 = expf(s[i][1] - mn);
            add += p0 + p1;
            const uint32_t hi = pf_pack(p0, p1);
            const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&hi));
            pa[2 * i] = hi;
            pa[2 * i + 1] = pf_pack(p0 - r.x, p1 - r.y);
        }
        sum = fmaf(sum, corr, add);
#pragma unroll
        for (int j = 0; j < NT; j++) { o[j][0] *= corr; o[j][1] *= corr; o[j][2] *= corr; o[j][3] *= corr; }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
            pf_mma(o[j], pa[0], pa[1], pa[2], pa[3], __byte_perm(vr[0][j >> 1], vr[1][j >> 1], sel), __byte_perm(vr[2][j >> 1], vr[3][j >> 1], sel));
        }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    // ---- merge the warps: every warp parks (max, sum, context) of its heads (the copies still pending are empty)
    __syncwarp();
    if (g < nh) {
        float* dst = s_o + warp * kRingFloats + g * HD + 2 * t * NT;
#pragma unroll
        for (int j = 0; j < NT; j++) { dst[j] = o[j][0] + o[j][2]; dst[NT + j] = o[j][1] + o[j][3]; }
        if (t == 0) { s_ml[(warp * kDaHeads + g) * 2] = mx; s_ml[(warp * kDaHeads + g) * 2 + 1] = sum; }
    }
    __syncthreads();
    if (used > 1) cluster_wait();
    constexpr int kQuads = HD / 4;  // four dimensions of one head per thread
    auto merge = [&](const float* ml, int ml_stride, const float* ctx, int ctx_stride, int n, float& gm, float& total) {
        gm = -INFINITY;
        for (int w = 0; w < n; w++) gm = fmaxf(gm, ml[w * ml_stride]);
        total = 0.f;
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int w = 0; w < n; w++) {
            const float f = ml[w * ml_stride] == -INFINITY ? 0.f : expf(ml[w * ml_stride] - gm);
            const float4 x = *reinterpret_cast<const float4*>(ctx + w * ctx_stride);
            total = fmaf(ml[w * ml_stride + 1], f, total);
            c.x = fmaf(x.x, f, c.x); c.y = fmaf(x.y, f, c.y); c.z = fmaf(x.z, f, c.z); c.w = fmaf(x.w, f, c.w);
        }
        return c;
    };
    constexpr int kStride = HD + 4;  // exchange: per (rank, head) context, max, sum
    auto store = [&](int h, int d, float4 c, float total) {
        const float inv = total > 0.f ? 1.0f / total : 0.f;
        c.x *= inv; c.y *= inv; c.z *= inv; c.w *= inv;
        store_parts4(p.ctx16, m.q_dim, row, (head0 + h) * HD + d, c, p.parts, p.bf16);
        if (p.debug && row == 0) *reinterpret_cast<float4*>(p.debug + (head0 + h) * HD + d) = c;
    };
#pragma unroll 1
    for (int i = threadIdx.x; i < nh * kQuads; i += NW * 32) {
        const int h = i / kQuads, d = (i - h * kQuads) * 4;
        float gm, total;
        const float4 c = merge(s_ml + h * 2, kDaHeads * 2, s_o + h * HD + d, kRingFloats, NW, gm, total);
        if (used == 1) {
            store(h, d, c, total);
        } else if (rank < used) {
            float* const at = s_rank + (rank * kDaHeads + h) * kStride;
            const uint32_t dst = mapa(smem_u32(at + d), 0);
            st_cluster(dst, c.x); st_cluster(dst + 4, c.y); st_cluster(dst + 8, c.z); st_cluster(dst + 12, c.w);
            if (d == 0) { st_cluster(mapa(smem_u32(at + HD), 0), gm); st_cluster(mapa(smem_u32(at + HD + 1), 0), total); }
        }
    }
    if (used == 1) return;
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (rank > 0) return;
#pragma unroll 1
    for (int i = threadIdx.x; i < nh * kQuads; i += NW * 32) {
        const int h = i / kQuads, d = (i - h * kQuads) * 4;
        float gm, total;
        const float4 c = merge(s_rank + h * kStride + HD, kDaHeads * kStride, s_rank + h * kStride + d, kDaHeads * kStride, used, gm, total);
        store(h, d, c, total);
    }
}

}  // namespace esp
