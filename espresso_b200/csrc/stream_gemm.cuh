// Products of few activation rows (up to 704, see step_path.h) with a 16-bit weight matrix, for decode steps and short prompts:
// Y[n][m] = sum_k W[m][k] * X[n][k] on tcgen05/TMEM, with everything the decode path does to a finished row of Y (bias,
// RoPE and cache append, residual, activation, arg-max) in the epilogue.
//
// Bound: HBM (the weights travel once), and below ~30 MB per launch the latency of the chain of dependent kernels.
//
// Mapping.  The weight rows are the MMA's M (128 TMEM lanes), the batch rows its N (16..64 columns).  Measured issue cost
// of tcgen05.mma M128 K16: 45 cycles up to N = 32, 48 at 64, so even the narrowest product moves 4 KB of
// weights per 45 cycles, four times an SM's share of HBM, and a row more costs nothing.  With lanes along the weight rows
// the accumulator leaves TMEM as consecutive output elements per batch row: every store is a contiguous run and no
// transposition is needed.
//
// K slices.  A small matrix has fewer 128-row tiles than the chip has SMs, so K is cut into up to eight slices, one CTA of
// a cluster each.  Every CTA pushes its partial sums of batch row r into the shared memory of CTA r % slices (distributed
// shared memory), and after one cluster barrier each CTA adds up the parts of its own rows.  One CTA thus holds complete
// sums - the epilogues can be non-linear, need no zeroed output, no atomics, and the result does not depend on the order of
// arrival.  (Pulling the parts instead needed a second barrier before anyone could leave: 1.2 us more per launch.)
//
// Few rows (<= 8).  A single sequence must not lose precision to 16-bit activations: every row is split exactly into
// 16-bit parts (two for fp16: 22 bits; three for bf16: 24 bits) that ride in columns r, r + 8 (, r + 16) of the same MMA,
// whose narrowest shape has 16 columns anyway; the epilogue adds the parts' sums.
//
// Operand rows.  Either 16-bit rows in memory (TMA, 128-byte swizzle), or the fp32 residual stream: the stage warps then apply
// RMSNorm / LayerNorm while they stage the operand (the row statistics come from the kernel that wrote the stream, as
// per-128-column (mean, M2) pairs), which saves the norm kernel in front of the product.
//
// Occupancy.  At most ~110 KB of shared memory and 64 TMEM columns per CTA: the next kernel of the stream (programmatic
// dependent launch) fits beside this one and fills its weight ring while this one drains.
#pragma once
#include "batch_kernels.cuh"
#include "tc_gemm.cuh"

namespace esp {

constexpr int kSgThreads = 256;   // warp 1 issues the MMAs, warps 2..7 feed one ring stage each; all eight run the epilogue
constexpr int kSgXWarps = 6;
constexpr int kSgRows = 128;      // weight rows of a tile: two 64-row halves, possibly of different matrices
constexpr int kSgHalf = 64;
constexpr int kSgMaxCols = 64;    // batch columns of one CTA: its ring and exchange buffer fit half an SM's shared memory
constexpr int kSgMaxStages = kSgXWarps;
constexpr int kSgMaxSplits = 8;   // portable cluster size
constexpr int kSgWBytes = kSgRows * kTcBlockK * 2;
constexpr int kSgSmemBudget = 110 * 1024;

// Weights that later kernels of the step will read, brought into L2 while this one waits for its predecessor (Engine::launch_step_stream
// says which): HBM would otherwise idle through the hand-over, the operand staging, the exchange and the attention of every stage.  Each CTA requests its
// share of every range.
constexpr int kL2Ranges = 4;
struct L2Ahead {
    const uint8_t* p[kL2Ranges];
    unsigned bytes[kL2Ranges];  // multiples of 16; 0 ends the list
};
__device__ __forceinline__ void l2_request(const L2Ahead& a, unsigned cta, unsigned n_cta, int lane) {
    constexpr unsigned kPiece = 8192;
#pragma unroll 1
    for (int r = 0; r < kL2Ranges && a.bytes[r]; r++) {
        const unsigned pieces = (a.bytes[r] + kPiece - 1) / kPiece;
#pragma unroll 1
        for (unsigned i = cta + n_cta * (unsigned)lane; i < pieces; i += n_cta * 32u)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.p[r] + (size_t)i * kPiece), "r"(min(kPiece, a.bytes[r] - i * kPiece)) : "memory");
    }
}

enum SgEpilogue { SG_STORE = 0, SG_RESIDUAL = 1, SG_QKV = 2, SG_GELU = 3, SG_SWIGLU = 4, SG_HEAD = 5 };

struct SgGroup {
    int M;              // weight rows of this matrix
    int half0;          // index of its first 64-row half in the launch's list of halves
    float* out;         // SG_STORE / SG_RESIDUAL: [n][ldo] fp32
    int ldo;
    const float* bias;  // [M] or null
};

struct SgArgs {
    SgGroup g[3];
    int n_groups;
    int K, kb_per_split;
    int rows;             // live batch rows
    int n_cols;           // MMA columns per CTA (a multiple of 16)
    int parts;            // 16-bit parts per row: 1, or 2 / 3 for at most 8 rows (column of part j of row r: r + 8 j)
    int stages;
    int epilogue;         // SgEpilogue
    int bf16;
    // operand staged from the fp32 residual stream (hidden != null): norm = NORM_RMS or NORM_LAYER
    const float* hidden;  // [rows][K]
    const float2* stat;   // [rows][stat_tiles] (mean, M2) of every 128 columns
    int stat_tiles;
    int norm;
    const float *norm_g, *norm_b;
    float eps;
    // epilogues
    ModelDims m;
    RowState rs;          // active, pos, seq; SG_HEAD: best, ticket
    int all_rows;         // write rows whose `active` is 0 too (tensor-parallel partial sums)
    KvLayout kv;
    const float2* rope;   // null for GPT-2
    int layer;
    float2* stat_out;     // SG_RESIDUAL: per-128-column statistics of the new residual stream, or null
    uint16_t* out16;      // SG_GELU / SG_SWIGLU: operand rows [parts * 8 or rows][ld16] of the next product
    int ld16;
    float* debug;         // optional capture of batch row 0
    float* logits;        // SG_HEAD: optional [n][M]
    int row_offset;       // SG_HEAD: added to the vocabulary row (shard of a tensor-parallel rank)
    L2Ahead ahead;
    int finalize;         // SG_HEAD: the last CTA turns the packed maxima into tokens with this head_finalize mode; -1 = a later kernel does
    int* error;
};

// Launch shape chosen by the host (sg_plan).
struct SgPlan {
    int n_cols = 16, col_tiles = 1, row_tiles = 1, splits = 1, kb_per_split = 1, stages = 2, parts = 1;
    int smem = 0;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
template <int NC>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[NC]);
template <>
__device__ __forceinline__ void tmem_ld_cols<8>(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// Operand staging from the residual stream.  One warp per 64-column block; lane = (row of a group of four, chunk of eight
// columns), so a row is one 256-byte read.  Gains and the first sixteen rows' values are requested ahead of their use.
struct SgNormPre {
    float4 g[2], b[2];
    float4 v[4][2];
};
__device__ __forceinline__ void sg_norm_gains(const SgArgs& a, SgNormPre& p, int k0, int lane) {
    const int k = k0 + (lane & 7) * 8;
    p.g[0] = __ldg(reinterpret_cast<const float4*>(a.norm_g + k));
    p.g[1] = __ldg(reinterpret_cast<const float4*>(a.norm_g + k) + 1);
    p.b[0] = p.b[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.norm_b) {
        p.b[0] = __ldg(reinterpret_cast<const float4*>(a.norm_b + k));
        p.b[1] = __ldg(reinterpret_cast<const float4*>(a.norm_b + k) + 1);
    }
}
__device__ __forceinline__ void sg_norm_rows(const SgArgs& a, SgNormPre& p, int n0, int r0, int rows, int k0, int lane) {
    const float* src = a.hidden + (size_t)n0 * a.K + k0 + (lane & 7) * 8;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = r0 + u * 4 + (lane >> 3);
        p.v[u][0] = p.v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            const float4* q = reinterpret_cast<const float4*>(src + (size_t)r * a.K);
            p.v[u][0] = __ldcg(q);
            p.v[u][1] = __ldcg(q + 1);
        }
    }
}
// Normalises and stores rows r0 .. r0 + 15 (128-byte rows, 16-byte chunks XOR-swizzled by the row).
template <bool BF16>
__device__ __forceinline__ void sg_norm_store(const SgArgs& a, const SgNormPre& p, uint8_t* sx, const float2* stat, int r0, int rows, int lane) {
    const int c = lane & 7;
    const float g[8] = {p.g[0].x, p.g[0].y, p.g[0].z, p.g[0].w, p.g[1].x, p.g[1].y, p.g[1].z, p.g[1].w};
    const float b[8] = {p.b[0].x, p.b[0].y, p.b[0].z, p.b[0].w, p.b[1].x, p.b[1].y, p.b[1].z, p.b[1].w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (r0 + u * 4 >= rows) break;  // (the whole warp)
        const int r = min(r0 + u * 4 + (lane >> 3), rows - 1);  // rows past the end repeat the last one
        const bool mine = r0 + u * 4 + (lane >> 3) < rows;
        const float2 st = stat[r];  // (mean or 0, 1 / sqrt(variance + eps))
        float y[8] = {p.v[u][0].x, p.v[u][0].y, p.v[u][0].z, p.v[u][0].w, p.v[u][1].x, p.v[u][1].y, p.v[u][1].z, p.v[u][1].w};
#pragma unroll
        for (int i = 0; i < 8; i++) y[i] = (y[i] - st.x) * st.y * g[i] + b[i];
        uint8_t* dst = sx + r * 128 + ((c ^ (r & 7)) << 4);  // (part j: eight rows further down, the same swizzle)
#pragma unroll 1
        for (int j = 0; j < a.parts; j++) {
            const uint4 w = make_uint4(part16x2(y[0], y[1], BF16), part16x2(y[2], y[3], BF16), part16x2(y[4], y[5], BF16), part16x2(y[6], y[7], BF16));
            if (mine) *reinterpret_cast<uint4*>(dst + j * 1024) = w;
        }
    }
}

// (mean, 1 / sqrt(var + eps)) of every row from its per-128-column statistics; RMSNorm: mean 0, mean square.  Eight lanes per
// row, four rows per stage warp, one round trip; the caller synchronises the warps.
__device__ __forceinline__ void sg_row_stats(const SgArgs& a, float2* stat, int n0, int rows, int xw, int lane) {
    const float inv_k = 1.0f / (float)a.K;
    const int l = lane & 7, tiles = a.stat_tiles;
    auto n_of = [&](int t) { return (float)min(kSgRows, a.K - t * kSgRows); };
    auto sum8 = [](float v) {
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        return v + __shfl_xor_sync(0xffffffffu, v, 4);
    };
#pragma unroll 1
    for (int r0 = xw * 4; r0 < rows; r0 += 4 * kSgXWarps) {
        const int r = min(r0 + (lane >> 3), rows - 1);
        const float2* src = a.stat + (size_t)(n0 + r) * tiles;
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = l + 8 * i < tiles ? __ldcg(src + l + 8 * i) : make_float2(0.f, 0.f);
        float mean = 0.f;
        if (a.norm == NORM_LAYER) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (l + 8 * i < tiles) mean = fmaf(v[i].x, n_of(l + 8 * i), mean);
#pragma unroll 1
            for (int t = l + 32; t < tiles; t += 8) mean = fmaf(__ldcg(&src[t].x), n_of(t), mean);
            mean = sum8(mean) * inv_k;
        }
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (l + 8 * i < tiles) ss += fmaf((v[i].x - mean) * (v[i].x - mean), n_of(l + 8 * i), v[i].y);
#pragma unroll 1
        for (int t = l + 32; t < tiles; t += 8) {
            const float2 s = __ldcg(src + t);
            ss += fmaf((s.x - mean) * (s.x - mean), n_of(t), s.y);
        }
        ss = sum8(ss);
        if (l == 0 && r0 + (lane >> 3) < rows) stat[r] = make_float2(mean, rsqrtf(fmaf(ss, inv_k, a.eps)));
    }
}

// Statistics of a 128-column tile of one row held as four values per lane (n valid columns; invalid lanes pass zeros):
// (mean, sum of squared deviations), or (0, sum of squares) where only RMSNorm will read them.
__device__ __forceinline__ float2 tile_stat(float4 v, bool valid, int n, bool rms) {
    const float mean = rms ? 0.f : warp_sum((v.x + v.y) + (v.z + v.w)) / (float)n;
    const float a = v.x - mean, b = v.y - mean, c = v.z - mean, d = v.w - mean;
    const float m2 = warp_sum(valid ? fmaf(a, a, fmaf(b, b, fmaf(c, c, d * d))) : 0.f);
    return make_float2(mean, m2);
}

// What the epilogue of a row reads besides its sums and its control words, requested while the products still run.
struct SgRowPre {
    float4 x0, x1;  // SG_RESIDUAL: the residual; SG_QKV: (cos, sin) of the lane's four rotation pairs
};
__device__ __forceinline__ SgRowPre sg_row_prefetch(const SgArgs& a, int row, int gi, int m0, bool ok) {
    SgRowPre p;
    p.x0 = p.x1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.epilogue == SG_RESIDUAL) {
        if (ok) p.x0 = __ldcg(reinterpret_cast<const float4*>(a.g[0].out + (size_t)row * a.g[0].ldo + m0));
    } else if (a.epilogue == SG_QKV) {
        if (a.rope && gi < 2) {
            const int half = a.m.head_dim >> 1, pos = rope_row(__ldcg(a.rs.pos + row), a.m.max_seq);
            const float4* cs = reinterpret_cast<const float4*>(a.rope + (size_t)pos * half + (m0 & (half - 1)));
            p.x0 = __ldg(cs);
            p.x1 = __ldg(cs + 1);
        }
    }
    return p;
}

// The activations of rows that are split into several 16-bit parts, as the single-row kernels compute them.  Not inlined: the
// kernel's code size is a cost of its own (see k_gemm_stream), and these rows are few.
__device__ __noinline__ float4 act_f4(float4 v, bool gelu) {
    if (gelu) return make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
    return make_float4(silu_f(v.x), silu_f(v.y), silu_f(v.z), silu_f(v.w));
}

// What happens to complete sums: lane l of the calling warp holds v = four consecutive weight rows of batch row `row`
// (lanes 0..15: half 0 of the tile, 16..31: half 1), first of them m0 of matrix gi; ok = false past the matrix' end (nothing is
// stored; the warp's exchanges still take place).
template <int EPI, bool BF16>
__device__ __forceinline__ void sg_epilogue_row(const SgArgs& a, int row, float4 v, const SgRowPre& pre, int4 ctl, float4 bias, int lane, int gi, int m0, bool ok) {
#define ESP_SG_G(field) (gi == 0 ? a.g[0].field : gi == 1 ? a.g[1].field : a.g[2].field)
    v.x += bias.x; v.y += bias.y; v.z += bias.z; v.w += bias.w;
    const bool dbg = a.debug && row == 0;
    if constexpr (EPI == SG_STORE) {
        if (ok) *reinterpret_cast<float4*>(ESP_SG_G(out) + (size_t)row * ESP_SG_G(ldo) + m0) = v;
    } else if constexpr (EPI == SG_RESIDUAL) {
        v.x += pre.x0.x; v.y += pre.x0.y; v.z += pre.x0.z; v.w += pre.x0.w;
        if (ok) *reinterpret_cast<float4*>(a.g[0].out + (size_t)row * a.g[0].ldo + m0) = v;
        else v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.stat_out) {
            const int n = min(kSgRows, a.g[0].M - (int)blockIdx.y * kSgRows);
            const float2 st = tile_stat(v, ok, n, a.m.arch == ARCH_LLAMA);
            if (lane == 0) a.stat_out[(size_t)row * gridDim.y + blockIdx.y] = st;
        }
    } else if constexpr (EPI == SG_QKV) {
        const int hd = a.m.head_dim, half = hd >> 1;
        const int i0 = m0 & (hd - 1), head = m0 / hd;
        if (a.rope) {  // lanes of a rotation pair are head_dim / 8 apart
            float4 p;
            p.x = __shfl_xor_sync(0xffffffffu, v.x, hd >> 3); p.y = __shfl_xor_sync(0xffffffffu, v.y, hd >> 3);
            p.z = __shfl_xor_sync(0xffffffffu, v.z, hd >> 3); p.w = __shfl_xor_sync(0xffffffffu, v.w, hd >> 3);
            if (gi < 2) {
                const float4 c0 = pre.x0, c1 = pre.x1;
                const float sg = i0 < half ? -1.f : 1.f;
                v.x = fmaf(v.x, c0.x, sg * p.x * c0.y); v.y = fmaf(v.y, c0.z, sg * p.y * c0.w);
                v.z = fmaf(v.z, c1.x, sg * p.z * c1.y); v.w = fmaf(v.w, c1.z, sg * p.w * c1.w);
            }
        }
        if (!ok) return;
        if (gi == 0) {
            *reinterpret_cast<float4*>(a.g[0].out + (size_t)row * a.g[0].ldo + m0) = v;
            if (dbg) *reinterpret_cast<float4*>(a.debug + m0) = v;
        } else {
            const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
            __half* dst = (gi == 1 ? a.kv.k : a.kv.v) + a.kv.offset(a.m, a.layer, ctl.z, head, ctl.y) + i0;
            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            if (dbg) {
                const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
                *reinterpret_cast<float4*>(a.debug + a.m.q_dim + (gi == 2 ? a.m.kv_dim : 0) + m0) = make_float4(f0.x, f0.y, f1.x, f1.y);
            }
        }
    } else if constexpr (EPI == SG_GELU) {
        if (a.parts > 1) v = act_f4(v, true);
        else v = make_float4(gelu_fast(v.x), gelu_fast(v.y), gelu_fast(v.z), gelu_fast(v.w));
        if (ok) store_parts4(a.out16, a.ld16, row, m0, v, a.parts, BF16);
        if (ok && dbg) *reinterpret_cast<float4*>(a.debug + m0) = v;
    } else if constexpr (EPI == SG_SWIGLU) {  // lanes 0..15 hold the gate values, 16..31 the up values of the same hidden units
        float4 u;
        u.x = __shfl_xor_sync(0xffffffffu, v.x, 16); u.y = __shfl_xor_sync(0xffffffffu, v.y, 16);
        u.z = __shfl_xor_sync(0xffffffffu, v.z, 16); u.w = __shfl_xor_sync(0xffffffffu, v.w, 16);
        if (a.parts > 1) v = act_f4(v, false);
        else v = make_float4(silu_fast(v.x), silu_fast(v.y), silu_fast(v.z), silu_fast(v.w));
        v = make_float4(v.x * u.x, v.y * u.y, v.z * u.z, v.w * u.w);
        if (ok && lane < 16) {
            store_parts4(a.out16, a.ld16, row, m0, v, a.parts, BF16);
            if (dbg) *reinterpret_cast<float4*>(a.debug + m0) = v;
        }
    }
#undef ESP_SG_G
}
// The rows a warp finishes (see k_gemm_stream) and where their partial sums lie.
struct SgFinish {
    const float* sums;  // this lane's four weight rows of (slice 0, part 0, the warp's first own row)
    const int4* ctl;
    int rows, n0, splits, own, r_first, r_step, lane, gi, m0;
    bool valid;
};
template <int EPI, bool BF16>
__device__ __forceinline__ void sg_finish_rows(const SgArgs& a, const SgFinish& f, SgRowPre now, float4 bias) {
    const float* src = f.sums;
    const int n_parts = f.splits * a.parts, stride = f.own * kSgRows;
#pragma unroll 1
    for (int r = f.r_first; r < f.rows; r += f.r_step) {
        SgRowPre next = now;  // the next row's reads are in flight while this one is finished
        if (r + f.r_step < f.rows) next = sg_row_prefetch(a, f.n0 + r + f.r_step, f.gi, f.m0, f.valid);
        const int4 ctl = f.ctl[r];
        float4 v = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
        for (int i = 1; i < n_parts; i++) {
            const float4 t = *reinterpret_cast<const float4*>(src + (size_t)i * stride);
            v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        if (ctl.x) sg_epilogue_row<EPI, BF16>(a, f.n0 + r, v, now, ctl, bias, f.lane, f.gi, f.m0, f.valid);
        now = next;
        src += (kSgThreads / 32) * kSgRows;  // the warp's next own row
    }
}

// Arg-max over the tile's 128 vocabulary rows: the CTA's threads are dealt out evenly over the batch columns (4 per row at 64
// columns .. 32 at 8); a row's threads interleave over its sums, each starting at a bank of its own.  The packed key keeps
// the first maximum whatever the order.
__device__ __forceinline__ void sg_head_rows(const SgArgs& a, const float* part, const int4* ctl, int rows, int n0, int own, int m_h0, int m_h1) {
    const int cols = a.parts > 1 ? 8 : a.n_cols;
    const int lg = cols <= 8 ? 5 : cols <= 16 ? 4 : cols <= 32 ? 3 : 2, tpr = 1 << lg, count = kSgRows >> lg;
    const int r = (int)threadIdx.x >> lg, sub = (int)threadIdx.x & (tpr - 1);
    unsigned long long key = 0ull;
    if (r < rows && ctl[r].x) {
        const float* src = part + r * kSgRows;
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        const int last0 = a.g[0].M - m_h0, last1 = a.g[0].M - m_h1 + kSgHalf;  // valid sums of the halves end here
#pragma unroll 4
        for (int i = 0; i < count; i++) {
            const int e = sub + (((i + r) & (count - 1)) << lg);
            float x = src[e];
            if (a.parts > 1) x += src[e + own * kSgRows];
            if (a.parts > 2) x += src[e + 2 * own * kSgRows];
            const int m = (e < kSgHalf ? m_h0 : m_h1 - kSgHalf) + e;
            const bool better = x > bv || (x == bv && m < bi);  // (a NaN logit is never chosen)
            if (better && e < (e < kSgHalf ? last0 : last1)) { bv = x; bi = m; }
        }
        if (a.logits) {
#pragma unroll 1
            for (int e = sub; e < kSgRows; e += tpr) {
                float x = src[e];
#pragma unroll 1
                for (int j = 1; j < a.parts; j++) x += src[e + j * own * kSgRows];
                if (e < (e < kSgHalf ? last0 : last1)) a.logits[(size_t)(n0 + r) * a.g[0].M + (e < kSgHalf ? m_h0 : m_h1 - kSgHalf) + e] = x;
            }
        }
        if (bi != 0x7fffffff) key = pack_best(bv, bi + a.row_offset);
    }
#pragma unroll 1
    for (int o = 1; o < tpr; o <<= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
    if (sub == 0 && key) atomicMax(a.rs.best + n0 + r, key);
}

// Pushes eight accumulator columns of this thread's lane (batch rows r .. r + 7 of one part) to the CTAs that finish those
// rows.  Straight-line on purpose: the buffer has room for every column, so columns without a row are stored as well (a
// branch per column cost 110 cycles each).
__device__ __forceinline__ void sg_push8(uint32_t taddr, uint32_t at, int r, int splits) {
    uint32_t v[8];
    tmem_ld_cols<8>(taddr, v);
    uint32_t q = (uint32_t)r / (uint32_t)splits, owner = (uint32_t)r - q * (uint32_t)splits;
    at += q * (kSgRows * 4);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) {
        st_cluster(mapa(at, owner), __uint_as_float(v[i]));  // (one slice: this CTA is its own cluster)
        const bool wrap = owner + 1 == (uint32_t)splits;
        owner = wrap ? 0u : owner + 1;
        at += wrap ? (uint32_t)(kSgRows * 4) : 0u;
    }
}

struct EmbedArgs {
    ModelDims m;
    RowState rs;
    const uint16_t* tok_emb;
    const uint16_t* pos_emb;  // GPT-2, else null
    int emb_type;
    float* hidden;            // [rows][d_model]
    float2* stat;             // [rows][stat_tiles], or null
    int stat_tiles;
};
// hidden = token embedding (+ position embedding) and its per-128-column statistics; one CTA per row, a warp per tile.
__global__ void __launch_bounds__(kThreads) k_embed_rows(const EmbedArgs p) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, lane = threadIdx.x & 31, d = p.m.d_model;
    if (!__ldcg(p.rs.active + r)) return;
    const uint16_t* te = p.tok_emb + (size_t)__ldcg(p.rs.tok + r) * d;
    const uint16_t* pe = p.pos_emb ? p.pos_emb + (size_t)__ldcg(p.rs.pos + r) * d : nullptr;
    for (int t = threadIdx.x >> 5; t < p.stat_tiles; t += kWarps) {
        const int k = t * kSgRows + lane * 4;
        const bool ok = k < d;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ok) {
            const uint2 a = __ldg(reinterpret_cast<const uint2*>(te + k));
            v = make_float4(emb_to_float((uint16_t)(a.x & 0xffffu), p.emb_type), emb_to_float((uint16_t)(a.x >> 16), p.emb_type),
                            emb_to_float((uint16_t)(a.y & 0xffffu), p.emb_type), emb_to_float((uint16_t)(a.y >> 16), p.emb_type));
            if (pe) {
                const uint2 b = __ldg(reinterpret_cast<const uint2*>(pe + k));
                v.x += emb_to_float((uint16_t)(b.x & 0xffffu), p.emb_type); v.y += emb_to_float((uint16_t)(b.x >> 16), p.emb_type);
                v.z += emb_to_float((uint16_t)(b.y & 0xffffu), p.emb_type); v.w += emb_to_float((uint16_t)(b.y >> 16), p.emb_type);
            }
            *reinterpret_cast<float4*>(p.hidden + (size_t)r * d + k) = v;
        }
        if (!p.stat) continue;
        const float2 st = tile_stat(v, ok, min(kSgRows, d - t * kSgRows), p.m.arch == ARCH_LLAMA);
        if (lane == 0) p.stat[(size_t)r * p.stat_tiles + t] = st;
    }
}

// grid = (column tiles, row tiles, K slices), cluster = (1, 1, K slices).
// One kernel for all epilogues, and small on purpose: with a few hundred instructions per warp and launch, instruction fetch
// was most of the time (no_instruction 7 to 12 of 15 stall cycles per issue at 137 KB of code; an instance per epilogue was
// slower still: 1079 against 800 us per step of the 1.1B shape at 5 rows).  Hence rolled loops wherever they are not hot.
template <bool BF16>
__global__ void __launch_bounds__(kSgThreads, 2) k_gemm_stream(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                                                               const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x,
                                                               const __grid_constant__ SgArgs a) {
    extern __shared__ __align__(1024) uint8_t sg_smem[];
    __shared__ uint64_t s_full[kSgMaxStages], s_empty[kSgMaxStages], s_acc;
    __shared__ uint32_t s_tmem;
    __shared__ float2 s_stat[kSgMaxCols];
    __shared__ int4 s_ctl[kSgMaxCols];  // {active, position, sequence} of the tile's rows
    __shared__ unsigned int s_ticket;
    uint8_t* const tiles = reinterpret_cast<uint8_t*>(((uintptr_t)sg_smem + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stages = a.stages, stage_bytes = kSgWBytes + a.n_cols * 128;
    const int splits = (int)gridDim.z, slice = (int)blockIdx.z;  // the cluster covers z: the rank is the slice
    const int n0 = (int)blockIdx.x * a.n_cols;
    const int rows = min(a.rows - n0, a.n_cols);
    // the two 64-row halves of this tile: (matrix, first row)
    int g0 = 0, g1 = 0, m_h0, m_h1;
    if (a.epilogue == SG_SWIGLU) {
        g1 = 1;
        m_h0 = m_h1 = (int)blockIdx.y * kSgHalf;
    } else {
        const int h0 = 2 * (int)blockIdx.y, h1 = h0 + 1;
        if (a.n_groups > 1) { g0 = h0 >= a.g[1].half0 ? 1 : 0; g1 = h1 >= a.g[1].half0 ? 1 : 0; }
        if (a.n_groups > 2) { if (h0 >= a.g[2].half0) g0 = 2; if (h1 >= a.g[2].half0) g1 = 2; }
        m_h0 = (h0 - (g0 == 0 ? 0 : g0 == 1 ? a.g[1].half0 : a.g[2].half0)) * kSgHalf;
        m_h1 = (h1 - (g1 == 0 ? 0 : g1 == 1 ? a.g[1].half0 : a.g[2].half0)) * kSgHalf;  // past the last matrix: loads as zeros
    }
    const CUtensorMap* const map_h0 = g0 == 0 ? &map_w0 : g0 == 1 ? &map_w1 : &map_w2;
    const CUtensorMap* const map_h1 = g1 == 0 ? &map_w0 : g1 == 1 ? &map_w1 : &map_w2;
    const int kb0 = slice * a.kb_per_split;
    const int num_kb = min(a.kb_per_split, a.K / kTcBlockK - kb0);
    const bool norm = a.hidden != nullptr;
    const uint32_t tx = (uint32_t)(kSgWBytes + (norm ? 0 : a.n_cols * 128));
    // exchange buffer [slice][part][own row][128]: behind the ring, or (one slice) over it
    const int own = ((a.parts > 1 ? 8 : a.n_cols) + splits - 1) / splits;  // batch rows a CTA finishes
    float* const part = reinterpret_cast<float*>(tiles + (splits > 1 ? (size_t)stages * stage_bytes : 0));
    const bool in1 = lane >= 16;
    const int gi = in1 ? g1 : g0;
    const int m0 = (in1 ? m_h1 : m_h0) + 4 * (lane & 15);
    const bool valid = m0 < (gi == 0 ? a.g[0].M : gi == 1 ? a.g[1].M : a.g[2].M);
    auto load_w = [&](int kb, int s) {
        uint8_t* dst = tiles + (size_t)s * stage_bytes;
        mbar_expect_tx(s_full + s, tx);
        tma_load_2d(dst, map_h0, (kb0 + kb) * kTcBlockK, m_h0, s_full + s);
        tma_load_2d(dst + kSgWBytes / 2, map_h1, (kb0 + kb) * kTcBlockK, m_h1, s_full + s);
    };

    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int s = 0; s < stages; s++) { mbar_init(s_full + s, norm ? 2 : 1); mbar_init(s_empty + s, 1); }
        mbar_init(&s_acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    uint32_t tmem_cols = 32;
    while ((int)tmem_cols < a.n_cols) tmem_cols <<= 1;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (splits > 1) cluster_arrive();  // every CTA of the cluster has started: waited for before the first remote store
    // Stage warps.  A warp serves one ring stage for good: it sees that stage's phases one after the other (a warp that moved
    // from stage to stage could ask for a phase two ahead, which a parity wait cannot tell from one that has completed), and
    // six warps issue their copies side by side - one warp took 320 cycles per copy, 610 per k block, and bounded the ring.
    const int xw = warp - 2;
    const bool feeds = xw >= 0 && xw < min(stages, num_kb);
    uint8_t* const sw = tiles + (size_t)max(xw, 0) * stage_bytes;
    SgNormPre pre_x;
    if (feeds) {
        if (elect_one()) load_w(xw, xw);  // weights do not depend on the previous kernel
        if (norm) sg_norm_gains(a, pre_x, (kb0 + xw) * kTcBlockK, lane);
    }
    float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
    {
        const float* bias = gi == 0 ? a.g[0].bias : gi == 1 ? a.g[1].bias : a.g[2].bias;
        if (bias && valid) bias4 = __ldg(reinterpret_cast<const float4*>(bias + m0));
    }
    if (warp == 0) l2_request(a.ahead, ((unsigned)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x, gridDim.x * gridDim.y * gridDim.z, lane);
    pdl_launch_dependents();  // (only now: a CTA of this kernel must never queue for TMEM behind its successor)
    pdl_wait();
    const uint32_t acc = s_tmem;
    if (warp == 0) {  // read by the epilogue, several barriers later
#pragma unroll 1
        for (int r = lane; r < rows; r += 32) {
            const bool kv_rows = a.epilogue == SG_QKV;
            s_ctl[r] = make_int4(a.all_rows ? 1 : __ldcg(a.rs.active + n0 + r), kv_rows ? __ldcg(a.rs.pos + n0 + r) : 0, kv_rows ? __ldcg(a.rs.seq + n0 + r) : 0, 0);
        }
    }

    if (warp == 1) {
        // ---------------- MMA issuer (see elect_one for the shape of this loop) ----------------
        const uint32_t idesc = umma_idesc_f16(kSgRows, a.n_cols, BF16);
        // Everything the loop needs is kept up by counting; the next stage's barrier is tested before this stage's MMAs.
        const uint64_t d_first = umma_smem_desc_sw128(tiles);
        const uint32_t d_step = (uint32_t)stage_bytes >> 4;
        const uint32_t full0 = smem_u32(s_full), empty0 = smem_u32(s_empty);
        uint32_t s = 0, phase = 0, accumulate = 0;
        uint64_t da = d_first;
        bool ready = mbar_test(full0, 0);
        for (int kb = 0; kb < num_kb; kb++) {
            const bool gave_up = !ready && !tc_wait(s_full + s, phase, a.error);  // (per lane: the vote below ends the loop for all)
            const bool wrap = (int)s + 1 == stages;
            const uint32_t s_next = wrap ? 0 : s + 1, phase_next = phase ^ (wrap ? 1u : 0u);
            ready = kb + 1 < num_kb && mbar_test(full0 + 8 * s_next, phase_next);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one() && !gave_up) {
                const uint64_t db = da + (kSgWBytes >> 4);
                umma_f16(acc, da, db, idesc, accumulate);
#pragma unroll
                for (int k = 1; k < kTcBlockK / 16; k++) umma_f16(acc, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, 1u);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(empty0 + 8 * s) : "memory");
            }
            if (__any_sync(0xffffffffu, gave_up)) break;
            accumulate = 1;
            s = s_next;
            phase = phase_next;
            da = wrap ? d_first : da + d_step;
        }
        if (elect_one()) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s_acc)) : "memory");
    } else if (xw >= 0) {
        // ---------------- stage warps ----------------
        if (norm) {
            if (feeds) sg_norm_rows(a, pre_x, n0, 0, rows, (kb0 + xw) * kTcBlockK, lane);
            sg_row_stats(a, s_stat, n0, rows, xw, lane);
            asm volatile("bar.sync 2, %0;" ::"n"(kSgXWarps * 32) : "memory");
        }
        if (feeds) {
            uint32_t phase = 1;
#pragma unroll 1
            for (int kb = xw; kb < num_kb; kb += stages) {
                const int k0 = (kb0 + kb) * kTcBlockK;
                phase ^= 1u;
                if (kb >= stages) {
                    if (norm) {  // (requested before the wait for the stage)
                        sg_norm_gains(a, pre_x, k0, lane);
                        sg_norm_rows(a, pre_x, n0, 0, rows, k0, lane);
                    }
                    if (!tc_wait_warp(s_empty + xw, phase ^ 1u, a.error)) break;
                    if (elect_one()) load_w(kb, xw);
                }
                if (!norm) {
                    if (elect_one()) tma_load_2d(sw + kSgWBytes, &map_x, k0, n0, s_full + xw);
                    __syncwarp();
                    continue;
                }
#pragma unroll 1
                for (int r0 = 0; r0 < rows; r0 += 16) {
                    if (r0 > 0) sg_norm_rows(a, pre_x, n0, r0, rows, k0, lane);
                    sg_norm_store<BF16>(a, pre_x, sw + kSgWBytes, s_stat, r0, rows, lane);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(s_full + xw);
            }
        }
    }
    __syncwarp();

    // ---------------- accumulator -> the shared memory of the CTA that finishes the row ----------------
    // This CTA finishes rows slice, slice + splits, ...: one per warp at a time; what their epilogues read is requested here.
    const int r_first = slice + splits * warp, r_step = splits * (kSgThreads / 32);
    SgRowPre ahead{};
    if (r_first < rows) ahead = sg_row_prefetch(a, n0 + r_first, gi, m0, valid);
    if (splits > 1) cluster_wait();
    const bool ok = tc_wait(&s_acc, 0, a.error);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok) {
        // a wait gave up (the results are void): the copies still in flight must land before the CTA may leave
        if (threadIdx.x == 0)
#pragma unroll 1
            for (int kb = max(0, num_kb - stages); kb < num_kb; kb++) {
                unsigned spins = 0;
                while (!mbar_try_wait(s_full + kb % stages, (kb / stages) & 1) && ++spins < kTcSpinLimit / 64) {}
            }
    }
    __syncwarp();  // (every MMA has read its stages: with one slice the buffer may overwrite them)
    {
        const uint32_t trow = acc + ((uint32_t)(32 * (warp & 3)) << 16);
        const int per = a.n_cols >> 1, c_begin = (warp >> 2) * per;
        const uint32_t lane_at = (uint32_t)(32 * (warp & 3) + lane) * 4;
        const uint32_t base = smem_u32(part) + (uint32_t)(slice * a.parts * own * kSgRows) * 4 + lane_at;
#pragma unroll 1
        for (int c = c_begin; c < c_begin + per; c += 8) {
            const int j = a.parts > 1 ? c >> 3 : 0;  // eight columns: one part of up to eight rows, or eight rows
            if (j < a.parts) sg_push8(trow + (uint32_t)c, base + (uint32_t)(j * own * kSgRows) * 4, a.parts > 1 ? 0 : c, splits);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (splits > 1) { cluster_arrive(); cluster_wait(); }
    else __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(acc), "r"(tmem_cols) : "memory");
    }

    // ---------------- complete sums and epilogue: this CTA's rows, a warp per row ----------------
    const float* const sums = part + warp * kSgRows + lane * 4;
    const SgFinish f{sums, s_ctl, rows, n0, splits, own, r_first, r_step, lane, gi, m0, valid};
    switch (a.epilogue) {
        case SG_STORE: sg_finish_rows<SG_STORE, BF16>(a, f, ahead, bias4); break;
        case SG_RESIDUAL: sg_finish_rows<SG_RESIDUAL, BF16>(a, f, ahead, bias4); break;
        case SG_QKV: sg_finish_rows<SG_QKV, BF16>(a, f, ahead, bias4); break;
        case SG_GELU: sg_finish_rows<SG_GELU, BF16>(a, f, ahead, bias4); break;
        case SG_SWIGLU: sg_finish_rows<SG_SWIGLU, BF16>(a, f, ahead, bias4); break;
        default: sg_head_rows(a, part, s_ctl, rows, n0, own, m_h0, m_h1); break;  // (never sliced along K)
    }
    if (a.epilogue == SG_HEAD && a.finalize >= 0) {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_ticket = atomicAdd(a.rs.ticket, 1u);
        __syncthreads();
        if (s_ticket == gridDim.x * gridDim.y * gridDim.z - 1) {
            __threadfence();
            head_finalize(a.m, a.rows, a.rs, a.finalize);
            if (threadIdx.x == 0) *a.rs.ticket = 0u;
        }
    }
}

}  // namespace esp
