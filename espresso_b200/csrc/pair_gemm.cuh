// Products of wide prompt passes (more than kSgMaxRows rows): Y[n][m] = sum_k W[m][k] * X[n][k] on pairs of SMs.
//
// Bound: the tensor pipe.  A single SM's 128 x 256 tile needs 48 KB of operands per 64-wide K block, 96 bytes per cycle at
// the pipe's rate of 512 cycles per block, more than an SM can pull out of L2 (about 64): such a kernel stood at 0.6 of the
// pipe.  tcgen05.mma.cta_group::2 multiplies a 256 x 256 tile with the operands of two SMs: each loads 128 batch rows and
// 128 weight rows per block, 64 bytes per cycle, and accumulates its 128 batch rows x 256 weight rows.
//
// Persistent: one CTA per SM, tiles dealt out in turn (batch tiles fastest, so that the tiles in flight share weights in L2);
// the accumulator is double-buffered (2 x 256 TMEM columns), the epilogue of a tile runs under the products of the next.
// The epilogue moves 32 columns at a time through a private staging area so that global accesses run along the weight rows.
//
// Roles (320 threads): warp 0 TMA, warp 1 MMA (in the pair's first CTA), warps 2..9 epilogue.  Barriers: `full` of the first
// CTA counts the bytes of both CTAs' copies; `empty` and `acc_full` are arrived in both CTAs by one commit; `acc_empty` of the
// first CTA collects the sixteen epilogue warps of the pair.  Every wait is bounded (error code 7).
#pragma once
#include "stream_gemm.cuh"

namespace esp {

constexpr int kPgThreads = 320;
constexpr int kPgEpiWarps = 8;
constexpr int kPgRows = 256;         // batch rows of a tile (128 per CTA)
constexpr int kPgStages = 5;
constexpr int kPgXBytes = 128 * kTcBlockK * 2, kPgWBytes = 128 * kTcBlockK * 2;
constexpr int kPgStageBytes = kPgXBytes + kPgWBytes;
constexpr int kPgStageStride = 36;   // floats per staged row of 32 columns: 16-byte aligned, conflict-free
constexpr int kPgEpiBytes = kPgEpiWarps * 32 * kPgStageStride * 4;
constexpr size_t kPgSmemBytes = (size_t)kPgStages * kPgStageBytes + kPgEpiBytes + 1024;

enum PgEpilogue { PG_STORE = 0, PG_RESIDUAL = 1, PG_GELU = 2, PG_SWIGLU = 3 };

struct PgGroup {
    int M;              // weight rows (a multiple of 4)
    int half0;          // index of its first 128-row half
    float* out;         // PG_STORE / PG_RESIDUAL: [n][ldo] fp32
    int ldo;
    const float* bias;  // [M] or null
};
struct PgArgs {
    PgGroup g[3];
    int n_groups;
    int K, rows;
    int tiles_n, tiles_w;  // batch tiles of 256 rows, weight tiles of two halves
    int epilogue, bf16;
    uint16_t* out16;       // PG_GELU / PG_SWIGLU: [n][ld16]
    int ld16;
    const int* active;     // [rows]: rows with 0 are not written
    float* debug;          // optional capture of batch row 0 (PG_GELU / PG_SWIGLU)
    int* error;
};

template <>
__device__ __forceinline__ void tmem_ld_cols<32>(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, "
        "%24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// A copy into this CTA's shared memory that completes on the pair's first CTA's barrier (same offset, rank bit cleared).
__device__ __forceinline__ void tma_load_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
                 "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar) & 0xFEFFFFFFu)
                 : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void arrive_first_cta(uint64_t* bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(smem_u32(bar), 0)) : "memory");
}

// The 32 x 32 block in a warp's staging rows (batch rows nrow0.., weight rows m0..) to memory: eight lanes x four columns per
// batch row, four rows per step; live = the rows to write.  Whole blocks take the branch-free form: all reads of the staging
// rows and of the residual are in flight before the first store.
template <int EPI, bool WHOLE>
__device__ __forceinline__ void pg_store_rows(const PgArgs& a, const float* stg, int rr, int c, int nrow0, unsigned live, float* out, size_t step, int m, const float4& b) {
    float4 res[8];
    if constexpr (EPI == PG_RESIDUAL) {
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (WHOLE || ((live >> (4 * i + rr)) & 1u)) res[i] = *reinterpret_cast<const float4*>(out + i * step);
    }
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = *reinterpret_cast<const float4*>(stg + (4 * i + rr) * kPgStageStride + c);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = 4 * i + rr;
        if (!WHOLE && !((live >> r) & 1u)) continue;
        v[i].x += b.x; v[i].y += b.y; v[i].z += b.z; v[i].w += b.w;
        if constexpr (EPI == PG_RESIDUAL) { v[i].x += res[i].x; v[i].y += res[i].y; v[i].z += res[i].z; v[i].w += res[i].w; }
        if constexpr (EPI == PG_STORE || EPI == PG_RESIDUAL) {
            *reinterpret_cast<float4*>(out + i * step) = v[i];
        } else {
            if constexpr (EPI == PG_GELU) v[i] = make_float4(gelu_fast(v[i].x), gelu_fast(v[i].y), gelu_fast(v[i].z), gelu_fast(v[i].w));
            *reinterpret_cast<uint2*>(a.out16 + (size_t)(nrow0 + r) * a.ld16 + m) = make_uint2(pack16x2(v[i].x, v[i].y, a.bf16), pack16x2(v[i].z, v[i].w, a.bf16));
            if (a.debug && nrow0 + r == 0) *reinterpret_cast<float4*>(a.debug + m) = v[i];
        }
    }
}
template <int EPI>
__device__ __forceinline__ void pg_store_block(const PgArgs& a, const float* stg, int lane, int nrow0, unsigned live, int gi, int m0) {
#define ESP_PG_G(field) (gi == 0 ? a.g[0].field : gi == 1 ? a.g[1].field : a.g[2].field)
    const int c = (lane & 7) * 4, rr = lane >> 3, m = m0 + c;
    if (m >= ESP_PG_G(M)) return;
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (const float* bias = ESP_PG_G(bias)) b = __ldg(reinterpret_cast<const float4*>(bias + m));
    float* const out = EPI <= PG_RESIDUAL ? ESP_PG_G(out) + (size_t)(nrow0 + rr) * ESP_PG_G(ldo) + m : nullptr;
    const size_t step = (size_t)4 * ESP_PG_G(ldo);
#undef ESP_PG_G
    if (live == 0xffffffffu) pg_store_rows<EPI, true>(a, stg, rr, c, nrow0, live, out, step, m, b);
    else pg_store_rows<EPI, false>(a, stg, rr, c, nrow0, live, out, step, m, b);
}

// One accumulator (this warp's 32 batch rows x its columns of both halves) to memory.  half_of: see k_gemm_pair.
template <int EPI, class HalfOf>
__device__ __forceinline__ void pg_epilogue(const PgArgs& a, float* stg, uint32_t base, int sub, int lane, int nrow0, unsigned live, int tile_w, HalfOf half_of) {
#pragma unroll 1
    for (int blk = 0; blk < (EPI == PG_SWIGLU ? 2 : 4); blk++) {  // 32 columns: half blk / 2, its columns sub * 64 + (blk & 1) * 32
        const int h = blk >> 1, col = sub * 64 + (blk & 1) * 32;
        uint32_t v[32];
        tmem_ld_cols<32>(base + (uint32_t)(h * 128 + col), v);
        if constexpr (EPI == PG_SWIGLU) {
            uint32_t u[32];
            tmem_ld_cols<32>(base + (uint32_t)(128 + col), u);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = __float_as_uint(silu_fast(__uint_as_float(v[i])) * __uint_as_float(u[i]));
        } else {
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        float* const mine = stg + lane * kPgStageStride;
#pragma unroll
        for (int i = 0; i < 8; i++) reinterpret_cast<uint4*>(mine)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        __syncwarp();
        int gi, m0;
        half_of(tile_w, h, gi, m0);
        pg_store_block<EPI>(a, stg, lane, nrow0, live, gi, m0 + col);
        __syncwarp();
    }
}

// grid = up to one CTA per SM (an even number), cluster = 2.
__global__ void __launch_bounds__(kPgThreads, 1) k_gemm_pair(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                                                             const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x,
                                                             const __grid_constant__ PgArgs a) {
    extern __shared__ __align__(1024) uint8_t pg_smem[];
    __shared__ uint64_t s_full[kPgStages], s_empty[kPgStages], s_acc_full[2], s_acc_empty[2];
    __shared__ uint32_t s_tmem;
    uint8_t* const tiles = reinterpret_cast<uint8_t*>(((uintptr_t)pg_smem + 1023) & ~(uintptr_t)1023);
    float* const stage_area = reinterpret_cast<float*>(tiles + (size_t)kPgStages * kPgStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1, pair = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;
    const int n_tiles = a.tiles_n * a.tiles_w, num_kb = a.K / kTcBlockK;
    // (matrix, first row) of a 128-row half; past the last matrix the rows load as zeros
    auto half_of = [&](int tile_w, int h, int& gi, int& m0) {
        if (a.epilogue == PG_SWIGLU) { gi = h; m0 = tile_w * 128; return; }  // half 0 gate, half 1 the same rows of the up matrix
        const int x = 2 * tile_w + h;
        gi = 0;
        if (a.n_groups > 1 && x >= a.g[1].half0) gi = 1;
        if (a.n_groups > 2 && x >= a.g[2].half0) gi = 2;
        m0 = (x - (gi == 0 ? 0 : gi == 1 ? a.g[1].half0 : a.g[2].half0)) * 128;
    };
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPgStages; s++) { mbar_init(s_full + s, 1); mbar_init(s_empty + s, 1); }
        for (int i = 0; i < 2; i++) { mbar_init(s_acc_full + i, 1); mbar_init(s_acc_empty + i, 2 * kPgEpiWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_arrive();  // both CTAs' barriers are initialised and their tensor memory is allocated before either is used
    cluster_wait();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tmem = s_tmem;

    if (warp == 0) {
        // ---------------- TMA producer: this CTA's 128 batch rows and its weight half ----------------
        int s = 0;
        uint32_t phase = 0;
        bool first_round = true, ok = true;
        for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
            const int tw = tile / a.tiles_n, n0 = (tile - tw * a.tiles_n) * kPgRows + rank * 128;
            int gi, m0;
            half_of(tw, rank, gi, m0);
            const CUtensorMap* const map = gi == 0 ? &map_w0 : gi == 1 ? &map_w1 : &map_w2;
            for (int kb = 0; kb < num_kb; kb++) {
                if (!first_round && !tc_wait(s_empty + s, phase ^ 1u, a.error)) { ok = false; break; }
                if (elect_one()) {
                    uint8_t* const sx = tiles + (size_t)s * kPgStageBytes;
                    if (rank == 0) mbar_expect_tx(s_full + s, 2 * kPgStageBytes);
                    tma_load_pair(sx, &map_x, kb * kTcBlockK, n0, s_full + s);
                    tma_load_pair(sx + kPgXBytes, map, kb * kTcBlockK, m0, s_full + s);
                }
                __syncwarp();
                if (++s == kPgStages) { s = 0; phase ^= 1u; first_round = false; }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer of the pair ----------------
        if (rank == 0) {
            const uint32_t idesc = umma_idesc_f16(256, 256, a.bf16);
            const uint64_t d_first = umma_smem_desc_sw128(tiles);
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            int it = 0;
            for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, it++) {
                const int buf = it & 1;
                if (it >= 2 && !tc_wait(s_acc_empty + buf, ((it >> 1) - 1) & 1, a.error)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)buf * 256u;
                uint32_t accumulate = 0;
                bool ready = mbar_try_wait(s_full + s, phase);
                for (int kb = 0; kb < num_kb; kb++) {
                    if (!ready && !tc_wait(s_full + s, phase, a.error)) { ok = false; break; }
                    const bool wrap = s + 1 == kPgStages;
                    const int s_next = wrap ? 0 : s + 1;
                    const uint32_t phase_next = phase ^ (wrap ? 1u : 0u);
                    ready = kb + 1 < num_kb && mbar_try_wait(s_full + s_next, phase_next);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const uint64_t da = d_first + (uint64_t)(s * (kPgStageBytes >> 4)), db = da + (kPgXBytes >> 4);
                        umma_pair(acc, da, db, idesc, accumulate);
#pragma unroll
                        for (int k = 1; k < kTcBlockK / 16; k++) umma_pair(acc, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, 1u);
                        commit_pair(s_empty + s);
                    }
                    __syncwarp();
                    accumulate = 1;
                    s = s_next;
                    phase = phase_next;
                }
                if (ok && elect_one()) commit_pair(s_acc_full + buf);
                __syncwarp();
            }
        }
    } else {
        // ---------------- epilogue: TMEM -> registers -> staging -> global ----------------
        const int ew = warp - 2, quad = warp & 3, sub = ew >> 2;  // lanes 32 * quad.. of TMEM; which 64 columns of each half
        float* const stg = stage_area + (size_t)ew * 32 * kPgStageStride;
        int it = 0;
        for (int tile = pair; tile < n_tiles; tile += n_pairs, it++) {
            const int buf = it & 1;
            const int tw = tile / a.tiles_n, nrow0 = (tile - tw * a.tiles_n) * kPgRows + rank * 128 + 32 * quad;
            if (!tc_wait(s_acc_full + buf, (it >> 1) & 1, a.error)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned live = __ballot_sync(0xffffffffu, nrow0 + lane < a.rows && (!a.active || __ldcg(a.active + nrow0 + lane)));
            const uint32_t base = tmem + (uint32_t)buf * 256u + ((uint32_t)(32 * quad) << 16);
            if (live) {
                if (a.epilogue == PG_STORE) pg_epilogue<PG_STORE>(a, stg, base, sub, lane, nrow0, live, tw, half_of);
                else if (a.epilogue == PG_RESIDUAL) pg_epilogue<PG_RESIDUAL>(a, stg, base, sub, lane, nrow0, live, tw, half_of);
                else if (a.epilogue == PG_GELU) pg_epilogue<PG_GELU>(a, stg, base, sub, lane, nrow0, live, tw, half_of);
                else pg_epilogue<PG_SWIGLU>(a, stg, base, sub, lane, nrow0, live, tw, half_of);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) arrive_first_cta(s_acc_empty + buf);
        }
    }
    // nobody leaves while the pair's copies, commits or arrivals may still reach this CTA (after a wait that gave up, copies
    // may be in flight without anyone waiting for them: they land within microseconds)
    if (__ldcg(a.error) != 0) __nanosleep(200000);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace esp
