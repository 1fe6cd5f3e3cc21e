// Products of passes with more rows than the streamed products take: Y[n][m] = sum_k W[m][k] * X[n][k] on pairs of SMs, or on
// single SMs where a pair's tile would be half empty.
//
// Bound: the tensor pipe; below a few hundred rows HBM and what comes before the first and after the last K block of a tile.
// A single SM's 128 x 256 tile needs 48 KB of operands per 64-wide K block, 96 bytes per cycle at the pipe's rate of 512 cycles
// per block, more than an SM can pull out of L2 (about 64).  tcgen05.mma.cta_group::2 multiplies a 256 x 256 tile with the operands of two SMs: each loads 128 batch rows and
// 128 weight rows per block, 64 bytes per cycle, and accumulates its 128 batch rows x 256 weight rows.
// A pair's tile has 256 batch rows: with 257 to 384 the second one is mostly empty and costs as much as the first.  The same
// kernel on a single SM (cta_group::1, 128 batch rows, both weight halves) pays 1.28 times per K block and row, and wins wherever
// it saves a wave; which one is the host's choice per product (pg_shape).  300 rows, us, pairs / single: gate/up 2 x 5632 x 2048
// 27.6 / 19.7, 2 x 14336 x 4096 91.0 / 85.4, 4096 x 14336 46.9 / 41.4; 224 rows of the second 57.9 / 64.1.  A single SM also requests
// the weights of its first stages before it waits for the previous kernel (0.3 us); on pairs the test for that in the copy loop
// costs more than it saves (27.6 -> 29.2 us).
//
// Persistent: one CTA per SM, tiles dealt out in turn (batch tiles fastest, so that the tiles in flight share weights in L2);
// the accumulator is double-buffered (2 x 256 TMEM columns), the epilogue of a tile runs under the products of the next.
// Sixteen epilogue warps move 16 columns at a time through a private staging area so that global accesses run along the weight
// rows (eight warps took 6.6 us per tile with the GELU epilogue, longer than the 4.1 us of a tile's products at K = 768).
// A residual product with too few tiles for the chip is cut along K; its slices add into the residual stream.
//
// Roles (576 threads): warp 0 TMA, warp 1 MMA (in the pair's first CTA), warps 2..17 epilogue.  Barriers: `full` of the first
// CTA counts the bytes of both CTAs' copies; `empty` and `acc_full` are arrived in both CTAs by one commit; `acc_empty` of the
// first CTA collects the epilogue warps of both.  Every wait is bounded (error code 7); after one that ran out, nobody leaves
// before the copies and MMAs in flight are done (`done` and `peer` barriers, pair_drain.h).
#pragma once
#include "pair_drain.h"
#include "stream_gemm.cuh"

namespace esp {

constexpr int kPgThreads = 576;
constexpr int kPgEpiWarps = 16;
constexpr int kPgXBytes = 128 * kTcBlockK * 2, kPgWBytes = 128 * kTcBlockK * 2;
constexpr int kPgEpiBytes = kPgEpiWarps * 32 * 16 * 4;  // 16 columns per staged row
// Tile of a pair (256 batch rows, 128 per CTA, a weight half per CTA) or of a single SM (128 batch rows, both weight halves)
template <bool PAIR>
struct PgTile {
    static constexpr int kRows = PAIR ? 256 : 128;
    static constexpr int kStages = PAIR ? 5 : 4;
    static constexpr int kStageBytes = kPgXBytes + (PAIR ? 1 : 2) * kPgWBytes;  // of one CTA
    static constexpr int kSmemBytes = kStages * kStageBytes + kPgEpiBytes + 1024;
};

enum PgEpilogue { PG_STORE = 0, PG_RESIDUAL = 1, PG_QKV = 2, PG_GELU = 3, PG_SWIGLU = 4 };

struct PgGroup {
    int M;              // weight rows (a multiple of 4)
    int half0;          // index of its first 128-row half
    float* out;         // PG_STORE / PG_RESIDUAL / q of PG_QKV: [n][ldo] fp32
    int ldo;
    const float* bias;  // [M] or null
};
struct PgArgs {
    PgGroup g[3];
    int n_groups;
    int K, rows;
    int tiles_n, tiles_w;  // batch tiles of 256 (pair) or 128 rows, weight tiles of two halves
    int epilogue, bf16;
    uint16_t* out16;       // PG_GELU / PG_SWIGLU: [n][ld16]
    int ld16;
    int splits, kb_per_split;  // K slices (PG_RESIDUAL only; else 1)
    const int* active;     // [rows]: rows with 0 are not written
    float* debug;          // optional capture of batch row 0 (PG_QKV / PG_GELU / PG_SWIGLU)
    // PG_QKV: groups q, k, v
    ModelDims m;
    RowState rs;           // pos, seq
    KvLayout kv;
    const float2* rope;    // null for GPT-2
    int layer;
    int* error;
};

template <>
__device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
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
template <bool PAIR>
__device__ __forceinline__ void pg_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR) umma_pair(tmem_d, da, db, idesc, accumulate);
    else umma_f16(tmem_d, da, db, idesc, accumulate);
}
template <bool PAIR>
__device__ __forceinline__ void pg_commit(uint64_t* bar) {
    if constexpr (PAIR) commit_pair(bar);
    else asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void arrive_first_cta(uint64_t* bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(smem_u32(bar), 0)) : "memory");
}

// Bounded wait that does not give up early because of a recorded error: what it waits for arrives within microseconds.
__device__ __forceinline__ bool pg_wait_quiet(uint64_t* bar, unsigned parity) {
    for (unsigned spins = 0; spins < (1u << 20); spins++) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(smem_u32(bar)), "r"(parity)
                     : "memory");
        if (ok) return true;
        __nanosleep(100);
    }
    return false;
}
__device__ __forceinline__ void mbar_complete_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// What a warp's epilogue works on: 32 batch rows (TMEM lanes) from nrow0, of which `live` are written.
struct PgWarp {
    float* stg;        // private staging rows
    uint32_t base;     // accumulator, this warp's lanes
    int lane, sub, nrow0;
    unsigned live;
    bool first_slice;
    size_t kv_row;     // PG_QKV: this lane's row: (sequence, position) part of its cache offset
    int pos;
};

// Staged rows are 64 bytes, two to a line of banks: XORing the 16-byte chunk with the row's line number makes both the row-wise
// stores and the reads of four lanes per row conflict-free.
__device__ __forceinline__ int pg_swizzle(int row) { return ((row >> 1) & 3) << 2; }

// The 32 x 16 block in the staging rows (weight rows m0.. of matrix gi) to memory: four lanes x four columns per batch row,
// eight rows per step.
template <int EPI>
__device__ __forceinline__ void pg_store_block(const PgArgs& a, const PgWarp& w, int gi, int m0) {
#define ESP_PG_G(field) (gi == 0 ? a.g[0].field : gi == 1 ? a.g[1].field : a.g[2].field)
    const int c = (w.lane & 3) * 4, rr = w.lane >> 2, m = m0 + c;
    const bool ok = m < ESP_PG_G(M);
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (const float* bias = ESP_PG_G(bias))
        if (ok && w.first_slice) b = __ldg(reinterpret_cast<const float4*>(bias + m));
    const bool to_cache = EPI == PG_QKV && gi > 0;
    const int ldo = EPI >= PG_GELU ? a.ld16 : ESP_PG_G(ldo);
    float* const out = EPI >= PG_GELU || to_cache ? nullptr : ESP_PG_G(out) + (size_t)(w.nrow0 + rr) * ldo + m;
#undef ESP_PG_G
    float4 res[4];
    const bool add = EPI == PG_RESIDUAL && a.splits == 1;
    if (add) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (ok && ((w.live >> (8 * i + rr)) & 1u)) res[i] = *reinterpret_cast<const float4*>(out + (size_t)(8 * i) * ldo);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = 8 * i + rr;
        float4 v = *reinterpret_cast<const float4*>(w.stg + r * 16 + (c ^ pg_swizzle(r)));
        size_t at = 0;
        if (EPI == PG_QKV) at = __shfl_sync(0xffffffffu, w.kv_row, r);
        if (!ok || !((w.live >> r) & 1u)) continue;
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
        if (EPI == PG_RESIDUAL) {
            if (add) {
                v.x += res[i].x; v.y += res[i].y; v.z += res[i].z; v.w += res[i].w;
                *reinterpret_cast<float4*>(out + (size_t)(8 * i) * ldo) = v;
            } else {
                red_add_v4(out + (size_t)(8 * i) * ldo, v.x, v.y, v.z, v.w);
            }
        } else if (EPI == PG_STORE || (EPI == PG_QKV && !to_cache)) {
            *reinterpret_cast<float4*>(out + (size_t)(8 * i) * ldo) = v;
            if (EPI == PG_QKV && a.debug && w.nrow0 + r == 0) *reinterpret_cast<float4*>(a.debug + m) = v;
        } else if (EPI == PG_QKV) {
            const int head = m / a.m.head_dim;
            const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
            __half* dst = (gi == 1 ? a.kv.k : a.kv.v) + at + (size_t)head * a.m.max_seq * a.m.head_dim + (m & (a.m.head_dim - 1));
            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            if (a.debug && w.nrow0 + r == 0) {
                const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
                *reinterpret_cast<float4*>(a.debug + a.m.q_dim + (gi == 2 ? a.m.kv_dim : 0) + m) = make_float4(f0.x, f0.y, f1.x, f1.y);
            }
        } else {
            if (EPI == PG_GELU) v = make_float4(gelu_fast(v.x), gelu_fast(v.y), gelu_fast(v.z), gelu_fast(v.w));
            *reinterpret_cast<uint2*>(a.out16 + (size_t)(w.nrow0 + r) * ldo + m) = make_uint2(pack16x2(v.x, v.y, a.bf16), pack16x2(v.z, v.w, a.bf16));
            if (a.debug && w.nrow0 + r == 0) *reinterpret_cast<float4*>(a.debug + m) = v;
        }
    }
}

__device__ __forceinline__ void pg_to_staging(const PgWarp& w, const uint32_t (&v)[16]) {
    float* const mine = w.stg + w.lane * 16;
    const int sw = pg_swizzle(w.lane);
    __syncwarp();  // the block staged before has been read
#pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<uint4*>(mine + ((4 * i) ^ sw)) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    __syncwarp();
}

// One accumulator to memory: per half of 128 weight rows this warp takes two 16-column blocks, chosen so that with RoPE they
// hold the two members of every rotation pair.  half_of: see k_gemm_pair.
template <int EPI, class HalfOf>
__device__ __forceinline__ void pg_epilogue(const PgArgs& a, const PgWarp& w, int tile_w, HalfOf half_of) {
    const bool rope = EPI == PG_QKV && a.rope;
    const int apart = rope ? a.m.head_dim >> 5 : 1;  // blocks between the members of a pair
    const int b0 = (w.sub / apart) * 2 * apart + w.sub % apart;
#pragma unroll 1
    for (int h = 0; h < (EPI == PG_SWIGLU ? 1 : 2); h++) {
        int gi, m0;
        half_of(tile_w, h, gi, m0);
        if (EPI == PG_SWIGLU) {
#pragma unroll 1
            for (int i = 0; i < 2; i++) {
                uint32_t v[16], u[16];
                tmem_ld_cols<16>(w.base + (uint32_t)((b0 + i) * 16), v);
                tmem_ld_cols<16>(w.base + (uint32_t)(128 + (b0 + i) * 16), u);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = __float_as_uint(silu_fast(__uint_as_float(v[j])) * __uint_as_float(u[j]));
                pg_to_staging(w, v);
                pg_store_block<EPI>(a, w, gi, m0 + (b0 + i) * 16);
            }
            continue;
        }
        uint32_t v[16], u[16];
        tmem_ld_cols<16>(w.base + (uint32_t)(h * 128 + b0 * 16), v);
        tmem_ld_cols<16>(w.base + (uint32_t)(h * 128 + (b0 + apart) * 16), u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (EPI == PG_QKV && rope && gi < 2) {  // halves of a head: v is the first, u the second member of sixteen rotation pairs
            const float4* cs = reinterpret_cast<const float4*>(a.rope + (size_t)rope_row(w.pos, a.m.max_seq) * (a.m.head_dim >> 1) + ((b0 * 16) & ((a.m.head_dim >> 1) - 1)));
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float4 f = __ldg(cs + j);
                const float v0 = __uint_as_float(v[2 * j]), u0 = __uint_as_float(u[2 * j]), v1 = __uint_as_float(v[2 * j + 1]), u1 = __uint_as_float(u[2 * j + 1]);
                v[2 * j] = __float_as_uint(v0 * f.x - u0 * f.y); u[2 * j] = __float_as_uint(v0 * f.y + u0 * f.x);
                v[2 * j + 1] = __float_as_uint(v1 * f.z - u1 * f.w); u[2 * j + 1] = __float_as_uint(v1 * f.w + u1 * f.z);
            }
        }
#pragma unroll 1
        for (int i = 0; i < 2; i++) {
            if (i == 1) {
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = u[j];
            }
            pg_to_staging(w, v);
            pg_store_block<EPI>(a, w, gi, m0 + (b0 + i * apart) * 16);
        }
    }
}

// grid = up to one CTA per SM; PAIR: an even number, cluster = 2.  Single SM: the CTA is the first and only one of its "pair".
template <bool PAIR>
__global__ void __launch_bounds__(kPgThreads, 1) k_gemm_pair(const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                                                             const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_x,
                                                             const __grid_constant__ PgArgs a) {
    extern __shared__ __align__(1024) uint8_t pg_smem[];
    using T = PgTile<PAIR>;
    constexpr int kPgStages = T::kStages, kPgStageBytes = T::kStageBytes, kPgRows = T::kRows;
    __shared__ uint64_t s_full[kPgStages], s_empty[kPgStages], s_acc_full[2], s_acc_empty[2], s_done, s_peer;
    __shared__ uint32_t s_tmem;
    __shared__ int s_peer_fills, s_consumed;  // first CTA: fills its peer has issued, fills the MMAs have waited for
    uint8_t* const tiles = reinterpret_cast<uint8_t*>(((uintptr_t)pg_smem + 1023) & ~(uintptr_t)1023);
    float* const stage_area = reinterpret_cast<float*>(tiles + (size_t)kPgStages * kPgStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)blockIdx.x & 1 : 0, pair = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, n_pairs = PAIR ? (int)gridDim.x >> 1 : (int)gridDim.x;
    const int n_tiles = a.tiles_n * a.tiles_w, n_units = n_tiles * a.splits, all_kb = a.K / kTcBlockK;  // a unit: one K slice of a tile, slices slowest
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
        for (int i = 0; i < 2; i++) { mbar_init(s_acc_full + i, 1); mbar_init(s_acc_empty + i, (PAIR ? 2 : 1) * kPgEpiWarps); }
        mbar_init(&s_done, 1);
        mbar_init(&s_peer, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) {  // both CTAs' barriers are initialised and their tensor memory is allocated before either is used
        cluster_arrive();
        cluster_wait();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // Weights do not depend on the previous kernel: those of the first stages are requested before the wait for it.
    const CUtensorMap *map0 = &map_w0, *map1 = &map_w0;  // this CTA's weight halves of the unit being loaded (PAIR: the first only)
    int m0 = 0, m1 = 0;
    auto weights_of = [&](int tw) {
        int gi;
        half_of(tw, rank, gi, m0);
        map0 = gi == 0 ? &map_w0 : gi == 1 ? &map_w1 : &map_w2;
        if constexpr (!PAIR) {
            half_of(tw, 1, gi, m1);
            map1 = gi == 0 ? &map_w0 : gi == 1 ? &map_w1 : &map_w2;
        }
    };
    auto load_weights = [&](int k, int s) {
        uint8_t* const sw = tiles + (size_t)s * kPgStageBytes + kPgXBytes;
        if (rank == 0) mbar_expect_tx(s_full + s, (PAIR ? 2 : 1) * kPgStageBytes);
        if constexpr (PAIR) {
            tma_load_pair(sw, map0, k, m0, s_full + s);
        } else {
            tma_load_2d(sw, map0, k, m0, s_full + s);
            tma_load_2d(sw + kPgWBytes, map1, k, m1, s_full + s);
        }
    };
    int ahead = 0;  // fills whose weights have been requested
    if (!PAIR && warp == 0) {
        const int slice = pair / n_tiles, kb0 = slice * a.kb_per_split;
        weights_of((pair - slice * n_tiles) / a.tiles_n);
        ahead = min(kPgStages, min(a.kb_per_split, all_kb - kb0));
        for (int s = 0; s < ahead; s++) {
            if (elect_one()) load_weights((kb0 + s) * kTcBlockK, s);
            __syncwarp();
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tmem = s_tmem;

    if (warp == 0) {
        // ---------------- TMA producer: this CTA's 128 batch rows and its weight halves ----------------
        int s = 0;
        uint32_t phase = 0;
        bool first_round = true, ok = true;
        int fills = 0;
        for (int unit = pair; unit < n_units && ok; unit += n_pairs) {
            const int slice = unit / n_tiles, tile = unit - slice * n_tiles, kb0 = slice * a.kb_per_split, num_kb = min(a.kb_per_split, all_kb - kb0);
            const int tw = tile / a.tiles_n, n0 = (tile - tw * a.tiles_n) * kPgRows + rank * 128;
            weights_of(tw);
            for (int kb = 0; kb < num_kb; kb++) {
                const bool gave_up = !first_round && !tc_wait(s_empty + s, phase ^ 1u, a.error);  // (per lane: the votes below end the loop for all)
                const bool issued = elect_one() && !gave_up;
                if (issued) {
                    const int k = (kb0 + kb) * kTcBlockK;
                    if (PAIR || fills >= ahead) load_weights(k, s);
                    if constexpr (PAIR) tma_load_pair(tiles + (size_t)s * kPgStageBytes, &map_x, k, n0, s_full + s);
                    else tma_load_2d(tiles + (size_t)s * kPgStageBytes, &map_x, k, n0, s_full + s);
                }
                if (__any_sync(0xffffffffu, gave_up)) {
                    fills += __any_sync(0xffffffffu, issued) ? 1 : 0;
                    ok = false;
                    break;
                }
                fills++;
                if (++s == kPgStages) { s = 0; phase ^= 1u; first_round = false; }
            }
        }
        __syncwarp();
        if (rank == 1) {
            if (lane == 0) {
                asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(mapa(smem_u32(&s_peer_fills), 0)), "r"(fills) : "memory");
                arrive_first_cta(&s_peer);
            }
        } else {
            asm volatile("bar.sync 3, 64;" ::: "memory");  // the MMA warp has recorded what it consumed
            if (lane == 0 && (!PAIR || pg_wait_quiet(&s_peer, 0))) {
                const int peer = PAIR ? s_peer_fills : fills;
                if (s_consumed < pg_drain_end(fills, peer)) {  // a wait gave up: copies may be in flight that nobody waited for
#pragma unroll 1
                    for (int f = pg_drain_begin(fills, peer, kPgStages); f < pg_drain_end(fills, peer); f++) {
                        const PgDrainStep d = pg_drain_step(f, fills, peer, kPgStages, kPgStageBytes);
                        if (d.expect) mbar_expect_tx(s_full + d.stage, d.expect);
                        if (d.complete) mbar_complete_tx(s_full + d.stage, d.complete);
                        pg_wait_quiet(s_full + d.stage, d.parity);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer of the pair ----------------
        if (rank == 0) {
            const uint32_t idesc = umma_idesc_f16(T::kRows, 256, a.bf16);
            const uint64_t d_first = umma_smem_desc_sw128(tiles);
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            int it = 0, consumed = 0;
            for (int unit = pair; unit < n_units && ok; unit += n_pairs, it++) {
                const int num_kb = min(a.kb_per_split, all_kb - unit / n_tiles * a.kb_per_split);
                const int buf = it & 1;
                if (it >= 2 && !tc_wait_warp(s_acc_empty + buf, ((it >> 1) - 1) & 1, a.error)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)buf * 256u;
                uint32_t accumulate = 0;
                bool ready = mbar_try_wait(s_full + s, phase);
                for (int kb = 0; kb < num_kb; kb++) {
                    const bool gave_up = !ready && !tc_wait(s_full + s, phase, a.error);  // (per lane: the vote below ends the loop for all)
                    const bool wrap = s + 1 == kPgStages;
                    const int s_next = wrap ? 0 : s + 1;
                    const uint32_t phase_next = phase ^ (wrap ? 1u : 0u);
                    ready = kb + 1 < num_kb && mbar_try_wait(s_full + s_next, phase_next);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one() && !gave_up) {
                        const uint64_t da = d_first + (uint64_t)(s * (kPgStageBytes >> 4)), db = da + (kPgXBytes >> 4);
                        pg_mma<PAIR>(acc, da, db, idesc, accumulate);
#pragma unroll
                        for (int k = 1; k < kTcBlockK / 16; k++) pg_mma<PAIR>(acc, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, 1u);
                        pg_commit<PAIR>(s_empty + s);
                    }
                    if (__any_sync(0xffffffffu, gave_up)) { ok = false; break; }
                    accumulate = 1;
                    consumed++;
                    s = s_next;
                    phase = phase_next;
                }
                if (ok && elect_one()) pg_commit<PAIR>(s_acc_full + buf);
                __syncwarp();
            }
            __syncwarp();
            if (lane == 0) s_consumed = consumed;
            if (elect_one()) pg_commit<PAIR>(&s_done);
            __syncwarp();
            asm volatile("bar.sync 3, 64;" ::: "memory");
        }
        if (lane == 0) pg_wait_quiet(&s_done, 0);  // every MMA of the pair has read its operands, every commit before has arrived
    } else {
        // ---------------- epilogue: TMEM -> registers -> staging -> global ----------------
        const int ew = warp - 2, quad = warp & 3, sub = ew >> 2;  // lanes 32 * quad.. of TMEM; which quarter of the columns
        PgWarp w{};
        w.stg = stage_area + (size_t)ew * 32 * 16;
        w.lane = lane; w.sub = sub;
        int it = 0;
        for (int unit = pair; unit < n_units; unit += n_pairs, it++) {
            const int buf = it & 1, slice = unit / n_tiles, tile = unit - slice * n_tiles;
            const int tw = tile / a.tiles_n;
            w.nrow0 = (tile - tw * a.tiles_n) * kPgRows + rank * 128 + 32 * quad;
            const int row = w.nrow0 + lane;
            w.live = __ballot_sync(0xffffffffu, row < a.rows && (!a.active || __ldcg(a.active + row)));
            w.first_slice = slice == 0;
            if (a.epilogue == PG_QKV && row < a.rows) {
                w.pos = __ldcg(a.rs.pos + row);
                w.kv_row = a.kv.offset(a.m, a.layer, __ldcg(a.rs.seq + row), 0, w.pos);
            }
            if (!tc_wait_warp(s_acc_full + buf, (it >> 1) & 1, a.error)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            w.base = tmem + (uint32_t)buf * 256u + ((uint32_t)(32 * quad) << 16);
            if (w.live) {
                if (a.epilogue == PG_STORE) pg_epilogue<PG_STORE>(a, w, tw, half_of);
                else if (a.epilogue == PG_RESIDUAL) pg_epilogue<PG_RESIDUAL>(a, w, tw, half_of);
                else if (a.epilogue == PG_QKV) pg_epilogue<PG_QKV>(a, w, tw, half_of);
                else if (a.epilogue == PG_GELU) pg_epilogue<PG_GELU>(a, w, tw, half_of);
                else pg_epilogue<PG_SWIGLU>(a, w, tw, half_of);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) {
                if constexpr (PAIR) arrive_first_cta(s_acc_empty + buf);
                else mbar_arrive(s_acc_empty + buf);
            }
        }
    }
    // nobody leaves while the pair's copies, commits or arrivals may still reach this CTA
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (PAIR) {
        cluster_arrive();
        cluster_wait();
    }
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace esp
