// Persistent whole-loop decode kernel for one sequence of a Llama-style fp16 model.
//
// One cooperative launch runs an entire greedy decode loop: `n_steps` heads and up to `n_steps - 1` forward
// passes.  The grid has one CTA per SM.  Inside a CTA one producer warp streams that CTA's weights from HBM into a
// shared-memory ring with bulk async copies (cp.async.bulk + mbarrier), always running ahead of the eight
// consumer warps (a watcher warp turns the copies' completions into a counter the consumers can read cheaply), so HBM keeps streaming while the consumers wait on the activation dependencies of the step.
// Weights are re-laid out once ("pack") so that everything a CTA needs for one layer is contiguous.
//
// Batch-1 decode is bound by the chain of dependent vector exchanges between CTAs, not by bytes, so the kernel has
// no grid barrier at all.  Every vector that crosses CTAs is self-validating:
//   * "tagged words": an 8-byte word {fp32 value, 32-bit sequence tag} with a single writer.  A reader polls the
//     word itself until the tag is the one it expects: flag and data travel in one 8-byte access, so neither a
//     fence nor a separate arrival counter nor a second round trip for the data is needed.
//   * "counted sums": an 8-byte accumulator that several CTAs add into with one `red.add.u64` each; the addend is
//     (fixed-point value << 8) + 1, so the low byte counts contributions and the upper 56 bits carry their sum.
//     The accumulators are never cleared: a reader remembers the total it saw the last time and subtracts it
//     (all arithmetic is modulo 2^64, so neither field can overflow into a wrong result as long as one exchange's
//     sum fits 55 bits).  Integer addition is associative: the sums are bit-identical from run to run.
// Per layer the consumers run
//   S1  x (tagged words from the previous layer, or the embedding row) -> RMSNorm folded into the products ->
//       this CTA's rows of Wq/Wk/Wv -> RoPE -> tagged words for the CTAs that share the KV head, KV-cache append
//   S2  attention of one query head (recomputed by the CTAs that share the head) -> this CTA's block of rows of Wo
//       restricted to the head's columns -> counted sums (one contribution per head and row)
//   S3  x_mid -> norm -> this CTA's (gate, up) row pairs -> SiLU*up -> tagged words; then the whole activation
//       vector -> this CTA's rows of W2 (+ residual) -> tagged words = the next layer's x
// and the LM head streams the CTA's vocabulary rows through the same ring; every CTA publishes its best
// (logit, index) as tagged words and every CTA reduces all of them, so the token is known everywhere at once.
// Inside a CTA the columns of a stage's operand belong to the warps (MegaWorker): a warp awaits, stages and multiplies its own.
// Products.  The fp16->fp32 conversion rate of the CUDA cores (measured: 20-26 weights per clock per SM from shared
// memory) would make the row products the longest link of the chain, so they are issued as m16n8k16 tensor-core
// instructions: sixteen weight rows are the A operand, and the fp32 activation vector, split into two fp16 vectors (x = hi + lo,
// off by at most 2^-22 |x|, or 2^-25 where the low part is subnormal; |x| up to 65504), occupies columns 0 and 1 of the B operand; the
// accumulators are fp32.  The pack stores every chunk in the order the A fragments are read.
// GGUF Q8_0 / Q4_0 matrices travel through the ring as their blocks (32 or 16 bytes per row and block of 32 columns,
// the fp16 scales behind them): 34/32 or 18/32 bytes per weight from HBM, never an fp16 copy; the activation becomes int8
// digits (qx_store_quads) and a block one int8 m16n8k32 step, scaled in fp32 (value = fp32(d) * q as in the GGUF definition).
// A warp's time per 16-row tile and block with the weights in shared memory was 40 cycles per scheduler for Q8_0 and 56 for Q4_0
// nibbles widened to fp16, most of it shared-memory wavefronts (one per scale) and conversions; hence the nibbles as int8.
//
// us per token (16 warps that staged and synchronised together, multiplying row tiles -> this): 6 layers d768 fp16 77.6 -> 61,
// GPT-2 117M 169.5 -> 135, 22 layers d2048 Q8_0 482 -> 361, Q4_0 477 -> 376.
// Every wait (mbarrier, tagged word, counted sum) is bounded: when a limit is hit the kernel records an error code,
// stops waiting everywhere and runs to completion; the host reports a timeout.
#pragma once
#include <algorithm>

#include "decode_kernels.cuh"
#include "mega_units.h"

namespace esp {

constexpr int kMegaConsumerWarps = 8;
constexpr int kMegaConsumers = kMegaConsumerWarps * 32;
constexpr int kMegaThreads = kMegaConsumers + 64;  // + the producer warp and the watcher warp
constexpr unsigned kMegaSpinLimit = 1u << 21;      // default attempts per wait before the kernel gives up (a few seconds)
constexpr int kMegaTraceLayer = 10;                // stamps per layer
constexpr int kMegaTraceHead = 4;                  // stamps of the head
constexpr int kMegaSlots = 4, kMegaSlotMax = 64 * 1024;  // ring slots and the most bytes of one (Q8_0, 22 layers of d2048: 4 slots of 44 KB 371 us per token, 5 of 35 KB 395, 7 of 25 KB 447)
constexpr int kMegaRingMin = 96 * 1024;  // less than that is consumed faster than a refill takes to arrive
constexpr int kMegaMaxTiles = 5;                   // 16-row tiles whose sums a warp keeps in registers
// Which exchanges give every CTA cache lines of its own is the plan's choice (act_wpc > 0).
// The arg-max candidates always have them (-4.6 us per token of the 6-layer d768 model against a compact array), the layer output x
// never (+0.3 us: five words per CTA, three times as many lines to poll for little contention saved).  The activation vector has them
// up to the width that a lane polls in one round.  us per token of six fp16 layers, lines / compact: d256 hidden 1280 54.7 / 60.5, d512
// 512 53.7 / 56.5, 1408 57.2 / 58.3, GPT-2 d384 1536 65.6 / 67.9; d512 2048 57.9 / 58.7, d768 2048 60.7 / 60.0; wider, where the padding only
// adds lines to poll: d768 3072 68.9 / 68.3, 4096 77.0 / 74.0, d1024 4096 81.8 / 80.1, d1536 4096 117.1 / 115.6, GPT-2 d768 3072 73.4 / 72.6.
constexpr int kMegaLinesMost = 2048;
constexpr int kMegaLineWords = 16;  // 8-byte words of a 128-byte cache line
constexpr int kMegaCandStride = kMegaLineWords;  // 8-byte words between the arg-max candidates of two CTAs: a cache line each
constexpr float kMegaFix = 4294967296.0f;          // counted sums: fixed point with 32 fractional bits
constexpr float kMegaUnfix = 2.3283064365386963e-10f;

// Stages in the order a CTA takes them: q/k/v rows, rows of Wo (one head's columns), (gate, up) rows, rows of W2, vocabulary rows.
enum MegaStageKind { MS_QKV = 0, MS_WO = 1, MS_UP = 2, MS_DOWN = 3, MS_HEAD = 4 };
struct MegaStage {
    int units;       // K units: 16 columns (fp16) or one block of 32 columns (quantised types)
    int group_rows;  // rows of a chunk; except for Wo also the rows whose products run side by side (at most 16 kMegaMaxTiles)
    int chunk_units; // consecutive units of a group's rows per chunk
};

struct MegaPlan {
    float inv_d;      // 1 / d_model
    int n_cta;
    int cph;          // CTAs per query head (S2 row blocks of Wo)
    int qpk;          // query heads per KV head
    int gsize;        // CTAs per KV-head group = cph * qpk
    int n_group_cta;  // CTAs that take part in S1/S2 = n_head * cph
    int group_items;  // S1 row pairs per KV-head group = (qpk + 2) * head_dim / 2
    int s1_max;       // largest number of S1 row pairs of a CTA
    int rpb;          // S2: output rows per block
    int hpc_max, dpc_max, vpc_max;  // largest number of FFN units / W2 rows / vocabulary rows of a CTA
    int act_wpc;  // exchange words reserved per CTA for its elements of the activation vector (whole cache lines); 0 = compact array
    int wt_layer, wt_head;  // storage type of the layer matrices and of the LM head: WT_F16, WT_Q8_0 or WT_Q4_0
    int ffn_rows;     // packed rows per FFN unit: (gate, up) pairs 2, GPT-2's single up projection 1
    MegaStage stage[5];  // by MegaStageKind
    int group_tiles;  // 16-row tiles of the largest group (partial sums are laid out for them)
    int s1_bytes, s2_bytes, s3a_bytes, s3b_bytes;  // packed bytes of a stage per layer (multiples of 128, sized for the largest CTA share)
    int slot_bytes, n_slots;
    long long layer_bytes, head_bytes, cta_bytes;  // packed bytes per CTA: one layer, the head, everything
    int smem_bytes;
    // byte offsets of the shared-memory areas behind the ring (see MegaShared)
    int off_bar, off_prev, off_key, off_xs, off_xq, off_xres, off_qs, off_ctx, off_kn, off_vn, off_part, off_red, off_ss, off_sums, off_flags, off_share, off_act, off_s1;
};

// K units of a storage type, and the packed bytes of one unit of `rows` rows: fp16 columns, or GGUF blocks (int8 / nibbles) and
// one fp16 scale per row, the scales for whole tiles of sixteen rows.
__host__ __device__ constexpr int mega_unit(int wt) { return wt == WT_F16 ? 16 : 32; }
__host__ __device__ inline int mega_scale_bytes(int wt, int rows) { return wt == WT_F16 ? 0 : (rows + 15) / 16 * 32; }
__host__ __device__ inline int mega_data_bytes(int wt, int rows) { return rows * (wt == WT_Q4_0 ? 16 : 32); }
__host__ __device__ inline int mega_unit_bytes(int wt, int rows) { return mega_data_bytes(wt, rows) + mega_scale_bytes(wt, rows); }
// Packed bytes of `rows` rows of a stage (every group but the last one is full).
__host__ __device__ inline long long mega_stage_bytes(const MegaStage& st, int wt, int rows) {
    const int full = rows / st.group_rows, rest = rows - full * st.group_rows;
    return (long long)st.units * ((long long)full * mega_unit_bytes(wt, st.group_rows) + (rest ? mega_unit_bytes(wt, rest) : 0));
}
__host__ __device__ inline int mega_stage_chunks(const MegaStage& st, int rows) {
    return (rows + st.group_rows - 1) / st.group_rows * ((st.units + st.chunk_units - 1) / st.chunk_units);
}

// Contiguous share [begin, end) of `n` items owned by part `i` of `parts` (every part gets floor or ceil of n/parts).
// (n * parts stays far below 2^32 for every model size the plan accepts)
__host__ __device__ inline int mega_share_begin(int n, int parts, int i) { return (int)((unsigned)n * (unsigned)i / (unsigned)parts); }

struct MegaArgs {
    ModelDims m;
    MegaPlan plan;
    const uint8_t* pack;      // [n_cta][cta_bytes]
    const float* norms;       // [2*L + 1][d_model]: norm1(l), norm2(l), ..., final
    const uint16_t* tok_emb;  // fp16 [vocab][d_model]
    // GPT-2 only.  The products run on the centred rows (x - mean) g; a row's result is inv sum + (W.b + bias), and the
    // constant of every row is computed once.
    const uint16_t* pos_emb;  // fp16 [max_seq][d_model]
    const float* ln;          // per layer [q_dim + 2 kv_dim + hidden], then [vocab] for the head: W.b + bias
    const float* out_bias;    // per layer [bias of Wo, bias of W2], d_model each
    const float2* rope;       // [max_seq][head_dim/2]
    KvLayout kv;
    // exchange arena (zero before the first launch; tags keep launches apart, the counted sums are zeroed at the end)
    unsigned long long* x_words;    // [d_model] tagged: output of a layer
    unsigned long long* act_words;  // [hidden] or [n_cta][act_wpc]; tagged: FFN activation
    unsigned long long* qkv_words;  // [n_kv_head][2 * group_items] tagged: post-RoPE q / k / v of one token
    unsigned long long* mid_sums;   // [d_model] counted: residual + attention projection
    unsigned long long* cand_words; // [n_cta][kMegaCandStride] {logit bits, index, 8-bit tag} of each CTA's best row in word 0, {request, 8-bit tag} in word 1
    float* hidden_io;         // [d_model] last hidden state of the sequence (in and out)
    int* error;               // [1] 0 = ok
    unsigned long long* stamps; // [4] globaltimer at kernel start and when the first token is known; {last token : 32}{number of tokens emitted : 32}; visible tokens
    unsigned long long* host_words;  // optional pinned host memory [n_steps]: {number of tokens emitted : 32}{token : 32} of every token as it becomes known, or null
    const unsigned* stop_request;    // optional pinned host word: not zero = the loop ends after the token at hand, or null
    unsigned long long* token_times; // optional [n_steps] globaltimer (ns) at which each token became known, or null
    long long* trace;         // optional [kMegaTraceLayer*L + kMegaTraceHead] SM clock stamps of the last step taken by CTA `trace_cta`, or null
    int trace_cta;
    RowState rs;              // row 0 carries pos / tok / n_out / out
    int n_steps;              // tokens to emit at most (>= 1)
    int first;                // 0: the loop starts with the head (the state holds the last hidden vector); 1: with a forward pass for `tok0`
    uint32_t tok0;
    unsigned tag0;            // added to every sequence tag, and cand0 to the candidates' step count: the arena is never cleared
    unsigned cand0;           // between launches, so the words of earlier launches must not look like this one's
    int pos0;                 // visible tokens at launch
    unsigned spin_limit;      // attempts per wait
};

// ------------------------------------------------------------------------------------------------ PTX helpers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Non-blocking test of a phase: the potentially blocking try_wait form costs about 0.25 us per call on this part even
// when the phase has already completed, which a chunk-by-chunk consumer cannot afford.
__device__ __forceinline__ bool mbar_test(uint32_t bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) { return mbar_test(smem_u32(bar), parity); }
// Weight chunks carry an evict-first L2 policy: they are used once per token, and keeping them out of the way
// leaves the KV cache and the exchange words resident in L2.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kMegaConsumers) : "memory"); }

// 16 bytes = two exchange words; each word is validated on its own, so the pair needs no 16-byte atomicity.
__device__ __forceinline__ ulonglong2 ld_words2(const unsigned long long* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_words2(unsigned long long* p, unsigned long long v0, unsigned long long v1) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(v0), "l"(v1) : "memory");
}
__device__ __forceinline__ void red_add_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long tagged(float v, unsigned tag) { return ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v); }
__device__ __forceinline__ unsigned long long counted(float v) { return ((unsigned long long)__float2ll_rn(v * kMegaFix) << 8) + 1ull; }

// ------------------------------------------------------------------------------------------------ work shares

struct MegaShare {
    bool in_group;       // takes part in S1 / S2
    int head, blk, kvh, hq, member;  // query head, Wo row block, KV head, head inside the KV group, CTA inside the KV group
    int s1_begin, s1_n;  // S1 row pairs inside the KV group
    int h_begin, h_n;    // FFN hidden units
    int d_begin, d_n;    // W2 rows
    int v_begin, v_n;    // vocabulary rows
};

__host__ __device__ inline MegaShare mega_share(const ModelDims& m, const MegaPlan& p, int cta) {
    MegaShare w{};
    w.in_group = cta < p.n_group_cta;
    if (w.in_group) {
        w.head = cta / p.cph;
        w.blk = cta - w.head * p.cph;
        w.kvh = w.head / p.qpk;
        w.hq = w.head - w.kvh * p.qpk;
        w.member = cta - w.kvh * p.gsize;
        w.s1_begin = mega_share_begin(p.group_items, p.gsize, w.member);
        w.s1_n = mega_share_begin(p.group_items, p.gsize, w.member + 1) - w.s1_begin;
    }
    w.h_begin = 2 * mega_share_begin(m.hidden / 2, p.n_cta, cta);  // (whole pairs: a reader takes two words at a time)
    w.h_n = 2 * mega_share_begin(m.hidden / 2, p.n_cta, cta + 1) - w.h_begin;
    w.d_begin = mega_share_begin(m.d_model, p.n_cta, cta);
    w.d_n = mega_share_begin(m.d_model, p.n_cta, cta + 1) - w.d_begin;
    w.v_begin = mega_share_begin(m.vocab, p.n_cta, cta);
    w.v_n = mega_share_begin(m.vocab, p.n_cta, cta + 1) - w.v_begin;
    return w;
}

// S1 row pair `item` of KV group `kvh`: which matrix (0 q, 1 k, 2 v) and which two rows.
__host__ __device__ inline void mega_s1_rows(const ModelDims& m, const MegaPlan& p, int kvh, int item, int& kind, int& row0, int& row1, int& idx) {
    const int half = m.head_dim / 2, lg_half = m.head_dim == 32 ? 4 : m.head_dim == 64 ? 5 : 6;  // head_dim is 32, 64 or 128
    if (item < p.qpk * half) {
        const int hq = item >> lg_half;
        idx = item - hq * half;
        kind = 0; row0 = (kvh * p.qpk + hq) * m.head_dim + idx; row1 = row0 + half;
    } else if (item < (p.qpk + 1) * half) {
        idx = item - p.qpk * half;
        kind = 1; row0 = kvh * m.head_dim + idx; row1 = row0 + half;
    } else {
        idx = item - (p.qpk + 1) * half;
        kind = 2; row0 = kvh * m.head_dim + 2 * idx; row1 = row0 + 1;
    }
}

// Bytes of a staged vector of K values for np positions: fp16 hi and lo parts (xa_index), or int8 digits (qx_store_quads).
__host__ __device__ constexpr int qx_digits(int wt) { return wt == WT_Q4_0 ? 4 : 3; }
__host__ __device__ constexpr int xa_bytes(int wt, int K, int np) { return wt == WT_F16 ? K / 16 * 64 * np : K / 32 * 32 * qx_digits(wt); }

// ------------------------------------------------------------------------------------------------ shared state

struct MegaShared {
    uint8_t* slots;
    uint64_t* full;
    uint64_t* empty;
    uint8_t* xa;   // staged operand vector, every unit written and read by the warp that owns it
    float* xq;     // quantised types: scale of every staged block
    float* xres;   // [np][d_model] the residual stream: entering the layer, then after the attention block
    unsigned long long* prev;  // [np][d_model] totals of the counted sums seen at the previous exchange
    float* qs;     // [np][head_dim] query of this CTA's head
    uint8_t* ctx;  // attention output of this CTA's head, staged like xa (block scales behind it)
    __half* kn;    // [np][head_dim] the new token's key, rounded as the cache stores it
    __half* vn;    // [np][head_dim]
    float* part;   // [warps][head_dim]
    float* red;    // [64]
    float* ss;     // [2][np][warps] sums of squares of the warps' columns (alternating with the partial sums)
    float* sums;   // [2][warps][np][16 group_tiles] partial row sums of a group
    unsigned long long* key;   // [32] arg-max keys
    struct MegaShare* share;  // this CTA's work shares, computed once
    uint16_t* act;  // [hidden / 2] word of every pair of the activation vector (act_wpc > 0)
    int4* s1;       // [s1_max] {kind, row, row, RoPE entry} of this CTA's S1 row pairs
    int* abort;    // [1] a wait gave up: no more waiting in this CTA
    int* stop;     // [1] the loop ended early (EOS): the producer stops issuing
    unsigned* landed;  // [1] number of chunks whose bytes have arrived (written by the watcher warp)
    unsigned* asked;   // [1] CTA 0: the host wants the loop to end (written by the producer warp)
};

// The areas sit at offsets the host computed once (mega_layout): an address is the base plus a kernel-argument
// constant, which costs no register to keep.
__device__ __forceinline__ MegaShared mega_carve(uint8_t* base, const MegaPlan& p) {
    MegaShared s;
    s.slots = base;
    s.full = reinterpret_cast<uint64_t*>(base + p.off_bar);
    s.empty = s.full + p.n_slots;
    s.prev = reinterpret_cast<unsigned long long*>(base + p.off_prev);
    s.key = reinterpret_cast<unsigned long long*>(base + p.off_key);
    s.xa = base + p.off_xs;
    s.xq = reinterpret_cast<float*>(base + p.off_xq);
    s.xres = reinterpret_cast<float*>(base + p.off_xres);
    s.qs = reinterpret_cast<float*>(base + p.off_qs);
    s.ctx = base + p.off_ctx;
    s.kn = reinterpret_cast<__half*>(base + p.off_kn);
    s.vn = reinterpret_cast<__half*>(base + p.off_vn);
    s.part = reinterpret_cast<float*>(base + p.off_part);
    s.red = reinterpret_cast<float*>(base + p.off_red);
    s.ss = reinterpret_cast<float*>(base + p.off_ss);
    s.sums = reinterpret_cast<float*>(base + p.off_sums);
    s.abort = reinterpret_cast<int*>(base + p.off_flags);
    s.stop = s.abort + 1;
    s.landed = reinterpret_cast<unsigned*>(s.abort + 2);
    s.asked = s.landed + 1;
    s.share = reinterpret_cast<MegaShare*>(base + p.off_share);
    s.act = reinterpret_cast<uint16_t*>(base + p.off_act);
    s.s1 = reinterpret_cast<int4*>(base + p.off_s1);
    return s;
}

// Fills the offsets and the total size for np token positions per pass (host side; p.n_slots and p.slot_bytes must be set).
inline void mega_layout(const ModelDims& m, MegaPlan& p, int np) {
    const int wide = m.d_model > m.hidden ? m.d_model : m.hidden;
    size_t o = (size_t)p.n_slots * p.slot_bytes;
    auto take = [&](size_t bytes) { size_t at = (o + 15) & ~(size_t)15; o = at + bytes; return (int)at; };
    auto staged = [&](int K) { return (size_t)xa_bytes(p.wt_layer, K, np); };
    const size_t xs = std::max(staged(wide), (size_t)xa_bytes(p.wt_head, m.d_model, np));
    p.off_bar = take(16 * (size_t)p.n_slots);
    p.off_prev = take(8 * (size_t)np * m.d_model);
    p.off_key = take(8 * 32);
    p.off_xs = take(xs);
    p.off_xq = take(p.wt_layer == WT_F16 ? 0 : sizeof(float) * (size_t)(wide / 32));
    p.off_xres = take(sizeof(float) * (size_t)np * m.d_model);
    p.off_qs = take(sizeof(float) * (size_t)np * m.head_dim);
    p.off_ctx = take(staged(m.head_dim) + sizeof(float) * (size_t)(m.head_dim / 32));
    p.off_kn = take(sizeof(__half) * (size_t)np * m.head_dim);
    p.off_vn = take(sizeof(__half) * (size_t)np * m.head_dim);
    p.off_part = take(sizeof(float) * (size_t)kMegaConsumerWarps * m.head_dim);
    p.off_red = take(sizeof(float) * 64);
    p.off_ss = take(sizeof(float) * 2 * (size_t)np * kMegaConsumerWarps);
    p.off_sums = take(sizeof(float) * 2 * (size_t)kMegaConsumerWarps * np * 16 * p.group_tiles);
    p.off_flags = take(16);
    p.off_share = take(sizeof(MegaShare));
    p.off_act = take(p.act_wpc ? sizeof(uint16_t) * (size_t)(m.hidden / 2) : 0);
    p.off_s1 = take(sizeof(int4) * (size_t)p.s1_max);
    p.smem_bytes = (int)((o + 127) & ~(size_t)127);
}

// Plans the persistent kernel for a model (host side): every CTA owns a contiguous share of the rows of every matrix.  False: the
// model does not fit.
inline bool mega_plan(const ModelDims& m, int wt_layer, int wt_head, int sms, int smem_max, MegaPlan& p) {
    p = MegaPlan{};
    const bool quant = wt_layer != WT_F16 || wt_head != WT_F16;
    if (quant && (m.d_model % 256 || m.hidden % 256)) return false;
    // every CTA must own at least one pair of FFN units and one row of W2 (it then takes part in every all-to-all exchange)
    const int P = std::min(sms, std::min(m.d_model, m.hidden / 2));
    if (P < m.n_head) return false;
    auto pad128 = [](long long v) { return (int)((v + 127) / 128 * 128); };
    auto ceil_div = [](int a, int b) { return (a + b - 1) / b; };
    p.inv_d = 1.0f / (float)m.d_model;
    p.n_cta = P;
    p.qpk = m.n_head / m.n_kv_head;
    p.group_items = (p.qpk + 2) * m.head_dim / 2;
    p.cph = std::max(1, std::min(std::min(P / m.n_head, m.d_model), p.group_items / p.qpk));
    p.gsize = p.cph * p.qpk;
    p.n_group_cta = p.cph * m.n_head;
    p.s1_max = ceil_div(p.group_items, p.gsize);
    p.rpb = ceil_div(m.d_model, p.cph);
    p.hpc_max = 2 * ceil_div(m.hidden / 2, P);
    p.dpc_max = ceil_div(m.d_model, P);
    p.vpc_max = ceil_div(m.vocab, P);
    p.wt_layer = wt_layer;
    p.wt_head = wt_head;
    p.ffn_rows = m.arch == ARCH_GPT2 ? 1 : 2;
    // Exchange arrays: the activation vector gets cache lines per CTA where a lane polls all of its pairs in one round (see
    // kMegaLinesMost; two positions share one round of twice as many loads); the layer output stays compact.
    p.act_wpc = !quant && m.hidden <= kMegaLinesMost ? ceil_div(p.hpc_max, kMegaLineWords) * kMegaLineWords : 0;
    // Row groups: as equal as whole tiles allow.
    const int rows[5] = {2 * p.s1_max, p.rpb, p.ffn_rows * p.hpc_max, p.dpc_max, p.vpc_max};
    for (int k = 0; k < 5; k++) {
        MegaStage& st = p.stage[k];
        st.units = (k == MS_WO ? m.head_dim : k == MS_DOWN ? m.hidden : m.d_model) / mega_unit(k == MS_HEAD ? wt_head : wt_layer);
        st.chunk_units = st.units;
        st.group_rows = rows[k];
        if (k == MS_WO) continue;
        const int groups = ceil_div(rows[k], 16 * kMegaMaxTiles);
        if (groups > 1) st.group_rows = ceil_div(ceil_div(rows[k], groups), 16) * 16;
        p.group_tiles = std::max(p.group_tiles, ceil_div(st.group_rows, 16));
    }
    // The ring: what the other areas leave, in kMegaSlots slots, and as many units of a group (for Wo: 16-row tiles) per chunk as
    // fit one, in equal shares.
    mega_layout(m, p, 1);
    const int room = smem_max - p.smem_bytes - 512;
    for (int ns = kMegaSlots; ns >= 2 && p.n_slots == 0; ns--) {
        const int slot = std::min(room / ns / 128 * 128, kMegaSlotMax);
        if (ns * slot < kMegaRingMin) continue;
        bool fits = true;
        for (int k = 0; k < 5; k++) {
            MegaStage& st = p.stage[k];
            const int wt = k == MS_HEAD ? wt_head : wt_layer;
            if (k == MS_WO) {
                int per = rows[k];
                for (int n = 2; per > 16 && st.units * mega_unit_bytes(wt, per) > slot; n++) per = ceil_div(ceil_div(rows[k], n), 16) * 16;
                st.group_rows = per;
                fits = fits && st.units * mega_unit_bytes(wt, per) <= slot;
            } else {
                const int most = slot / mega_unit_bytes(wt, st.group_rows);
                fits = fits && most >= 1;
                if (most >= 1) st.chunk_units = ceil_div(st.units, ceil_div(st.units, most));
            }
        }
        if (fits) { p.n_slots = ns; p.slot_bytes = slot; }
    }
    if (p.n_slots == 0) return false;
    mega_layout(m, p, 1);
    if (p.smem_bytes > smem_max) return false;
    p.s1_bytes = pad128(mega_stage_bytes(p.stage[MS_QKV], wt_layer, rows[MS_QKV]));
    p.s2_bytes = pad128(mega_stage_bytes(p.stage[MS_WO], wt_layer, rows[MS_WO]));
    p.s3a_bytes = pad128(mega_stage_bytes(p.stage[MS_UP], wt_layer, rows[MS_UP]));
    p.s3b_bytes = pad128(mega_stage_bytes(p.stage[MS_DOWN], wt_layer, rows[MS_DOWN]));
    p.layer_bytes = (long long)p.s1_bytes + p.s2_bytes + p.s3a_bytes + p.s3b_bytes;
    p.head_bytes = pad128(mega_stage_bytes(p.stage[MS_HEAD], wt_head, rows[MS_HEAD]));
    p.cta_bytes = p.layer_bytes * m.n_layer + p.head_bytes;
    return true;
}

// Shared state before the roles part (all threads of the CTA; the caller synchronises).
__device__ __forceinline__ void mega_init(const MegaArgs& a, const MegaShared& s, int np) {
    const ModelDims& m = a.m;
    const MegaPlan& p = a.plan;
    const int tid = threadIdx.x;
    if (tid == 0) {
        *s.share = mega_share(m, p, (int)blockIdx.x);
        for (int i = 0; i < p.n_slots; i++) { mbar_init(s.full + i, 1); mbar_init(s.empty + i, kMegaConsumerWarps); }
        *s.abort = 0;
        *s.stop = 0;
        *s.landed = 0u;
        *s.asked = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int k = tid; k < np * m.d_model; k += kMegaThreads) s.prev[k] = 0ull;  // the counted sums are zero at launch
    if (p.act_wpc)
        for (int c = tid; c < p.n_cta; c += kMegaThreads) {
            const int b = mega_share_begin(m.hidden / 2, p.n_cta, c), e = mega_share_begin(m.hidden / 2, p.n_cta, c + 1);
            for (int i = b; i < e; i++) s.act[i] = (uint16_t)(c * p.act_wpc + 2 * (i - b));
        }
    if ((int)blockIdx.x < p.n_group_cta) {
        const MegaShare w = mega_share(m, p, (int)blockIdx.x);
        for (int i = tid; i < w.s1_n; i += kMegaThreads) {
            int4 e;
            mega_s1_rows(m, p, w.kvh, w.s1_begin + i, e.x, e.y, e.z, e.w);
            s.s1[i] = e;
        }
    }
}

__device__ __forceinline__ void mega_fail(const MegaArgs& a, const MegaShared& s, int code) {
    *reinterpret_cast<volatile int*>(s.abort) = 1;
    atomicCAS(a.error, 0, code);
}
__device__ __forceinline__ bool mega_aborting(const MegaShared& s) { return *reinterpret_cast<volatile int*>(s.abort) != 0; }

// One failed attempt of a polling loop: true when the loop must give up (limit reached, or the kernel is aborting).  Polls of global
// memory go out back to back: a pause of 50 ns between them makes a token of the 6-layer d768 model 74 us instead of 64.
__device__ __forceinline__ bool mega_spin_out(const MegaArgs& a, const MegaShared& s, unsigned& spins, int code) {
    ++spins;
    if (spins > a.spin_limit) { mega_fail(a, s, code); return true; }
    if ((spins & 0x3ffu) == 0 && (__ldcg(a.error) != 0 || mega_aborting(s))) { *reinterpret_cast<volatile int*>(s.abort) = 1; return true; }
    return false;
}

// Bounded wait on an mbarrier phase.  Returns immediately once the kernel is aborting.
__device__ __forceinline__ void mega_wait(const MegaArgs& a, const MegaShared& s, uint64_t* bar, unsigned parity, int code) {
    if (mega_aborting(s)) return;
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (*reinterpret_cast<volatile int*>(s.stop)) return;
        if (mega_spin_out(a, s, spins, code)) return;
    }
}

// Ring bookkeeping shared by the producer and the consumers: chunk c lives in slot c % n_slots and completes phase
// (c / n_slots) & 1 of that slot's barriers.  Kept incrementally: a division by a run-time value on the critical path
// of every chunk costs a lone thread a quarter of a microsecond.
struct MegaCursor {
    unsigned slot = 0, phase = 0;
    __device__ __forceinline__ void next(unsigned n_slots) {
        if (++slot == n_slots) { slot = 0; phase ^= 1u; }
    }
};

// A consumer does not test the slot's mbarrier itself: that test costs ~280 cycles per call on this part even when the
// phase completed long ago.  The watcher warp (one thread) follows the chunks in order, waits on each barrier and
// publishes the count of landed chunks in a plain shared-memory word (release), which the consumers read (acquire).
__device__ __forceinline__ unsigned ld_acquire_cta_shared(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta_shared(unsigned* p, unsigned v) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
// `landed` is the count the warp read last: the ring runs ahead, so most chunks are known to be there without a read
// (the read and the warp barrier behind it took 3 % of the token time of the quantised models).  It is the same in every lane:
// lane 0 polls and hands its count to the others, so that a wait which gives up leaves the warp together, whatever each
// lane would have seen of the count and of the abort flag.  The shuffle and the barrier order the lanes' reads of the chunk.
__device__ __forceinline__ const uint8_t* mega_acquire(const MegaArgs& a, const MegaShared& s, const MegaCursor& c, unsigned index, unsigned& landed) {
    if ((int)(landed - index) <= 0) {
        if ((threadIdx.x & 31) == 0) {
            unsigned spins = 0;
            while ((int)((landed = ld_acquire_cta_shared(s.landed)) - index) <= 0) {
                if (mega_aborting(s) || mega_spin_out(a, s, spins, 3)) break;
            }
        }
        __syncwarp();
        landed = __shfl_sync(0xffffffffu, landed, 0);
    }
    return s.slots + (size_t)c.slot * a.plan.slot_bytes;
}
__device__ __forceinline__ void mega_release(const MegaArgs& a, const MegaShared& s, MegaCursor& c) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(s.empty + c.slot);
    c.next((unsigned)a.plan.n_slots);
}
// Hands back `n` consecutive slots starting at `from` whose release was put off (see the kernel's group_products).
__device__ __forceinline__ void mega_release_deferred(const MegaArgs& a, const MegaShared& s, MegaCursor from, int n) {
    __syncwarp();
    for (int i = 0; i < n; i++) {
        if ((threadIdx.x & 31) == 0) mbar_arrive(s.empty + from.slot);
        from.next((unsigned)a.plan.n_slots);
    }
}

// ------------------------------------------------------------------------------------------------ staged operands

// Where element k of a staged fp16 vector lives (in halves): unit of 16 columns, column c of the B operand (position q's
// hi part is column 2q, its lo part column 2q + 1; NP positions are staged side by side), piece t; the 8 bytes of a piece
// are the B registers of the unit's m16n8k16 step.
template <int NP>
__device__ __forceinline__ int xa_index(int k, int c) {
    return (((k >> 4) * 2 * NP + c) * 4 + ((k & 7) >> 1)) * 4 + ((k >> 3) & 1) * 2 + (k & 1);
}
// hi saturates: it stays finite on any finite value
__device__ __forceinline__ uint32_t xa_hi(float v) {
    unsigned short h;
    asm("cvt.rn.satfinite.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
    return h;
}
// Stores elements k, k + 1 (k even) of position q as hi + lo fp16 parts.
template <int NP>
__device__ __forceinline__ void xa_store_pair(uint8_t* xa, int k, float v0, float v1, int q) {
    const uint32_t h0 = xa_hi(v0), h1 = xa_hi(v1);
    const __half2 lo = __floats2half2_rn(v0 - __half2float(__ushort_as_half((unsigned short)h0)), v1 - __half2float(__ushort_as_half((unsigned short)h1)));
    __half* const at = reinterpret_cast<__half*>(xa) + xa_index<NP>(k, 2 * q);
    *reinterpret_cast<uint32_t*>(at) = h0 | (h1 << 16);
    *reinterpret_cast<__half2*>(at + 16) = lo;
}
template <int NP>
__device__ __forceinline__ void xa_store(uint8_t* xa, int k, float v, int q) {
    const __half hi = __ushort_as_half((unsigned short)xa_hi(v));
    __half* const at = reinterpret_cast<__half*>(xa) + xa_index<NP>(k, 2 * q);
    at[0] = hi;
    at[16] = __float2half_rn(v - __half2float(hi));
}

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- GGUF blocks: the activation as int8 digits, the products on the int8 tensor-core path ----
// A Q8_0 weight is an int8, a Q4_0 nibble becomes one (times 16) with a mask: instead of widening the weights to fp16, the
// staged activation is turned into integers.  Per block of 32 columns x_i ~ q I_i with q a power of two and |I_i| <= 2^22, and
// I = 65536 d0 + 256 d1 + d2 (+ d3 / 256) with int8 digits: 22 bits relative to the block's largest value, for Q4_0 30.  The
// weights stay exact.  The digits are B columns 0, 1, .. of one mma.sync.m16n8k32 (s8 x s8), the int32 results are combined
// and scaled by q and the weight block's scale in fp32.  Error of a product against 64 bits (2-norm, K = 64 .. 5632, three
// distributions): Q8_0 1.7e-7 to 5.9e-7 (three digits per quotient of the block's maximum: 3.3e-7 to 9.5e-7), Q4_0 0.4e-7 to 1.3e-7
// (fp16 parts times nibbles widened to fp16: 0.5e-7 to 1.3e-7; three digits: 1.6e-7 to 6.7e-7).
//
// Staged layout: block kb holds [digit c][piece t][8 bytes: columns 4t..4t+3 then 16+4t..16+4t+3], the B
// registers of lane (g = c, t).
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23: added to a float of magnitude up to 2^22 it leaves the nearest integer in the low mantissa bits

// Maximum that keeps a NaN.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// Stages N quads of elements k .. k + 3 (k a multiple of 4) per lane; groups of eight lanes with consecutive quads hold one block of
// 32 columns each (`mask`: the lanes that take part; `live`: which quads of this lane are stored).  The N quads go side by side: a
// block's maximum takes three shuffles.  (A digit at a time with a quotient per block took 22 operations per element instead
// of six, and __reduce_max_sync over groups of lanes is executed group by group: 500 cycles per quad.)
// An Inf or a NaN has no digits: it makes the block's scale NaN, and so every row's sum, as a product with the value itself would.
template <int WT, int N>
__device__ __forceinline__ void qx_store_quads(uint8_t* xq, float* qs, const int (&k)[N], const float4 (&v)[N], const bool (&live)[N], unsigned mask) {
    float top[N];
#pragma unroll
    for (int j = 0; j < N; j++) top[j] = max_nan(max_nan(fabsf(v[j].x), fabsf(v[j].y)), max_nan(fabsf(v[j].z), fabsf(v[j].w)));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int j = 0; j < N; j++) top[j] = max_nan(top[j], __shfl_xor_sync(mask, top[j], o));
#pragma unroll
    for (int j = 0; j < N; j++) {
        const unsigned e = max(__float_as_uint(top[j]) >> 23, 22u);  // the largest value lies below 2^(e - 126)
        const float up = __uint_as_float((275u - e) << 23);                     // 2^(148 - e)
        // the low three bytes of (I + 0x8080) ^ 0x8080 are the digits, each in -128 .. 127 (0x400000: the low bits of the magic number)
        auto digits = [&](float x, uint32_t& rest) {
            const float t = fmaf(x, up, kRoundMagic);
            if (WT == WT_Q4_0) rest = __float_as_uint(fmaf(fminf(fmaf(x, up, kRoundMagic - t), 127.0f / 256.0f), 256.0f, kRoundMagic));  // what is left, in 1 / 256
            return (__float_as_uint(t) + 0x8080u - 0x400000u) ^ 0x8080u;
        };
        uint32_t ra = 0, rb = 0, rc = 0, rd = 0;
        const uint32_t a = digits(v[j].x, ra), b = digits(v[j].y, rb), c = digits(v[j].z, rc), d = digits(v[j].w, rd);
        const uint32_t ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);
        const int e0 = k[j] & 31;
        uint32_t* const dst = reinterpret_cast<uint32_t*>(xq + (k[j] >> 5) * (32 * qx_digits(WT)) + ((e0 & 15) << 1) + ((e0 >> 4) << 2));
        if (live[j]) {
            dst[0] = __byte_perm(__byte_perm(a, b, 0x0062), __byte_perm(c, d, 0x0062), 0x5410);
            dst[8] = __byte_perm(ab, cd, 0x7632);
            dst[16] = __byte_perm(ab, cd, 0x5410);
            if (WT == WT_Q4_0) dst[24] = __byte_perm(__byte_perm(ra, rb, 0x0040), __byte_perm(rc, rd, 0x0040), 0x5410);
            if (e0 == 0) qs[k[j] >> 5] = fmaf(top[j], 0.f, __uint_as_float((e - 21u) << 23));  // 2^(e - 148), or NaN
        }
    }
}

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------------------------------------ products

// Sums of NT tiles of sixteen rows, kept in registers while a warp goes through the units it owns.
// fp16: kSets accumulator quads per tile in turn, so that few tiles do not wait for the MMA before (a dependent one comes 35
// cycles later); quantised: scaled fp32 sums of rows g and g + 8 (lanes t = 0: digits 0 and 1, t = 1: digits 2 and 3).
template <int WT, int NP, int NT>
struct MegaSums {
    static constexpr bool kF16 = WT == WT_F16;
    static constexpr int kSets = NT == 1 ? 4 : NT == 2 ? 2 : 1;
    static constexpr int kBatch = NT == 1 ? (kF16 ? 8 : 4) : NT == 2 ? (kF16 ? 6 : 4) : 2;  // units whose loads go out together
    float f[kF16 ? NT : 1][kF16 ? kSets : 1][4];
    float a[kF16 ? 1 : NT][2];
    __device__ __forceinline__ void clear() {
        if constexpr (kF16) {
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int x = 0; x < kSets; x++) { f[j][x][0] = 0.f; f[j][x][1] = 0.f; f[j][x][2] = 0.f; f[j][x][3] = 0.f; }
        } else {
#pragma unroll
            for (int j = 0; j < NT; j++) { a[j][0] = 0.f; a[j][1] = 0.f; }
        }
    }
    // Units first, first + step, ... of a chunk's nu (unit i is unit u0 + i of the vector): tiles tile0 .. tile0 + NT - 1 of its
    // `rows` rows.  Without branches: a batch's units past the last one multiply the weights of its first one by zeros, and a
    // tile's rows past the last one read whatever lies behind it in shared memory; their sums are never stored.
    __device__ __forceinline__ void add(const uint8_t* chunk, int rows, int nu, int first, int step, int u0, const uint8_t* xa, const float* xq, int lane, int tile0) {
        const int g = lane >> 2, t = lane & 3;
        const int db = mega_data_bytes(WT, rows), sb = mega_scale_bytes(WT, rows);
        constexpr int kPiece = WT == WT_Q4_0 ? 4 : 8, kRow = 4 * kPiece, kTile = 16 * kRow, kXUnit = kF16 ? 64 * NP : 32 * qx_digits(WT);
        const bool feeds = lane < (kF16 ? 8 * NP : 4 * qx_digits(WT));  // lanes that hold a column of the B operand
        const uint8_t* const wp = chunk + tile0 * kTile + g * kRow + t * kPiece;
        const uint8_t* const xp = xa + u0 * kXUnit + lane * 8;  // (quantised: digit g's piece t, 32 g + 8 t)
        const uint8_t* const sp = chunk + nu * db + tile0 * 32 + g * 4;  // quantised: (scale of row g, of row g + 8) of every tile
#pragma unroll 1
        for (int i0 = first; i0 < nu; i0 += step * kBatch) {
            uint2 b[kBatch], w0[kBatch][NT], w8[kBatch][NT];
            __half2 sc[kBatch][NT];
            float q[kBatch];
#pragma unroll
            for (int x = 0; x < kBatch; x++) {
                const int i = mega_batch_unit(i0, x, step, nu);
                b[x] = make_uint2(0, 0);
                if (feeds && (x == 0 || i0 + x * step < nu)) b[x] = *reinterpret_cast<const uint2*>(xp + i * kXUnit);
                if (!kF16) q[x] = xq[u0 + i];
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    const uint8_t* const at = wp + i * db + j * kTile;
                    if constexpr (WT == WT_Q4_0) {
                        w0[x][j].y = *reinterpret_cast<const uint32_t*>(at);
                        w8[x][j].y = *reinterpret_cast<const uint32_t*>(at + 8 * kRow);
                    } else {
                        w0[x][j] = *reinterpret_cast<const uint2*>(at);
                        w8[x][j] = *reinterpret_cast<const uint2*>(at + 8 * kRow);
                    }
                    if (!kF16) sc[x][j] = *reinterpret_cast<const __half2*>(sp + i * sb + j * 32);
                }
            }
#pragma unroll
            for (int x = 0; x < kBatch; x++)
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    if constexpr (kF16) {
                        mma_16816(f[j][x % kSets], w0[x][j].x, w8[x][j].x, w0[x][j].y, w8[x][j].y, b[x].x, b[x].y);
                    } else {
                        if constexpr (WT == WT_Q4_0) {  // two's-complement nibbles: bytes of 16 times the weight (the low ones: columns 4t.., the high ones: 16 + 4t..)
                            w0[x][j].x = (w0[x][j].y << 4) & 0xF0F0F0F0u; w0[x][j].y &= 0xF0F0F0F0u;
                            w8[x][j].x = (w8[x][j].y << 4) & 0xF0F0F0F0u; w8[x][j].y &= 0xF0F0F0F0u;
                        }
                        int c[4] = {0, 0, 0, 0};
                        mma_s8(c, w0[x][j].x, w8[x][j].x, w0[x][j].y, w8[x][j].y, b[x].x, b[x].y);
                        // a lane's two result columns are one number, 256 c[0] + c[1] (at most 2^27 + 2^19)
                        const float2 s = __half22float2(sc[x][j]);
                        a[j][0] = fmaf(s.x * q[x], (float)(c[0] * 256 + c[1]), a[j][0]);
                        a[j][1] = fmaf(s.y * q[x], (float)(c[2] * 256 + c[3]), a[j][1]);
                    }
                }
        }
    }
    // The sums of rows tile * 16 + g (.x) and + 8 (.y) of position t, in the lanes with t < NP.
    __device__ __forceinline__ float2 take(int j, int lane) {
        if constexpr (kF16) {
            float v[4] = {f[j][0][0], f[j][0][1], f[j][0][2], f[j][0][3]};
#pragma unroll
            for (int x = 1; x < kSets; x++) { v[0] += f[j][x][0]; v[1] += f[j][x][1]; v[2] += f[j][x][2]; v[3] += f[j][x][3]; }
            return make_float2(v[0] + v[1], v[2] + v[3]);  // column 2q of the product is w . x_hi, column 2q + 1 is w . x_lo
        } else {
            constexpr float kOne = WT == WT_Q4_0 ? 1.0f / 16.0f : 1.0f;
            const float unit = (lane & 3) == 0 ? 256.0f * kOne : kOne / 256.0f;  // t = 0: digits 0 and 1; t = 1: digits 2 and 3 (the other lanes' columns are zero)
            float x = a[j][0] * unit, y = a[j][1] * unit;
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            return make_float2(x, y);
        }
    }
};

// The sums over the warps of rows r and r + 1 (r even): all loads are issued before the first addition.
__device__ __forceinline__ float2 mega_take_sum2(const float* sums, int stride, int r) {
    float2 v[kMegaConsumerWarps];
#pragma unroll
    for (int x = 0; x < kMegaConsumerWarps; x++) v[x] = *reinterpret_cast<const float2*>(sums + x * stride + r);
#pragma unroll
    for (int o = kMegaConsumerWarps / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int x = 0; x < o; x++) { v[x].x += v[x + o].x; v[x].y += v[x + o].y; }
    }
    return v[0];
}
__device__ __forceinline__ float mega_sum_warps(const float* red) {
    const float4* r4 = reinterpret_cast<const float4*>(red);
    float v[kMegaConsumerWarps / 4];
#pragma unroll
    for (int i = 0; i < kMegaConsumerWarps / 4; i++) v[i] = (r4[i].x + r4[i].y) + (r4[i].z + r4[i].w);
    static_assert(kMegaConsumerWarps == 8, "two quads");
    return v[0] + v[1];
}
// The sum of v0 and the maximum of v1 >= 0 over the consumer threads (GPT-2).  One CTA barrier.
__device__ __forceinline__ float2 mega_block_sum_max(float v0, float v1, float* red) {
    v1 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v1)));  // (non-negative floats order as their bits)
    v0 = warp_sum(v0);
    if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = v0; red[kMegaConsumerWarps + (threadIdx.x >> 5)] = v1; }
    consumer_sync();
    const float4* r4 = reinterpret_cast<const float4*>(red + kMegaConsumerWarps);
    float top = 0.f;
#pragma unroll
    for (int q = 0; q < kMegaConsumerWarps / 4; q++) top = fmaxf(top, fmaxf(fmaxf(r4[q].x, r4[q].y), fmaxf(r4[q].z, r4[q].w)));
    return make_float2(mega_sum_warps(red), top);
}

// ------------------------------------------------------------------------------------------------ attention

// S2: attention of one head over the cached positions [0, n_cached) plus the new ones (whose keys and values are in
// shared memory).
// Each warp owns the positions t = warp + NW*i (8 kSt per round).  Four neighbouring lanes share one position: each loads
// a quarter of its K row with 16-byte vectors and the score is completed with two shuffles.  The probabilities are
// then broadcast position by position while every lane accumulates its own channels of V.  The K and V rows of the
// first round are requested before the query is known, and the new positions take their place in the round like cached ones.  The
// per-warp (max, sum, ctx) triples are merged once, by all threads: a few lanes per output channel, combined with
// shuffles (two warps walking all triples took 0.3 us longer per layer).
template <int HD, int NW, int ST>  // NW = warps that share one query
struct MegaKvRound {
    static constexpr int kPieces = HD / 32, kPer = HD / 32;  // 16-byte pieces of a quarter of a key; channels of a lane
    static constexpr int kSt = ST;  // positions of a lane (of a warp: 8 kSt)
    uint4 k[kSt][kPieces];
    uint2 v[8 * kSt];
    // K, V: the head's rows of the cache; positions past the cached ones read as zeros.
    __device__ __forceinline__ void load(const __half* K, const __half* V, int base, int n_cached, int warp, int lane) {
        const int sub = lane & 3, tl = lane >> 2, left = n_cached - base - warp;
        const __half* kp = K + (size_t)(base + warp + NW * tl) * HD + sub * (HD / 4);
#pragma unroll
        for (int st = 0; st < kSt; st++)
#pragma unroll
            for (int c = 0; c < kPieces; c++) {
                k[st][c] = make_uint4(0, 0, 0, 0);
                if (NW * (st * 8 + tl) < left) k[st][c] = __ldcg(reinterpret_cast<const uint4*>(kp + st * 8 * NW * HD) + c);
            }
        const __half* vp = V + (size_t)(base + warp) * HD + lane * kPer;
#pragma unroll
        for (int j = 0; j < 8 * kSt; j++) {
            v[j] = make_uint2(0, 0);
            if (NW * j < left) {
                if (kPer == 4) v[j] = __ldcg(reinterpret_cast<const uint2*>(vp + j * NW * HD));
                else if (kPer == 2) v[j].x = __ldcg(reinterpret_cast<const unsigned int*>(vp + j * NW * HD));
                else v[j].x = (unsigned int)__ldcg(reinterpret_cast<const unsigned short*>(vp + j * NW * HD));
            }
        }
    }
    // The keys of the new positions n_cached .. last that fall into this round, from shared memory.
    __device__ __forceinline__ void take_new(const __half* kn, int base, int n_cached, int last, int warp, int lane) {
        const int sub = lane & 3, tl = lane >> 2;
#pragma unroll
        for (int st = 0; st < kSt; st++) {
            const int t = base + warp + NW * (st * 8 + tl);
            if (t >= n_cached && t <= last) {
#pragma unroll
                for (int c = 0; c < kPieces; c++) k[st][c] = *(reinterpret_cast<const uint4*>(kn + (t - n_cached) * HD + sub * (HD / 4)) + c);
            }
        }
    }
};

// Row of the cache (head_dim elements each) of sequence 0; a cache that fits the device has fewer than 2^32 of them.
__device__ __forceinline__ unsigned mega_kv_row(const ModelDims& m, int layer, int kvh, int pos) {
    return ((unsigned)layer * (unsigned)m.n_seq * (unsigned)m.n_kv_head + (unsigned)kvh) * (unsigned)m.max_seq + (unsigned)pos;
}
// Maximum over a warp through the integer reduction: the bits of a float, the lower 31 flipped where it is negative, order like it.
__device__ __forceinline__ float mega_warp_max(float v) {
    int i = __float_as_int(v);
    i ^= (i >> 31) & 0x7fffffff;
    i = __reduce_max_sync(0xffffffffu, i);
    i ^= (i >> 31) & 0x7fffffff;
    return __int_as_float(i);
}

// With NP positions per pass the consumer warps split into NP teams of NW = kMegaConsumerWarps / NP warps, one team per query: query qi
// sees the n_cached cached positions and the new positions 0 .. qi, whose keys and values are rows of s.kn / s.vn; its
// context lands in position qi of the staged s.ctx.  The teams run side by side (each reads the cached rows itself).
// The context is staged as the products of weights of type WT read it.
template <int HD, int NP, int WT, int ST, class WaitQ>
__device__ __forceinline__ void mega_attention_rounds(const MegaShared& s, const MegaShare& w, const ModelDims& m, const KvLayout& kv, int layer, int n_cached, WaitQ wait_q) {
    constexpr int NW = kMegaConsumerWarps / NP;
    const int tid = threadIdx.x, lane = tid & 31;
    const int qi = (tid >> 5) / NW, warp = (tid >> 5) - qi * NW;  // this warp's query and its place in the team
    constexpr int cpl = HD / 32, KV4 = HD / 32;
    const int last = n_cached + qi;  // newest position this query sees
    const size_t head = (size_t)mega_kv_row(m, layer, w.kvh, 0) * HD;
    const __half* K = kv.k + head;
    const __half* V = kv.v + head;
    const int sub = lane & 3, tl = lane >> 2;
    constexpr int kSt = MegaKvRound<HD, NW, ST>::kSt, kRound = NW * 8 * kSt;  // positions per round of a team
    constexpr float scale = HD == 32 ? 0.17677669529663687f : HD == 64 ? 0.125f : 0.08838834764831845f;  // 1 / sqrt(HD)
    const float4* const qv = reinterpret_cast<const float4*>(s.qs + qi * HD + sub * (HD / 4));  // this lane's quarter of the query
    float m_w = -INFINITY, l_w = 0.f;  // l_w: this lane's share (every probability sits in four lanes)
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int base = 0; base < n_cached + NP; base += kRound) {
        MegaKvRound<HD, NW, ST> cur;
        cur.load(K, V, base, n_cached, warp, lane);
        if (base == 0) wait_q();  // the loads above are in flight while the query is awaited
        const bool news = base + kRound > n_cached;  // the new positions may fall into this round
        if (news) cur.take_new(s.kn, base, n_cached, last, warp, lane);
        float sc[kSt], top = -INFINITY;
#pragma unroll
        for (int st = 0; st < kSt; st++) {
            const int t = base + warp + NW * (st * 8 + tl);
            float d0 = 0.f, d1 = 0.f;
#pragma unroll
            for (int c = 0; c < KV4; c++) {
                const uint32_t ww[4] = {cur.k[st][c].x, cur.k[st][c].y, cur.k[st][c].z, cur.k[st][c].w};
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float4 q = qv[2 * c + i];
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&ww[2 * i])), h = __half22float2(*reinterpret_cast<const __half2*>(&ww[2 * i + 1]));
                    d0 = fmaf(f.x, q.x, d0);
                    d1 = fmaf(f.y, q.y, d1);
                    d0 = fmaf(h.x, q.z, d0);
                    d1 = fmaf(h.y, q.w, d1);
                }
            }
            float dot = (d0 + d1) * scale;
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
            sc[st] = t <= last ? dot : -INFINITY;
            top = fmaxf(top, sc[st]);
        }
        const float m_new = fmaxf(m_w, mega_warp_max(top));
        float pr[kSt], psum = 0.f;
#pragma unroll
        for (int st = 0; st < kSt; st++) {
            pr[st] = sc[st] == -INFINITY ? 0.f : __expf(sc[st] - m_new);
            psum += pr[st];
        }
        const float corr = m_w == -INFINITY ? 0.f : __expf(m_w - m_new);
        l_w = fmaf(l_w, corr, psum);
#pragma unroll
        for (int c = 0; c < 4; c++) acc[c] *= corr;
#pragma unroll
        for (int j = 0; j < 8 * kSt; j++) {
            const float pj = __shfl_sync(0xffffffffu, pr[j >> 3], (j & 7) * 4);
            const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&cur.v[j].x));
            const float2 f1 = __half22float2(*reinterpret_cast<const __half2*>(&cur.v[j].y));
            acc[0] = fmaf(pj, f0.x, acc[0]);
            if (cpl >= 2) acc[1] = fmaf(pj, f0.y, acc[1]);
            if (cpl == 4) { acc[2] = fmaf(pj, f1.x, acc[2]); acc[3] = fmaf(pj, f1.y, acc[3]); }
        }
        if (news) {  // (their values were zeros above)
#pragma unroll
            for (int jj = 0; jj < NP; jj++) {
                const int at = n_cached + jj - base - warp;  // position n_cached + jj is this warp's number at / NW
                if (jj <= qi && at >= 0 && at < kRound && at % NW == 0) {
                    const int j = at / NW;
                    float mine = pr[0];
#pragma unroll
                    for (int st = 1; st < kSt; st++) mine = j >> 3 == st ? pr[st] : mine;
                    const float pj = __shfl_sync(0xffffffffu, mine, (j & 7) * 4);
                    const __half* vn = s.vn + jj * HD + lane * cpl;
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (c < cpl) acc[c] = fmaf(pj, __half2float(vn[c]), acc[c]);
                }
            }
        }
        m_w = m_new;
    }
    l_w = 0.25f * warp_sum(l_w);
    // merge the per-warp partial results of every team (a warp that saw no position carries max = -inf, sum = 0)
    const int gw = tid >> 5;  // warp index among all consumers
#pragma unroll
    for (int c = 0; c < 4; c++)
        if (c < cpl) s.part[gw * HD + lane * cpl + c] = acc[c];
    if (lane == 0) { s.red[gw] = m_w; s.red[kMegaConsumerWarps + gw] = l_w; }
    consumer_sync();
    {
        // G lanes per output channel, each with cpl of the team's NW partial results; the lanes combine with shuffles
        constexpr int G = kMegaConsumers / (NP * HD);
        static_assert(G >= 1 && G <= 32 && G * cpl == NW, "merge layout");
        const int o = tid / G, xr = tid - o * G;
        const int qq = o / HD, ch = o - qq * HD;
        float mv[cpl], gm = -INFINITY;
#pragma unroll
        for (int k = 0; k < cpl; k++) { mv[k] = s.red[qq * NW + xr * cpl + k]; gm = fmaxf(gm, mv[k]); }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, off));
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int k = 0; k < cpl; k++) {
            const int x = qq * NW + xr * cpl + k;
            const float f = mv[k] == -INFINITY ? 0.f : __expf(mv[k] - gm);
            num = fmaf(s.part[x * HD + ch], f, num);
            den = fmaf(s.red[kMegaConsumerWarps + x], f, den);
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
            num += __shfl_xor_sync(0xffffffffu, num, off);
            den += __shfl_xor_sync(0xffffffffu, den, off);
        }
        // the staged operand of the Wo products
        const float cv = den > 0.f ? __fdividef(num, den) : 0.f;
        if constexpr (WT != WT_F16) {
            // int8 digit staging works on whole blocks of consecutive elements: the channel values are gathered first
            // (in the query's place: every warp is past its scores)
            static_assert(NP == 1, "int8 context staging handles one position");
            if (xr == 0) s.qs[ch] = cv;
            consumer_sync();
            if (tid < HD / 4) {
                const int k[1] = {4 * tid};
                const float4 v[1] = {*reinterpret_cast<const float4*>(s.qs + 4 * tid)};
                const bool live[1] = {true};
                qx_store_quads<WT, 1>(s.ctx, reinterpret_cast<float*>(s.ctx + xa_bytes(WT, HD, 1)), k, v, live, 0xffu << (lane & 24));
            }
        } else {
            if (xr == 0) xa_store<NP>(s.ctx, ch, cv, qq);
        }
    }
    consumer_sync();
}

// Positions per round: 8 of a lane's group times ST times the warps of a query.  fp16 models: short contexts take half rounds (6 layers
// d768: 1.05 -> 0.87 us per layer and attention up to 128 positions); quantised ones, whose kernel is larger, are slower with a second
// copy of the code.
template <int HD, int NP, int WT, class WaitQ>
__device__ __forceinline__ void mega_attention(const MegaShared& s, const MegaShare& w, const ModelDims& m, const KvLayout& kv, int layer, int n_cached, WaitQ wait_q) {
    if constexpr (HD == 128) mega_attention_rounds<HD, NP, WT, 2>(s, w, m, kv, layer, n_cached, wait_q);
    else if (WT == WT_F16 && n_cached + NP <= 16 * (kMegaConsumerWarps / NP)) mega_attention_rounds<HD, NP, WT, 2>(s, w, m, kv, layer, n_cached, wait_q);
    else mega_attention_rounds<HD, NP, WT, 4>(s, w, m, kv, layer, n_cached, wait_q);
}

// ------------------------------------------------------------------------------------------------ consumers

// The model a pass runs through.
struct MegaModel {
    const float* norms;       // [2 n_layer + 1][d_model]
    const uint16_t* tok_emb;
    KvLayout kv;
};

// The larger of two arg-max words held by the lanes of a warp: [ordered logit bits : 32][0xffffff - index : 24][tag : 8].  Two
// integer reductions: the largest logit, then the largest rest among the lanes that have it.
__device__ __forceinline__ unsigned long long mega_warp_best(unsigned long long k) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
    return ((unsigned long long)hi << 32) | lo;
}

// The candidate of a CTA in which a wait ran out: it went on with operands that never arrived, and what it published is
// complete by its tags.  No logit orders as high (a NaN is never a best row), so every CTA finds the mark as the largest candidate.
constexpr unsigned long long kMegaGaveUp = 0xffffffffffffff00ull;

// The consumer warps of a CTA.  A pass is one forward step for NP consecutive token positions, or only its LM head.
// Every stage's operand vector is dealt out to the warps by K units (unit u to warp u % 8): a warp polls the words of its own
// columns, stages them for the tensor cores and multiplies them with all rows of the CTA, and nothing is shared between the
// warps before their partial sums meet.  One CTA barrier per stage remains: the norm's sum of squares meets there too (RMSNorm
// scales the sums, so the products need not wait for it), and a warp's products start when its own columns have arrived.
//
// The bound of the small models is the issue rate: a layer is one pass over straight-line code, and every warp issues it.  Eight
// warps instead of sixteen, two per scheduler, halve what the set-up, the polling and the reductions cost and leave each warp the
// registers to keep twice the loads in flight; an own copy of the code per stage keeps the selection between the stages out
// of it.
template <int HD, int WT, bool GPT2, int NP>
struct MegaWorker {
    static constexpr bool kQuant = WT != WT_F16;
    static constexpr int half = HD / 2;
    const MegaArgs& a;
    const MegaShared& s;
    const MegaShare& w;  // in shared memory, read wherever it is needed: no registers, no recomputation
    const int tid, warp, lane;
    MegaCursor c, pend_from;           // ring position, advances in lock step with the producer's; first slot whose release was put off
    unsigned n_chunk = 0, landed = 0;  // chunks consumed so far; chunks known to have arrived
    int par = 0;                       // which half of s.sums the next group's sums go to
    int n_pend = 0;
    int n_stamp = 0;
    bool tracing = false;
    bool asked = false;                // the host wants the loop to end: the same pass tells every CTA

    __device__ __forceinline__ MegaWorker(const MegaArgs& a_, const MegaShared& s_)
        : a(a_), s(s_), w(*s_.share), tid((int)threadIdx.x), warp((int)threadIdx.x >> 5), lane((int)threadIdx.x & 31) {}

    __device__ __forceinline__ void stamp() {
        if (tracing) a.trace[n_stamp++] = clock64();
    }

    // A freed slot makes the producer request the chunk that is n_slots ahead at once: megabytes of reads over all
    // CTAs, which would travel through L2 together with the words of the exchange that follows the stage and delay
    // them by microseconds.  The last chunk of a stage is therefore handed back only after that exchange (the chunk it
    // makes room for is needed later; 22-layer d2048 model, Q8_0: 441 us per token without, 429 with).
    __device__ __forceinline__ void release_pending() {
        if (n_pend) mega_release_deferred(a, s, pend_from, n_pend);
        n_pend = 0;
    }
    __device__ __forceinline__ void hand_back(bool later) {
        if (later) {
            if (n_pend == 0) pend_from = c;
            n_pend++;
            c.next((unsigned)a.plan.n_slots);
        } else {
            mega_release(a, s, c);
        }
    }

    // Brings the count of arrived chunks up to date while there is something else to wait for: the products then find their chunk
    // without a read.
    __device__ __forceinline__ void peek() {
        const unsigned n = ld_acquire_cta_shared(s.landed);
        landed = __shfl_sync(0xffffffffu, n, 0);
    }

    // ---- products

    // One group of rows: this warp's partial sums to `mine`.
    template <int W2, int NT>
    __device__ __forceinline__ void group_products(const MegaStage& st, int n, int keep, float* mine) {
        const int tiles = (n + 15) >> 4;
        MegaSums<W2, NP, NT> acc;
        acc.clear();
#pragma unroll 1
        for (int u0 = 0; u0 < st.units; u0 += st.chunk_units) {
            const int nu = min(st.chunk_units, st.units - u0);
            const uint8_t* ch = mega_acquire(a, s, c, n_chunk++, landed);
            acc.add(ch, n, nu, (warp - u0) & (kMegaConsumerWarps - 1), kMegaConsumerWarps, u0, s.xa, s.xq, lane, 0);
            hand_back(u0 + keep * st.chunk_units >= st.units);
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const float2 y = acc.take(j, lane);
            if (j < tiles && (lane & 3) < NP) {
                float* dst = mine + (lane & 3) * 16 * a.plan.group_tiles + j * 16 + (lane >> 2);
                dst[0] = y.x;
                dst[8] = y.y;
            }
        }
    }
    // This CTA's rows of Wo restricted to its head's columns: every row's sum is one contribution to the counted sum of that row
    // (head 0 also carries the residual).  A warp owns whole 16-row tiles: its lanes hold finished sums, and no barrier follows.
    template <int NT>
    __device__ __forceinline__ void wo_tiles(const uint8_t* ch, int n, int r0, int l) {
        const int d = a.m.d_model, all = (n + 15) >> 4;
#pragma unroll 1
        for (int tile = NT * warp; tile < all; tile += NT * kMegaConsumerWarps) {
            MegaSums<WT, NP, NT> acc;
            acc.clear();
            acc.add(ch, n, HD / mega_unit(WT), 0, 1, 0, s.ctx, reinterpret_cast<const float*>(s.ctx + xa_bytes(WT, HD, NP)), lane, tile);
            const int q = lane & 3, first = w.blk * a.plan.rpb + r0, row = first + tile * 16 + (lane >> 2), last = min(d, first + n);
            float v[2 * NT];
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const float2 y = acc.take(j, lane);
                v[2 * j] = y.x; v[2 * j + 1] = y.y;
            }
            if (w.head == 0 && q < NP) {
#pragma unroll
                for (int i = 0; i < 2 * NT; i++) {
                    const int orow = min(row + 8 * i, d - 1);
                    v[i] += s.xres[q * d + orow] + (GPT2 ? __ldg(a.out_bias + (size_t)2 * l * d + orow) : 0.f);
                }
            }
            unsigned long long* const dst = a.mid_sums + (q < NP ? q * d : 0) + row;
            unsigned long long c64[2 * NT];
#pragma unroll
            for (int i = 0; i < 2 * NT; i++) c64[i] = counted(v[i]);
#pragma unroll
            for (int i = 0; i < 2 * NT; i++)
                if (q < NP && row + 8 * i < last) red_add_u64(dst + 8 * i, c64[i]);
        }
    }
    __device__ __forceinline__ void wo_products(const MegaStage& st, int l) {
#pragma unroll 1
        for (int r0 = 0; r0 < a.plan.rpb; r0 += st.group_rows) {
            const int n = min(st.group_rows, a.plan.rpb - r0);
            const uint8_t* ch = mega_acquire(a, s, c, n_chunk++, landed);
            if (n <= 16 * kMegaConsumerWarps) wo_tiles<1>(ch, n, r0, l);
            else wo_tiles<4>(ch, n, r0, l);
            hand_back(r0 + st.group_rows >= a.plan.rpb);
        }
    }

    // ---- staging

    // A lane handles four columns of a quantised type's block, or two of an fp16 unit: eight lanes share a unit.  Items of this warp,
    // numbered through its units: how many, and which column item `it` starts at.
    template <int W2>
    __device__ __forceinline__ int items(int units) const {
        return units > warp ? (units - warp + kMegaConsumerWarps - 1) / kMegaConsumerWarps * 8 : 0;
    }
    template <int W2>
    __device__ __forceinline__ int column(int it) const {
        return (warp + (it >> 3) * kMegaConsumerWarps) * mega_unit(W2) + (it & 7) * (mega_unit(W2) / 8);
    }
    // N items per lane (of position q, columns k .., `live` or not): the residual stream's raw copy (`stream`), gained copy as the
    // products' operand, sum of squares.  Without branches, so that the items' latencies overlap; all lanes of the warp call.
    template <int W2, int N>
    __device__ __forceinline__ void stage_items(bool stream, const bool (&live)[N], const int (&q)[N], const int (&k)[N], const float (&v)[N][mega_unit(W2) / 8],
                                                const float (&g)[N][mega_unit(W2) / 8], float (&ss)[NP]) {
        if constexpr (W2 != WT_F16) {
            float4 x[N];
#pragma unroll
            for (int j = 0; j < N; j++) {
                if (stream && live[j]) *reinterpret_cast<float4*>(s.xres + k[j]) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
                if (stream) ss[0] += fmaf(v[j][0], v[j][0], fmaf(v[j][1], v[j][1], fmaf(v[j][2], v[j][2], v[j][3] * v[j][3])));
                x[j] = make_float4(v[j][0] * g[j][0], v[j][1] * g[j][1], v[j][2] * g[j][2], v[j][3] * g[j][3]);
            }
            qx_store_quads<W2, N>(s.xa, s.xq, k, x, live, 0xffffffffu);
        } else {
#pragma unroll
            for (int j = 0; j < N; j++) {
                if (stream && live[j]) *reinterpret_cast<float2*>(s.xres + q[j] * a.m.d_model + k[j]) = make_float2(v[j][0], v[j][1]);
                if (GPT2 && stream) {  // (staged by layer_norm)
                    ln_sum += v[j][0] + v[j][1];
                    ln_top = fmaxf(ln_top, fmaxf(fabsf(v[j][0]), fabsf(v[j][1])));
                    continue;
                }
                if (live[j]) xa_store_pair<NP>(s.xa, k[j], v[j][0] * g[j][0], v[j][1] * g[j][1], q[j]);
                if (!stream) continue;
                const float sq = fmaf(v[j][0], v[j][0], v[j][1] * v[j][1]);
                if (NP == 2) {
                    ss[0] += q[j] ? 0.f : sq;
                    ss[NP - 1] += q[j] ? sq : 0.f;
                } else {
                    ss[0] += sq;
                }
            }
        }
    }
    // Polls this warp's columns of an exchanged vector and stages them.  MS_UP: counted sums, complete after n_head contributions;
    // else words with the tag.  Up to kPolls items of a lane are in flight, words that validated are not read again, and what else
    // an item needs is requested before its words are awaited.
    template <int KIND, int W2>
    __device__ __forceinline__ void stage_words(unsigned tag, const float* gain, float (&ss)[NP]) {
        constexpr bool kSums = KIND == MS_UP, kAct = KIND == MS_DOWN;
        constexpr int kCols = mega_unit(W2) / 8, kLoads = kCols / 2;
        // One round of polls holds d_model 1024 and hidden 2048 (GPT-2: 3072), of quantised types 2048 and 6144, for two positions 768
        // and 2048; a wider vector takes another round, a round trip to L2 each.  (Two positions of the 6-layer model with two and
        // four items per lane instead of three and eight: a two-token pass took 113 us instead of 104.)
        constexpr int kPolls = NP == 2 ? (kAct ? 8 : 3) : kAct ? (GPT2 || kQuant ? 6 : 4) : 2;
        constexpr int kCode = kSums ? 7 : kAct ? 8 : KIND == MS_QKV ? 5 : 9;
        const int K = kAct ? a.m.hidden : a.m.d_model, n = items<W2>(K / mega_unit(W2)), total = NP * n;
        const bool lines = kAct && !kQuant && a.plan.act_wpc > 0;
        const unsigned long long* const base = kAct ? a.act_words : kSums ? a.mid_sums : a.x_words;
        const unsigned n_contrib = (unsigned)a.m.n_head;
#pragma unroll 1
        for (int i0 = 0; i0 < total; i0 += 32 * kPolls) {
            ulonglong2 wd[kPolls][kLoads];
            float g[kAct || GPT2 ? 1 : kPolls][kCols];
            const unsigned long long* src[kPolls];
            const ulonglong2* prev[kPolls];
            bool ok[kPolls];
#pragma unroll
            for (int j = 0; j < kPolls; j++) {
                const int it = i0 + 32 * j + lane;
                ok[j] = it >= total;
                const int q = NP == 2 && it >= n ? 1 : 0, k = ok[j] ? 0 : column<W2>(it - q * n);
                src[j] = base + (lines ? q * a.plan.n_cta * a.plan.act_wpc + (int)s.act[k >> 1] : q * K + k);
                prev[j] = reinterpret_cast<const ulonglong2*>(s.prev + (kSums ? q * K + k : 0));
#pragma unroll
                for (int i = 0; i < kLoads; i++) wd[j][i] = make_ulonglong2(0, 0);
                if constexpr (!kAct && !GPT2) {
#pragma unroll
                    for (int i = 0; i < kLoads; i++) {
                        const float2 f = __ldg(reinterpret_cast<const float2*>(gain + k) + i);
                        g[j][2 * i] = f.x; g[j][2 * i + 1] = f.y;
                    }
                }
            }
            unsigned spins = 0;
            if (!mega_aborting(s)) {
                while (true) {
                    bool all = true;
#pragma unroll
                    for (int j = 0; j < kPolls; j++)
                        if (!ok[j]) {
#pragma unroll
                            for (int i = 0; i < kLoads; i++) wd[j][i] = ld_words2(src[j] + 2 * i);
                        }
#pragma unroll
                    for (int j = 0; j < kPolls; j++)
                        if (!ok[j]) {
                            ok[j] = true;
#pragma unroll
                            for (int i = 0; i < kLoads; i++) {
                                if constexpr (kSums) {
                                    const ulonglong2 pv = prev[j][i];
                                    ok[j] = ok[j] && (((unsigned)wd[j][i].x - (unsigned)pv.x) & 0xffu) == n_contrib && (((unsigned)wd[j][i].y - (unsigned)pv.y) & 0xffu) == n_contrib;
                                } else {
                                    ok[j] = ok[j] && (unsigned)(wd[j][i].x >> 32) == tag && (unsigned)(wd[j][i].y >> 32) == tag;
                                }
                            }
                            all = all && ok[j];
                        }
                    if (all) break;
                    if (mega_spin_out(a, s, spins, kCode)) break;
                }
            }
            __syncwarp();
            int q[kPolls], k[kPolls];
            float v[kPolls][kCols], gain_of[kPolls][kCols];
            bool live[kPolls];
#pragma unroll
            for (int j = 0; j < kPolls; j++) {
                const int it = i0 + 32 * j + lane;
                live[j] = it < total;
                q[j] = NP == 2 && it >= n ? 1 : 0;
                k[j] = live[j] ? column<W2>(it - q[j] * n) : 0;
#pragma unroll
                for (int i = 0; i < kLoads; i++) {
                    if constexpr (kSums) {
                        ulonglong2* const p = const_cast<ulonglong2*>(prev[j]) + i;
                        const ulonglong2 pv = *p;
                        if (live[j]) *p = wd[j][i];
                        v[j][2 * i] = (float)((long long)(wd[j][i].x - pv.x - (unsigned long long)n_contrib) >> 8) * kMegaUnfix;
                        v[j][2 * i + 1] = (float)((long long)(wd[j][i].y - pv.y - (unsigned long long)n_contrib) >> 8) * kMegaUnfix;
                        if (!live[j]) v[j][2 * i] = v[j][2 * i + 1] = 0.f;
                    } else {
                        v[j][2 * i] = __uint_as_float((unsigned)wd[j][i].x);
                        v[j][2 * i + 1] = __uint_as_float((unsigned)wd[j][i].y);
                    }
                    gain_of[j][2 * i] = gain_of[j][2 * i + 1] = 1.f;
                    if constexpr (!kAct && !GPT2) { gain_of[j][2 * i] = g[j][2 * i]; gain_of[j][2 * i + 1] = g[j][2 * i + 1]; }
                }
            }
            stage_items<W2, kPolls>(!kAct, live, q, k, v, gain_of, ss);
        }
    }
    // The same for a pass's first vector: the embedding of the tokens, or (the head alone) the sequence's last hidden state.
    template <int W2>
    __device__ __forceinline__ void stage_first(bool hidden, const uint32_t (&tok)[NP], int pos, const uint16_t* tok_emb, const float* gain, float (&ss)[NP]) {
        constexpr int kCols = mega_unit(W2) / 8;
        const int d = a.m.d_model, n = items<W2>(d / mega_unit(W2));
#pragma unroll 1
        for (int i0 = 0; i0 < NP * n; i0 += 32) {
            const int it = i0 + lane;
            const bool live[1] = {it < NP * n};
            const int q[1] = {NP == 2 && it >= n ? 1 : 0}, k[1] = {live[0] ? column<W2>(it - q[0] * n) : 0};
            float v[1][kCols], g[1][kCols];
#pragma unroll
            for (int i = 0; i < kCols; i += 2) {
                float2 x;
                if (hidden) {
                    x = __ldcg(reinterpret_cast<const float2*>(a.hidden_io + k[0] + i));
                } else {
                    x = __half22float2(*reinterpret_cast<const __half2*>(tok_emb + (size_t)(q[0] ? tok[NP - 1] : tok[0]) * d + k[0] + i));
                    if (GPT2) {
                        const float2 pe = __half22float2(*reinterpret_cast<const __half2*>(a.pos_emb + (size_t)pos * d + k[0] + i));
                        x.x += pe.x; x.y += pe.y;
                    }
                }
                const float2 f = GPT2 ? make_float2(1.f, 1.f) : __ldg(reinterpret_cast<const float2*>(gain + k[0] + i));
                v[0][i] = live[0] ? x.x : 0.f; v[0][i + 1] = live[0] ? x.y : 0.f;
                g[0][i] = f.x; g[0][i + 1] = f.y;
            }
            stage_items<W2, 1>(true, live, q, k, v, g, ss);
        }
    }
    // GPT-2's LayerNorm.  The values are staged only when the mean is known: with a mean far from zero both E[x^2] - mean^2 and
    // W.(x g) - mean W.g cancel (one barrier less, but a stream of mean 32 and deviation 0.05 had no correct digit left).  The
    // centred values carry a power of two that puts the largest of them near 32: the fp16 parts then neither saturate on a large
    // residual stream nor lose their low half to subnormals on a small one.  Every lane normalises the pairs that it received;
    // ln_down becomes the inverse of the power of two, ss the centred squares.
    float ln_sum, ln_top, ln_down;
    __device__ __forceinline__ void layer_norm(const float* gain, float (&ss)[NP]) {
        const int total = items<WT_F16>(a.m.d_model / mega_unit(WT_F16));
        float2 ahead[2];  // (d_model <= 1024: all gains; requested before the barrier)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            ahead[j] = make_float2(0.f, 0.f);
            if (lane + 32 * j < total) ahead[j] = __ldg(reinterpret_cast<const float2*>(gain + column<WT_F16>(lane + 32 * j)));
        }
        const float2 t = mega_block_sum_max(ln_sum, ln_top, s.red);
        const float mean = t.x * (a.plan.inv_d);
        const unsigned e = min(__float_as_uint(t.y + fabsf(mean)) >> 23, 254u), f = min(258u - e, 253u);
        const float up = __uint_as_float(f << 23);
        ln_down = __uint_as_float((254u - f) << 23);
        auto pair = [&](int it, float2 g) {
            const int k = column<WT_F16>(it);
            const float2 x = *reinterpret_cast<const float2*>(s.xres + k);
            const float v0 = x.x - mean, v1 = x.y - mean;
            ss[0] = fmaf(v0, v0, fmaf(v1, v1, ss[0]));
            xa_store_pair<1>(s.xa, k, v0 * up * g.x, v1 * up * g.y, 0);
        };
#pragma unroll
        for (int j = 0; j < 2; j++)
            if (lane + 32 * j < total) pair(lane + 32 * j, ahead[j]);
#pragma unroll 1
        for (int it = lane + 64; it < total; it += 32) pair(it, __ldg(reinterpret_cast<const float2*>(gain + column<WT_F16>(it))));
    }
    // Factor of the products' sums of position q.
    __device__ __forceinline__ float norm_factor(const float* sq, int q) const {
        const float mean_sq = fmaf(mega_sum_warps(sq + q * kMegaConsumerWarps), a.plan.inv_d, a.m.eps);
        float r = rsqrtf(mean_sq);  // (a correctly rounded division and square root cost ~200 cycles here)
        if (GPT2) {
            r = r * fmaf(-0.5f * mean_sq * r, r, 1.5f);  // one Newton step: rounding error only
            r *= ln_down;
        }
        return r;
    }

    // ---- S2: attention of this CTA's head
    __device__ __forceinline__ void attention(const ModelDims& md, const KvLayout& kv, int l, int pos, unsigned seq) {
        const MegaPlan& p = a.plan;
        mega_attention<HD, NP, WT>(s, w, md, kv, l, pos, [&]() {
            // q of this CTA's head, k and v of the KV head: pairs in the order S1 published them
            for (int x = tid; x < NP * 3 * half; x += kMegaConsumers) {
                const int q = NP == 2 && x >= 3 * half ? 1 : 0, r = x - q * 3 * half;
                const int section = r / half, idx = r - section * half;
                const int item = (section == 0 ? w.hq * half : section == 1 ? p.qpk * half : (p.qpk + 1) * half) + idx;
                const unsigned long long* const src = a.qkv_words + (w.kvh * NP + q) * 2 * p.group_items + 2 * item;
                ulonglong2 v = make_ulonglong2(0, 0);
                unsigned spins = 0;
                if (!mega_aborting(s)) {
                    while (true) {
                        v = ld_words2(src);
                        if ((unsigned)(v.x >> 32) == seq && (unsigned)(v.y >> 32) == seq) break;
                        if (mega_spin_out(a, s, spins, 6)) break;
                    }
                }
                const float v0 = __uint_as_float((unsigned)v.x), v1 = __uint_as_float((unsigned)v.y);
                if (section == 0) { s.qs[q * HD + idx] = v0; s.qs[q * HD + idx + half] = v1; }
                else if (section == 1) { s.kn[q * HD + idx] = __float2half_rn(v0); s.kn[q * HD + idx + half] = __float2half_rn(v1); }
                else { s.vn[q * HD + 2 * idx] = __float2half_rn(v0); s.vn[q * HD + 2 * idx + 1] = __float2half_rn(v1); }
            }
            __syncwarp();
            release_pending();  // the q/k/v chunk
            peek();
            consumer_sync();
            stamp();
        });
        stamp();
    }

    // ---- the stages whose operand is a whole vector

    // Best row of this thread in the LM head.
    float best_v;
    int best_i;

    // Stage KIND of layer l: awaits and stages its operand (`first`: the pass's first vector), multiplies this CTA's rows, finishes and
    // publishes them.
    template <int KIND, int W2>
    __device__ __forceinline__ void stage(const MegaModel& mo, const ModelDims& md, int l, bool first, const uint32_t (&tok)[NP], int pos, unsigned seq) {
        constexpr bool kNorm = KIND == MS_QKV || KIND == MS_UP || (GPT2 && KIND == MS_HEAD);  // the sums get the norm's factor (RMSNorm's is positive: the arg-max does not need it)
        const MegaPlan& p = a.plan;
        const int d = a.m.d_model;
        const int gq = NP == 2 && tid >= kMegaConsumers / NP ? 1 : 0, gi = tid - gq * (kMegaConsumers / NP);  // epilogue: position of this thread, and which pair of a group's rows
        const int rows_of = KIND == MS_QKV ? 2 * w.s1_n : KIND == MS_UP ? p.ffn_rows * w.h_n : KIND == MS_DOWN ? w.d_n : w.v_n;
        // What the epilogue needs besides its sums is worked out before the words are awaited (a later group's with its products).
        float e0 = 0.f, e1 = 0.f;
        float2 cs;
        __half *kv0 = nullptr, *kv1 = nullptr;
        unsigned long long* dst = nullptr;
        auto prepare = [&](int r) {
            if (2 * gi >= rows_of - r) return;
            int i0 = r + 2 * gi, i1 = min(i0 + 1, rows_of - 1);
            const float* ln = nullptr;  // GPT-2: the constants of the rows
            const int ln_rows = a.m.q_dim + 2 * a.m.kv_dim + a.m.hidden;
            if constexpr (KIND == MS_QKV) {
                const int4 pair = s.s1[i0 >> 1];
                cs = make_float2(1.f, 0.f);  // (a later group's value pair must not keep the angle of an earlier one's key)
                if (!GPT2 && pair.x < 2) cs = a.rope[(size_t)(gq ? min(pos + 1, a.m.max_seq - 1) : pos) * half + pair.w];
                dst = a.qkv_words + (w.kvh * NP + gq) * 2 * p.group_items + 2 * w.s1_begin + i0;
                kv0 = nullptr;
                if (pair.x > 0 && (NP == 1 || pos + gq < md.max_seq)) {
                    kv0 = (pair.x == 1 ? mo.kv.k : mo.kv.v) + (size_t)mega_kv_row(md, l, w.kvh, pos + gq) * HD + (pair.y - w.kvh * HD);
                    kv1 = kv0 + (pair.z - pair.y);
                }
                ln = a.ln + (size_t)l * ln_rows + (pair.x == 0 ? 0 : pair.x == 1 ? a.m.q_dim : a.m.q_dim + a.m.kv_dim);
                i0 = pair.y; i1 = pair.z;
            } else if constexpr (KIND == MS_UP) {
                dst = a.act_words + (p.act_wpc ? (gq * p.n_cta + (int)blockIdx.x) * p.act_wpc : gq * a.m.hidden + w.h_begin) + (GPT2 ? i0 : i0 >> 1);
                ln = a.ln + (size_t)l * ln_rows + a.m.q_dim + 2 * a.m.kv_dim + w.h_begin;
            } else if constexpr (KIND == MS_DOWN) {
                dst = a.x_words + gq * d + w.d_begin + i0;
                ln = a.out_bias + (size_t)(2 * l + 1) * d + w.d_begin;
            } else {
                ln = a.ln + (size_t)md.n_layer * ln_rows + w.v_begin;
            }
            if (GPT2) { e0 = __ldg(ln + i0); e1 = __ldg(ln + i1); }
        };
        prepare(0);
        float ss[NP];
#pragma unroll
        for (int q = 0; q < NP; q++) ss[q] = 0.f;
        ln_sum = ln_top = 0.f;
        // The arg-max candidate words are used once per token; between two uses a whole model's worth of weights streams
        // through L2.  Reading them once per layer keeps their lines resident, so that the token exchange does not
        // start with a round trip to memory.
        if (KIND == MS_UP)
            for (int i = tid; i < NP * p.n_cta; i += kMegaConsumers) { unsigned long long keep; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(keep) : "l"(a.cand_words + (size_t)i * kMegaCandStride) : "memory"); }
        // Everything this CTA wrote with plain stores during the step (KV-cache rows; the CTA barriers since then order
        // them before these threads) is made visible before the candidate words that are published at the end of the
        // head.  Issued here, the fence overlaps the wait for the last layer's output.
        if (KIND == MS_HEAD && warp < NP && lane == 0) __threadfence();
        const float* const gain = mo.norms + (size_t)(2 * l + (KIND == MS_UP ? 1 : 0)) * d;
        peek();
        if ((KIND == MS_QKV || KIND == MS_HEAD) && first) stage_first<W2>(KIND == MS_HEAD, tok, pos, mo.tok_emb, gain, ss);
        else stage_words<KIND, W2>(KIND == MS_QKV ? seq - 1 : seq, gain, ss);
        release_pending();  // the last chunks of the stage before
        if (GPT2 && KIND != MS_DOWN) layer_norm(gain, ss);
        __syncwarp();
        stamp();
        const MegaStage& st = p.stage[KIND];
        const int stride = NP * 16 * p.group_tiles;
#pragma unroll 1
        for (int r0 = 0; r0 < rows_of; r0 += st.group_rows) {
            const int n = min(st.group_rows, rows_of - r0);
            if (r0 > 0) prepare(r0);
            const int keep = r0 + n < rows_of ? 0 : KIND == MS_HEAD ? 2 : 1;  // chunks at the end of the stage that are handed back later
            float* const sums = s.sums + par * kMegaConsumerWarps * stride;  // warp x, position q, row r: [(x NP + q) 16 group_tiles + r]
            float* const sq = s.ss + par * NP * kMegaConsumerWarps;
            par ^= 1;
            if (KIND != MS_HEAD && n <= 16) group_products<W2, 1>(st, n, keep, sums + warp * stride);
            else if (KIND != MS_HEAD && n <= 32) group_products<W2, 2>(st, n, keep, sums + warp * stride);
            else if (KIND != MS_HEAD && n <= 48) group_products<W2, 3>(st, n, keep, sums + warp * stride);
            else group_products<W2, kMegaMaxTiles>(st, n, keep, sums + warp * stride);
            if (kNorm) {
#pragma unroll
                for (int q = 0; q < NP; q++) {
                    const float t = warp_sum(ss[q]);
                    if (lane == 0) sq[q * kMegaConsumerWarps + warp] = t;
                }
            }
            consumer_sync();
            if (2 * gi < n) {
                float2 v = mega_take_sum2(sums + gq * 16 * p.group_tiles, stride, 2 * gi);
                if (kNorm) {
                    const float inv = norm_factor(sq, gq);
                    v.x *= inv; v.y *= inv;
                }
                if (GPT2) { v.x += e0; v.y += e1; }
                const bool two = 2 * gi + 1 < n;
                if constexpr (KIND == MS_QKV) {
                    // RoPE ((cos, sin) = (1, 0) for a value pair), words for the CTAs that share the KV head, KV-cache append
                    if (!GPT2) v = make_float2(v.x * cs.x - v.y * cs.y, v.x * cs.y + v.y * cs.x);
                    st_words2(dst, tagged(v.x, seq), tagged(v.y, seq));
                    if (kv0) {
                        *kv0 = __float2half_rn(v.x);
                        *kv1 = __float2half_rn(v.y);
                    }
                } else if constexpr (KIND == MS_UP) {
                    if (GPT2) st_words2(dst, tagged(gelu_f(v.x), seq), tagged(gelu_f(v.y), seq));
                    else st_word(dst, tagged(__fdividef(v.x, 1.0f + __expf(-v.x)) * v.y, seq));  // silu(gate) up
                } else if constexpr (KIND == MS_DOWN) {
                    const float* const res = s.xres + gq * d + w.d_begin + r0 + 2 * gi;
                    st_word(dst, tagged(v.x + res[0], seq));
                    if (two) st_word(dst + 1, tagged(v.y + res[1], seq));
                } else {
                    // a thread keeps the best of its rows (ascending: '>' keeps the first maximum)
                    const int row = w.v_begin + r0 + 2 * gi;
                    if (v.x > best_v) { best_v = v.x; best_i = row; }
                    if (two && v.y > best_v) { best_v = v.y; best_i = row + 1; }
                }
            }
            __syncwarp();
        }
    }

    // One pass: tokens tok[q] at positions pos + q through `layers` layers (0: the head alone, on the last hidden state), then the LM
    // head with its first-max arg-max; every CTA learns out[q].  seq: tag of everything the layer publishes, counted up by
    // every layer; tag8: tag of the arg-max candidates.  False (in every thread of the CTA): a wait ran out in this CTA, or in another
    // one before it published its candidate, and out[q] means nothing.
    __device__ __forceinline__ bool pass(const MegaModel& mo, const ModelDims& md, int layers, const uint32_t (&tok)[NP], int pos, unsigned& seq, unsigned long long tag8,
                                         uint32_t (&out)[NP]) {
        const MegaPlan& p = a.plan;
        // Why the exchange arrays need no second buffer: x_words is re-written by the W2 stage of this layer, which starts only
        // after every CTA has published its activation, i.e. after every group CTA has read x; qkv_words one layer
        // later, after x_words is complete, which needs every CTA's W2 rows, hence the whole activation, hence every
        // group CTA past its S2; mid_sums receives the next layer's contributions only after that layer's S1, which needs every
        // CTA past its read of them; act_words is re-written after mid_sums of the next layer is complete, which needs
        // every group CTA past x_words, i.e. every CTA past its W2 rows.  (A CTA publishes behind the barrier that all of its
        // warps pass after their reads.)
#pragma unroll 1
        for (int l = 0; l < layers; l++) {
            seq++;
            stamp();
            if (w.in_group) {
                stage<MS_QKV, WT>(mo, md, l, l == 0, tok, pos, seq);
                stamp();
                attention(md, mo.kv, l, pos, seq);
                wo_products(p.stage[MS_WO], l);
                stamp();
            } else if (tracing) {
                for (int i = 0; i < 5; i++) stamp();
            }
            stage<MS_UP, WT>(mo, md, l, false, tok, pos, seq);
            stamp();
            stage<MS_DOWN, WT>(mo, md, l, false, tok, pos, seq);
            stamp();
        }
        stamp();
        best_v = -INFINITY;
        best_i = 0x7fffffff;
        if (kQuant && p.wt_head == WT_F16) stage<MS_HEAD, WT_F16>(mo, md, md.n_layer, layers == 0, tok, pos, seq);  // an fp16 head on quantised layers reads the fp16 staging
        else stage<MS_HEAD, WT>(mo, md, md.n_layer, layers == 0, tok, pos, seq);
        // CTA-wide best (larger value first, then smaller index), published as one word per CTA:
        // [ordered logit bits : 32][0xffffff - index : 24][tag : 8].  The tag is the same in every word of a step, so the
        // largest word is the best candidate.
        constexpr int kTeam = kMegaConsumerWarps / NP;  // warps whose threads hold one position's rows
        constexpr bool kAsks = NP == 1;  // (the two-token loop is never asked to end, and a second word costs it 0.2 %)
        {
            const unsigned long long k = mega_warp_best(best_i != 0x7fffffff ? ((unsigned long long)ordered_bits(best_v) << 32) | ((unsigned long long)(0xffffffu - (unsigned)best_i) << 8) : 0ull);
            if (lane == 0) s.key[warp] = k;
        }
        consumer_sync();
        if (warp < NP) {
            unsigned long long k = mega_warp_best(lane < kTeam ? s.key[warp * kTeam + lane] : 0ull);
            if (mega_aborting(s)) k = kMegaGaveUp;
            unsigned long long* const dst = a.cand_words + (size_t)(warp * p.n_cta + (int)blockIdx.x) * kMegaCandStride;
            if (kAsks && lane == 0) st_words2(dst, k | tag8, ((unsigned long long)*reinterpret_cast<volatile unsigned*>(s.asked) << 8) | tag8);
            if (!kAsks && lane == 0) st_word(dst, k | tag8);
        }
        stamp();
        unsigned long long k[NP], ask = 0ull;  // the best of the candidates that this thread read, per position; their requests
#pragma unroll
        for (int q = 0; q < NP; q++) {
            k[q] = 0ull;
            for (int i = tid; i < p.n_cta; i += kMegaConsumers) {
                const unsigned long long* const src = a.cand_words + (size_t)(q * p.n_cta + i) * kMegaCandStride;
                ulonglong2 x = make_ulonglong2(0, 0);
                unsigned spins = 0;
                if (!mega_aborting(s)) {
                    while (true) {
                        if (kAsks) x = ld_words2(src);
                        else asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x.x) : "l"(src) : "memory");
                        if ((x.x & 0xffull) == tag8 && (!kAsks || (x.y & 0xffull) == tag8)) break;
                        if (mega_spin_out(a, s, spins, 10)) break;
                    }
                }
                k[q] = max(k[q], x.x);
                ask |= x.y >> 8;
            }
        }
        // a reader orders its later loads (the KV-cache rows other CTAs appended during this step) after the
        // candidate words it saw; the writers' side of the pair is the fence at the start of the head
        if (tid < p.n_cta) __threadfence();
        __syncwarp();
        consumer_sync();  // s.key was read above
#pragma unroll
        for (int q = 0; q < NP; q++) {
            const unsigned long long kq = mega_warp_best(k[q]);
            if (lane == 0) s.key[q * kMegaConsumerWarps + warp] = kq;
        }
        if (tid == 0) s.red[63] = mega_aborting(s) ? 1.f : ask ? 2.f : 0.f;  // one decision for the whole CTA (thread 0 reads CTA 0's word)
        consumer_sync();
        const float decision = s.red[63];
        bool valid = decision != 1.f;
        asked = decision == 2.f;
#pragma unroll
        for (int q = 0; q < NP; q++) {
            const unsigned long long best = mega_warp_best(lane < kMegaConsumerWarps ? s.key[q * kMegaConsumerWarps + lane] : 0ull);
            valid = valid && (best | 0xffull) != (kMegaGaveUp | 0xffull);
            out[q] = min(0xffffffu - (uint32_t)((best >> 8) & 0xffffffull), (uint32_t)(a.m.vocab - 1));  // in range even if every logit was NaN
        }
        release_pending();  // the last head chunks
        stamp();
        return valid;
    }
};

// ------------------------------------------------------------------------------------------------ the kernel

// Issues a CTA's chunks in consumption order (one thread).
struct MegaProducer {
    const MegaArgs& a;
    const MegaShared& s;
    MegaCursor c;
    unsigned issued = 0;
    uint64_t policy;
    __device__ __forceinline__ MegaProducer(const MegaArgs& a_, const MegaShared& s_) : a(a_), s(s_), policy(l2_evict_first_policy()) {}
    __device__ __forceinline__ bool stopped() const { return mega_aborting(s) || *reinterpret_cast<volatile int*>(s.stop) != 0; }
    // The chunks of stages first .. last of a layer (or the head) at src.
    __device__ __forceinline__ void stages(const uint8_t* src, int first, int last, const MegaShare& w) {
        const MegaPlan& p = a.plan;
        const unsigned n_slots = (unsigned)p.n_slots;
#pragma unroll 1
        for (int kind = first; kind <= last; kind++) {
            const MegaStage st = p.stage[kind];
            const int wt = kind == MS_HEAD ? p.wt_head : p.wt_layer;
            int rows = kind == MS_QKV ? 2 * w.s1_n : kind == MS_WO ? p.rpb : kind == MS_UP ? p.ffn_rows * w.h_n : kind == MS_DOWN ? w.d_n : w.v_n;
            if (kind <= MS_WO && !w.in_group) rows = 0;
            const uint8_t* at = src;
#pragma unroll 1
            for (int r0 = 0; r0 < rows; r0 += st.group_rows) {
                const int ub = mega_unit_bytes(wt, min(st.group_rows, rows - r0));
#pragma unroll 1
                for (int u0 = 0; u0 < st.units; u0 += st.chunk_units) {
                    const unsigned bytes = (unsigned)(min(st.chunk_units, st.units - u0) * ub);
                    if (stopped()) return;  // nothing more is copied
                    if (issued >= n_slots) mega_wait(a, s, s.empty + c.slot, c.phase ^ 1u, 4);  // the previous use of the slot was released
                    if (stopped()) return;
                    mbar_expect_tx(s.full + c.slot, bytes);
                    bulk_copy_g2s(s.slots + (size_t)c.slot * p.slot_bytes, at, bytes, s.full + c.slot, policy);
                    at += bytes;
                    c.next(n_slots);
                    issued++;
                }
            }
            src += kind == MS_QKV ? p.s1_bytes : kind == MS_WO ? p.s2_bytes : kind == MS_UP ? p.s3a_bytes : p.s3b_bytes;
        }
    }
    // Every copy that was issued must have landed before the CTA may exit: walks the last n_slots chunks backwards.
    __device__ __forceinline__ void drain() {
        const unsigned n_slots = (unsigned)a.plan.n_slots, back = issued < n_slots ? issued : n_slots;
        MegaCursor k = c;
        for (unsigned i = 0; i < back; i++) {
            if (k.slot == 0) { k.slot = n_slots - 1; k.phase ^= 1u; } else k.slot--;
            unsigned spins = 0;
            while (!mbar_try_wait(s.full + k.slot, k.phase) && ++spins < kMegaSpinLimit) {}
        }
    }
};
__device__ __forceinline__ unsigned mega_layer_chunks(const MegaPlan& p, const MegaShare& w) {
    return (unsigned)((w.in_group ? mega_stage_chunks(p.stage[MS_QKV], 2 * w.s1_n) + mega_stage_chunks(p.stage[MS_WO], p.rpb) : 0) +
                      mega_stage_chunks(p.stage[MS_UP], p.ffn_rows * w.h_n) + mega_stage_chunks(p.stage[MS_DOWN], w.d_n));
}
// The watcher: follows the chunks in order and counts the ones whose bytes have arrived (one thread).
__device__ __forceinline__ void mega_watch(const MegaArgs& a, const MegaShared& s, unsigned total) {
    MegaCursor k;
    for (unsigned i = 0; i < total; i++) {
        unsigned spins = 0;
        while (!mbar_try_wait(s.full + k.slot, k.phase)) {
            if (*reinterpret_cast<volatile int*>(s.stop) || mega_spin_out(a, s, spins, 3)) return;
        }
        st_release_cta_shared(s.landed, i + 1);
        k.next((unsigned)a.plan.n_slots);
    }
}

template <int HD, int WT, bool GPT2>
__global__ void __launch_bounds__(kMegaThreads, 1) k_decode_mega(const __grid_constant__ MegaArgs a) {
    extern __shared__ __align__(128) uint8_t mega_smem[];
    const MegaPlan& p = a.plan;
    const MegaShared s = mega_carve(mega_smem, p);
    const ModelDims& m = a.m;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int L = m.n_layer;
    mega_init(a, s, 1);
    __syncthreads();
    const MegaShare& w = *s.share;

    if (warp == kMegaConsumerWarps) {
        // ---------------- producer: one thread streams this CTA's chunks in consumption order ----------------
        if (lane == 0) {
            const uint8_t* blob = a.pack + (size_t)blockIdx.x * p.cta_bytes;
            const uint8_t* head = blob + (long long)L * p.layer_bytes;
            uint64_t keep_policy;
            asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep_policy));
            // head bytes behind the first (n_slots - 1) chunks: what still has to come from memory when the head begins
            const long long head_bytes = mega_stage_bytes(p.stage[MS_HEAD], p.wt_head, w.v_n);
            const long long tail_off = min(head_bytes, (long long)(p.n_slots - 1) * p.stage[MS_HEAD].chunk_units * mega_unit_bytes(p.wt_head, min(w.v_n, p.stage[MS_HEAD].group_rows)));
            const long long tail_bytes = head_bytes - tail_off;
            MegaProducer prod(a, s);
            for (int step = a.first; step < a.first + a.n_steps && !prod.stopped(); step++) {  // (nothing for the steps behind the one that ended the loop)
                for (int l = 0; step > 0 && l < L; l++) {
                    // HBM idles during the layers (their weights are a full layer ahead in the ring): the part of the head
                    // that the ring cannot hold before the head begins is brought into L2 now, a slice per layer
                    if (tail_bytes > 0 && !prod.stopped()) {
                        const long long b0 = tail_bytes * l / L / 16 * 16, b1 = l + 1 == L ? tail_bytes : tail_bytes * (l + 1) / L / 16 * 16;
                        if (b1 > b0)
                            asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(head + tail_off + b0), "r"((unsigned)(b1 - b0)), "l"(keep_policy)
                                         : "memory");
                    }
                    prod.stages(blob + (long long)l * p.layer_bytes, MS_QKV, MS_DOWN, w);
                }
                prod.stages(head, MS_HEAD, MS_HEAD, w);
                // The ring is full and the consumers are a few chunks into the head: the one moment of a token at which a read of
                // host memory (a microsecond or two) holds nothing up.
                if (a.stop_request && blockIdx.x == 0) {
                    unsigned v;
                    asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(a.stop_request) : "memory");
                    if (v) *reinterpret_cast<volatile unsigned*>(s.asked) = 1u;
                }
            }
            prod.drain();
        }
        return;
    }
    if (warp == kMegaConsumerWarps + 1) {
        if (lane == 0)
            mega_watch(a, s, (unsigned)a.n_steps * mega_stage_chunks(p.stage[MS_HEAD], w.v_n) + (unsigned)(a.n_steps - 1 + a.first) * L * mega_layer_chunks(p, w));
        return;
    }

    // ---------------- consumers ----------------
    if (blockIdx.x == 0 && tid == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        a.stamps[0] = t;
    }
    MegaWorker<HD, WT, GPT2, 1> work(a, s);
    const MegaModel model{a.norms, a.tok_emb, a.kv};
    int pos = a.pos0;    // visible tokens
    uint32_t tok[1] = {a.tok0};
    int emitted = 0;
    unsigned seq = a.tag0;
    const int d = m.d_model;
    for (int step = a.first; step < a.first + a.n_steps; step++) {
        work.tracing = a.trace && (int)blockIdx.x == a.trace_cta && tid == 0 && step == a.first + a.n_steps - 1;
        if (!work.pass(model, m, step > 0 ? L : 0, tok, pos, seq, (unsigned long long)((a.cand0 + (unsigned)step) % 255u + 1u), tok)) {
            if (tid == 0) *reinterpret_cast<volatile int*>(s.stop) = 1;
            break;
        }
        if (step > 0) pos++;  // the token that was just processed is now visible
        const bool gpt2_stop = GPT2 && tok[0] == GPT2_EOS;  // GPT-2 rule: the stop token ends the loop without being emitted
        if (!gpt2_stop) emitted++;
        if (blockIdx.x == 0 && tid == 0 && !gpt2_stop) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (emitted == 1) a.stamps[1] = t;
            a.rs.out[emitted - 1] = tok[0];
            if (a.host_words) asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(a.host_words + emitted - 1), "l"(((unsigned long long)emitted << 32) | tok[0]) : "memory");
            if (a.token_times) a.token_times[emitted - 1] = t;
        }
        // Llama rule: the end-of-sequence token is emitted, then the loop stops (every CTA sees the same token)
        const bool eos = GPT2 ? gpt2_stop : m.eos_token >= 0 && tok[0] == (uint32_t)m.eos_token;
        if (eos || work.asked) {
            if (tid == 0) *reinterpret_cast<volatile int*>(s.stop) = 1;
            break;
        }
    }
    if (blockIdx.x == 0) {
        // the sequence's last hidden state (what the head just read)
        for (int k = tid; k < d; k += kMegaConsumers) a.hidden_io[k] = s.xres[k];
        if (tid == 0) {
            a.rs.pos[0] = pos;
            a.rs.tok[0] = tok[0];
            a.rs.next[0] = tok[0];
            a.rs.n_out[0] = emitted;
            a.stamps[2] = (unsigned long long)emitted | ((unsigned long long)tok[0] << 32);
            a.stamps[3] = (unsigned long long)pos;
        }
    }
    // The counted sums go back to zero for the next launch: the token exchange above proves that every contribution has
    // arrived and every CTA has read the last layer's totals.
    for (int k = w.d_begin + tid; k < w.d_begin + w.d_n; k += kMegaConsumers) a.mid_sums[k] = 0ull;
}

// ------------------------------------------------------------------------------------------------ pack builder

// One source matrix: row-major [rows][cols] fp16, or the split GGUF storage of the engine (Q8_0: int8 [rows][cols] +
// fp16 scales [rows][cols/32]; Q4_0: 16-byte nibble groups [rows][cols/32] + scales).
struct PackMatrix {
    const void* data;
    const __half* scales;
};
struct PackSources {
    const PackMatrix* wq;  // per-layer device arrays
    const PackMatrix* wk;
    const PackMatrix* wv;
    const PackMatrix* wo;
    const PackMatrix* w1;
    const PackMatrix* w2;
    const PackMatrix* w3;
    PackMatrix lm_head;
};

// Where a row starts: matrix `m` of `cols` columns, row `row`, first column `col0` (a multiple of 32).
struct PackRow {
    const uint8_t* data;     // null: a row of zeros
    const __half* scales;
};
__device__ __forceinline__ PackRow pack_row(int wt, const PackMatrix& m, int cols, size_t row, int col0) {
    PackRow r;
    const uint8_t* d = static_cast<const uint8_t*>(m.data);
    if (wt == WT_Q8_0) r.data = d + row * cols + col0;
    else if (wt == WT_Q4_0) r.data = d + (row * (cols / 32) + col0 / 32) * 16;
    else r.data = d + (row * cols + col0) * 2;
    r.scales = m.scales ? m.scales + row * (cols / 32) + col0 / 32 : nullptr;
    return r;
}

// Writes a stage's `rows` rows in the order the products read them: group by group of rows, chunk by chunk of K units, inside a
// chunk [unit][row][four pieces] and behind it, for the quantised types, the scales [unit][tile][g][rows g and g + 8 of the tile].
// fp16: piece t of a unit of 16 columns holds columns {2t, 2t+1, 2t+8, 2t+9} (the A registers of an m16n8k16 step for the lanes
// with that t).  Q8_0: the int8 of columns 4t..4t+3 and 16+4t..16+4t+3 of a block (the A registers of one m16n8k32 step); Q4_0:
// bytes 4t..4t+3 of the GGUF block, whose low and high nibbles are the same columns, as two's-complement nibbles (8 less).
// row_of(r) names the row's source.
template <class RowOf>
__device__ __forceinline__ void pack_stage(int wt, uint8_t* dst, const MegaStage& st, int rows, RowOf row_of) {
    const int piece = wt == WT_Q4_0 ? 4 : 8;
    for (int r0 = 0; r0 < rows; r0 += st.group_rows) {
        const int n = min(st.group_rows, rows - r0);
        for (int u0 = 0; u0 < st.units; u0 += st.chunk_units) {
            const int nu = min(st.chunk_units, st.units - u0);
            for (int i = threadIdx.x; i < nu * n * 4; i += blockDim.x) {
                const int t = i & 3, x = i >> 2, u = x / n, r = x - u * n;
                const PackRow src = row_of(r0 + r);
                uint8_t* out = dst + (size_t)i * piece;
                if (wt == WT_F16) {
                    uint2 v = make_uint2(0, 0);
                    if (src.data) {
                        const uint32_t* s32 = reinterpret_cast<const uint32_t*>(src.data + (size_t)(u0 + u) * 32);
                        v = make_uint2(s32[t], s32[t + 4]);
                    }
                    *reinterpret_cast<uint2*>(out) = v;
                } else if (wt == WT_Q8_0) {
                    uint2 v = make_uint2(0, 0);
                    if (src.data) {
                        const uint32_t* s32 = reinterpret_cast<const uint32_t*>(src.data + (size_t)(u0 + u) * 32);  // four columns each
                        v = make_uint2(s32[t], s32[4 + t]);
                    }
                    *reinterpret_cast<uint2*>(out) = v;
                } else {
                    uint32_t v = 0u;
                    if (src.data) v = reinterpret_cast<const uint32_t*>(src.data + (size_t)(u0 + u) * 16)[t] ^ 0x88888888u;
                    *reinterpret_cast<uint32_t*>(out) = v;
                }
            }
            if (wt != WT_F16) {
                const int padded = (n + 15) / 16 * 16;
                __half* sc = reinterpret_cast<__half*>(dst + (size_t)nu * mega_data_bytes(wt, n));
                for (int i = threadIdx.x; i < nu * padded; i += blockDim.x) {
                    const int u = i / padded, x = i - u * padded, r = (x & ~15) + ((x & 15) >> 1) + 8 * (x & 1);
                    __half v = __float2half(0.f);
                    if (r < n) {
                        const PackRow src = row_of(r0 + r);
                        if (src.data) v = src.scales[u0 + u];
                    }
                    sc[i] = v;
                }
            }
            dst += (size_t)nu * mega_unit_bytes(wt, n);
        }
    }
}

// One CTA builds the blob of one CTA of the decode kernel: per layer [S1 | S2 | S3 gate/up | S3 W2], then the head.
__global__ void k_build_pack(PackSources src, MegaPlan p, ModelDims m, uint8_t* pack) {
    const int cta = blockIdx.x;
    uint8_t* blob = pack + (size_t)cta * p.cta_bytes;
    const int d = m.d_model, hd = m.head_dim;
    const int wt = p.wt_layer;
    const MegaShare w = mega_share(m, p, cta);
    for (int l = 0; l < m.n_layer; l++) {
        uint8_t* base = blob + (size_t)l * p.layer_bytes;
        // S1: pairs of rows in RoPE order
        if (w.in_group)
            pack_stage(wt, base, p.stage[MS_QKV], 2 * w.s1_n, [&](int r) {
                int kind, row0, row1, idx;
                mega_s1_rows(m, p, w.kvh, w.s1_begin + (r >> 1), kind, row0, row1, idx);
                const PackMatrix& W = kind == 0 ? src.wq[l] : kind == 1 ? src.wk[l] : src.wv[l];
                return pack_row(wt, W, d, (size_t)((r & 1) ? row1 : row0), 0);
            });
        base += p.s1_bytes;
        // S2: rows [blk*rpb, +rpb) of Wo, columns of one head
        if (w.in_group)
            pack_stage(wt, base, p.stage[MS_WO], p.rpb, [&](int r) {
                const int orow = w.blk * p.rpb + r;
                return orow < d ? pack_row(wt, src.wo[l], m.q_dim, (size_t)orow, w.head * hd) : PackRow{nullptr, nullptr};
            });
        base += p.s2_bytes;
        // S3: (gate_j, up_j) row pairs
        const int fr = p.ffn_rows;
        pack_stage(wt, base, p.stage[MS_UP], fr * w.h_n, [&](int r) {
            return pack_row(wt, fr == 2 && (r & 1) ? src.w3[l] : src.w1[l], d, (size_t)(w.h_begin + (fr == 2 ? r >> 1 : r)), 0);
        });
        base += p.s3a_bytes;
        // S3: this CTA's rows of W2
        pack_stage(wt, base, p.stage[MS_DOWN], w.d_n, [&](int r) { return pack_row(wt, src.w2[l], m.hidden, (size_t)(w.d_begin + r), 0); });
    }
    pack_stage(p.wt_head, blob + (size_t)m.n_layer * p.layer_bytes, p.stage[MS_HEAD], w.v_n, [&](int r) { return pack_row(p.wt_head, src.lm_head, d, (size_t)(w.v_begin + r), 0); });
}

// GPT-2: W.b + bias of every row of a matrix [rows][K] (see MegaArgs::ln).  One warp per row.
__global__ void k_fold_norm(const uint16_t* w, int rows, int K, const float* b, const float* bias, float* out) {
    const int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    float sb = 0.f;
    for (int k = lane; k < K; k += 32) sb = fmaf(__half2float(__ushort_as_half(w[(size_t)r * K + k])), b[k], sb);
    sb = warp_sum(sb);
    if (lane == 0) out[r] = sb + (bias ? bias[r] : 0.f);
}

}  // namespace esp
