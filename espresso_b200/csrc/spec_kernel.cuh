// Exact two-token generation as ONE cooperative launch: a draft model proposes the token after `current`, the target
// model verifies `current` and the proposal in a single pass over its weights, and the commit rule of
// Sources/Espresso/GenerationHarness.swift:1281-1344 (commit two tokens when the proposal equals the target's own
// choice, otherwise one) runs inside the kernel, replicated in every CTA.  No host round trip separates the passes.
//
// The kernel is the persistent decode kernel (mega_kernel.cuh) widened to two token positions per pass:
//   * the products run on mma.sync with the weights as the A operand; the staged activations of the second position
//     occupy two more of the eight B columns the instruction computes anyway, so the weights are read from the ring
//     once for both positions and every position is summed in the single-position kernel's order;
//   * every exchange (tagged words, counted sums, arg-max candidates) carries one value per position;
//   * attention runs once per query; the second query also sees the first new position, whose key and value sit in
//     shared memory beside its own.
// Draft and target must have the same widths (d_model, heads, hidden, vocabulary, fp16 storage); they differ in depth
// only, so one plan and one ring serve both and a pass is a fixed sequence of weight chunks: draft layers, draft head,
// target layers, target head.  The draft always processes the two newest tokens (`prev`, `current`): when the
// previous pass committed one token the first of them was processed before, and writing the same key and value to the
// same cache row again is harmless; this keeps every pass the same shape.
#pragma once

#include "mega_kernel.cuh"

namespace esp {

constexpr int kSpecNP = 2;  // token positions per pass

struct SpecModel {
    ModelDims m;            // this model's dimensions (the KV-cache strides depend on its max_seq and sequence slots)
    const uint8_t* pack;    // [n_cta][cta_bytes] packed weights (see k_build_pack)
    long long cta_bytes;
    const float* norms;     // [2 * n_layer + 1][d_model]
    const uint16_t* tok_emb;
    KvLayout kv;
};

struct SpecArgs {
    MegaArgs base;          // target dimensions, the shared plan (shared-memory layout for two positions), rope table,
                            // exchange arena (every array holds two positions), error word, spin limit
    SpecModel model[2];     // 0 = draft, 1 = target
    uint32_t* out;          // emitted tokens; out[0 .. gen0) were written by the host
    int* result;            // [8]: tokens emitted in total, passes, committed, accepted, stopped on EOS, visible tokens of the
                            // target, visible tokens of the draft, row of the last target pass that produced the pending token
    float* hidden_out;      // [d_model] hidden state that produced the pending token (target), or null
    uint32_t prev, current; // the two newest tokens; `current` is emitted but not yet fed
    int pos;                // position of `current`
    int gen0;               // tokens emitted so far
    int eff;                // emission limit
    int max_seq;            // context limit (min over the two models)
    int eos_token;
    int verify_only;        // 1: a single target pass over (prev at pos, current at pos + 1), no draft, no loop: result[0..1] =
                            // the two greedy tokens, hidden_out[2][d_model] = both rows' hidden states (verify2 of the C ABI)
};

template <int HD>
__global__ void __launch_bounds__(kMegaThreads, 1) k_spec_mega(const __grid_constant__ SpecArgs sa) {
    constexpr int NP = kSpecNP;
    extern __shared__ __align__(128) uint8_t mega_smem[];
    const MegaArgs& a = sa.base;
    const MegaPlan& p = a.plan;
    const MegaShared s = mega_carve(mega_smem, p);
    const ModelDims& m = a.m;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    mega_init(a, s, NP);
    __syncthreads();
    const MegaShare& w = *s.share;
    const int max_passes = sa.verify_only ? 1 : sa.eff - sa.gen0;  // every pass emits at least one token
    const int first_model = sa.verify_only ? 1 : 0;

    if (warp == kMegaConsumerWarps) {
        // ---------------- producer: one thread streams this CTA's chunks in consumption order ----------------
        if (lane == 0) {
            MegaProducer prod(a, s);
            for (int pass = 0; pass < max_passes && !prod.stopped(); pass++) {
                for (int mi = first_model; mi < 2; mi++) {
                    const SpecModel& M = sa.model[mi];
                    const uint8_t* blob = M.pack + (size_t)blockIdx.x * M.cta_bytes;
                    for (int l = 0; l < M.m.n_layer; l++) prod.stages(blob + (long long)l * p.layer_bytes, MS_QKV, MS_DOWN, w);
                    prod.stages(blob + (long long)M.m.n_layer * p.layer_bytes, MS_HEAD, MS_HEAD, w);
                }
            }
            prod.drain();
        }
        return;
    }
    if (warp == kMegaConsumerWarps + 1) {
        if (lane == 0) {
            const unsigned layers = (unsigned)((first_model ? 0 : sa.model[0].m.n_layer) + sa.model[1].m.n_layer);
            mega_watch(a, s, (unsigned)max_passes * (layers * mega_layer_chunks(p, w) + (first_model ? 1u : 2u) * mega_stage_chunks(p.stage[MS_HEAD], w.v_n)));
        }
        return;
    }

    // ---------------- consumers ----------------
    MegaWorker<HD, WT_F16, false, NP> work(a, s);
    unsigned seq = 0;      // tag of everything the current layer publishes: layers are numbered through both models
    unsigned n_heads = 0;  // heads run so far (tag of the arg-max words)
    const int d = m.d_model;
    // ---- the generation loop (Sources/Espresso/GenerationHarness.swift:1281-1344; every CTA takes the same decisions)
    int gen = sa.gen0, total = sa.pos + 1;  // `current` sits at position sa.pos and has been emitted
    uint32_t prev = sa.prev, current = sa.current;
    int P = sa.pos;
    int passes = 0, committed = 0, accepted = 0, hit_eos = 0, row_sel = 0;
    int visible = sa.pos;  // tokens of the target's context that are committed
    int draft_visible = sa.pos;  // positions the draft has processed
    const bool writer = blockIdx.x == 0 && tid == 0;
    auto is_eos = [&](uint32_t t) { return sa.eos_token >= 0 && t == (uint32_t)sa.eos_token; };
    while (true) {
        const int remaining = min(sa.eff - gen, sa.max_seq - total);
        passes++;
        // verify-only launches (verify2 of the C ABI) take the target's pass alone: `prev` and `current` of the arguments
        // are then the two tokens to verify
        uint32_t proposed = sa.verify_only ? sa.current : 0u, next = 0, future = 0;
        if (sa.verify_only) current = sa.prev;
        bool gave_up = false;
        for (int mi = first_model; mi < 2 && !gave_up; mi++) {  // the only call site: the draft's pass, then the target's
            const SpecModel& M = sa.model[mi];
            ModelDims md = m;  // the widths are the target's; depth and cache strides are the model's own
            md.n_layer = M.m.n_layer; md.n_seq = M.m.n_seq; md.max_seq = M.m.max_seq;
            const uint32_t in[NP] = {mi ? current : prev, mi ? proposed : current};
            uint32_t o[NP];
            gave_up = !work.pass(MegaModel{M.norms, M.tok_emb, M.kv}, md, md.n_layer, in, mi ? P : P - 1, seq, (unsigned long long)(n_heads % 255 + 1), o);
            ++n_heads;
            if (mi == 0) { proposed = o[1]; draft_visible = P + 1; }
            else { next = o[0]; future = o[1]; }
        }
        if (gave_up) break;
        if (sa.verify_only) {
            // both greedy tokens and both rows' hidden states; nothing is committed or emitted
            if (blockIdx.x == 0) {
                if (sa.hidden_out)
                    for (int k = tid; k < NP * d; k += kMegaConsumers) sa.hidden_out[k] = s.xres[k];
                if (tid == 0) { sa.result[0] = (int)next; sa.result[1] = (int)future; }
            }
            if (tid == 0) *reinterpret_cast<volatile int*>(s.stop) = 1;
            return;
        }
        const bool two = remaining > 1 && total + 1 < sa.max_seq;
        if (two && proposed == next) {
            // both tokens are exact: the proposal is committed and emitted, the token after it becomes `current`
            if (writer) sa.out[gen] = next;
            gen++; total++;
            committed += 2; accepted += 1;
            visible = P + 2;
            row_sel = 1;
            if (is_eos(next)) { hit_eos = 1; break; }
            if (gen >= sa.eff || total >= sa.max_seq) break;
            prev = next; current = future; P += 2;
        } else {
            committed += 1;
            visible = P + 1;
            row_sel = 0;
            prev = current; current = next; P += 1;
        }
        if (writer) sa.out[gen] = current;
        gen++; total++;
        if (is_eos(current)) { hit_eos = 1; break; }
        if (gen >= sa.eff || total >= sa.max_seq) break;
    }
    if (tid == 0) *reinterpret_cast<volatile int*>(s.stop) = 1;
    if (blockIdx.x == 0) {
        if (sa.hidden_out)
            for (int k = tid; k < d; k += kMegaConsumers) sa.hidden_out[k] = s.xres[row_sel * d + k];
        if (tid == 0) {
            sa.result[0] = gen;
            sa.result[1] = passes;
            sa.result[2] = committed;
            sa.result[3] = accepted;
            sa.result[4] = hit_eos;
            sa.result[5] = visible;
            sa.result[6] = draft_visible;
            sa.result[7] = row_sel;
        }
    }
}

}  // namespace esp
