// Which kernels serve a pass over the model.  Plain C++ without CUDA, so that the rule can be checked on the host.
#pragma once

namespace esp {

// Rows of a pass that take the streamed products; wider passes take the products on SM pairs.  Decode batches (one position per
// sequence) up to kSgMaxRows.  Prompt passes, whose attention is the same tiled kernel either way, cross where a second or
// third read of the weights by the 64-row tiles costs more than idle pairs: measured (us, streamed / pairs) 1.1B 160 rows 1500 /
// 1590, 200 rows 1925 / 1657, 300 rows 2290 / 2110; 8 layers of 8B 100 rows 1310 / 1310, 144 rows 1675 / 1318; GPT-2 300 rows
// 662 / 800, 512 rows 771 / 892, 700 rows 908 / 945, 768 rows 934 / 943.
constexpr int kSgMaxRows = 320, kSgMaxRowsWide = 192;  // decode: d_model <= 2048 / above
constexpr int sg_decode_rows(int d_model) { return d_model <= 2048 ? kSgMaxRows : kSgMaxRowsWide; }
constexpr int sg_prompt_rows(int d_model) { return d_model <= 1024 ? 704 : d_model <= 2048 ? 192 : 128; }

enum StepPath {
    PATH_ROWWISE,  // one kernel per stage on the stored weights, any row count
    PATH_STREAM,   // streamed products
    PATH_PAIRS,    // products on SM pairs
    PATH_REFUSED,  // a tensor-parallel rank without tensor-core operands: only the two batched paths sum over the ranks
};

// tc_ready: the model has 16-bit tensor-core operands, or (quantised) can build them.  tiled: a prompt pass with the tiled attention.
inline StepPath step_path(bool tc_ready, bool quantised, int tp_size, int d_model, int rows, bool tiled) {
    if (!tc_ready) return tp_size > 1 ? PATH_REFUSED : PATH_ROWWISE;
    // A quantised model's single rows stay on the kernels that read the GGUF blocks themselves (the persistent kernel and the
    // row-wise ones): an engine that only ever decodes one sequence then never builds the fp16 expansion.  A tensor-parallel
    // rank holds a slice of every matrix, and the row-wise kernels neither sum over the ranks nor know the vocabulary shard.
    if (quantised && rows == 1 && tp_size <= 1) return PATH_ROWWISE;
    return rows <= (tiled ? sg_prompt_rows(d_model) : sg_decode_rows(d_model)) ? PATH_STREAM : PATH_PAIRS;
}

}  // namespace esp
