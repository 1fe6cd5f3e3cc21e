// Which kernels serve a pass over the model.  Plain C++ without CUDA, so that the rule can be checked on the host.
#pragma once

namespace esp {

// Rows of a pass, decode batch or prompt, that take the streamed products; more rows take the products on 128- and 256-row
// tiles.  A streamed product reads the weights once per 64 rows (through L2 from the second time on) and cuts small matrices
// along K; the tiles read them once per 128 or 256 rows.  us per pass,
// streamed / tiles, prompts: d_model 768 700 rows 803 / 866; 2048 (22 layers) 192 rows 1462 / 1570, 224 rows 1925 / 1610; 4096 (4 layers)
// 64 rows 478 / 545, 100 rows 663 / 552.
constexpr int sg_rows(int d_model) { return d_model <= 1024 ? 704 : d_model <= 2048 ? 192 : 64; }

// Words of a pinned pass slot in front of its int4 lists: six control words per row, rounded up to 16 bytes (an engine of an odd
// number of sequences has an odd number of rows).
constexpr unsigned long long slot_row_words(int max_rows) { return (6ull * (unsigned)max_rows + 3) / 4 * 4; }

enum StepPath {
    PATH_ROWWISE,  // one kernel per stage on the stored weights, any row count
    PATH_STREAM,   // streamed products
    PATH_TILES,    // products on 256-row tiles of SM pairs or 128-row tiles of single SMs
    PATH_REFUSED,  // a tensor-parallel rank without tensor-core operands: only the two batched paths sum over the ranks
};

// tc_ready: the model has 16-bit tensor-core operands, or (quantised) can build them.
inline StepPath step_path(bool tc_ready, bool quantised, int tp_size, int d_model, int rows) {
    if (!tc_ready) return tp_size > 1 ? PATH_REFUSED : PATH_ROWWISE;
    // A quantised model's single rows stay on the kernels that read the GGUF blocks themselves (the persistent kernel and the
    // row-wise ones): an engine that only ever decodes one sequence then never builds the fp16 expansion.  A tensor-parallel
    // rank holds a slice of every matrix, and the row-wise kernels neither sum over the ranks nor know the vocabulary shard.
    if (quantised && rows == 1 && tp_size <= 1) return PATH_ROWWISE;
    return rows <= sg_rows(d_model) ? PATH_STREAM : PATH_TILES;
}

}  // namespace esp
