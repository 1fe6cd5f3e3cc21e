// Host side of the tensor-core GEMM: TMA tensor maps, launch dispatch over the batch tile width, and the
// stand-alone entry point used for parity checks and tensor-pipe measurements.
#include "engine.h"
#include "pair_gemm.cuh"

namespace esp {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// 2-D map over a row-major [rows, cols] matrix of 16-bit elements: boxes of 64 columns x box_rows rows, 128-byte
// swizzle, out-of-range elements read as zero.
int32_t tc_make_map(CUtensorMap* map, const void* base, bool bf16, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return esp::fail(ESP_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    if (cols % 8 != 0 || (reinterpret_cast<uintptr_t>(base) & 15)) return esp::fail(ESP_CUDA_ERR_INVALID_ARGUMENT, "tensor map: base or row pitch not 16-byte aligned");
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)kTcBlockK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), gdim, gstride, box,
                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        std::ostringstream os;
        os << "cuTensorMapEncodeTiled failed with code " << (int)r;
        return esp::fail(ESP_CUDA_ERR_CUDA, os.str());
    }
    return ESP_CUDA_OK;
}

// Launch shape of a streamed product: w_tiles 128-row weight tiles, K of kb 64-wide blocks, `rows` batch rows in `parts`
// 16-bit parts.  K slices: as many as fit two CTAs per SM with some room for the placement of clusters.  Measured (fp16, us
// per launch in a warm chain; 1 slice -> rule): 2048 x 2048, 5 rows 13.8 -> 6.7 (8); 11264 x 2048 15.7 -> 11.5 (3);
// 6144 x 4096, 1 row 30.7 -> 12.5 (5); 28672 x 4096 43 (1).  One slice more than the SMs can place costs a whole wave
// (6144 x 4096 in 6 slices: 21.7).
SgPlan sg_plan(int w_tiles, int rows, int kb, int parts, bool may_split, int sms) {
    SgPlan p;
    p.parts = parts;
    p.n_cols = parts > 1 ? (parts == 2 ? 16 : 32) : std::min((rows + 15) / 16 * 16, kSgMaxCols);
    p.col_tiles = parts > 1 ? 1 : (rows + p.n_cols - 1) / p.n_cols;
    p.row_tiles = w_tiles;
    const int tiles = std::max(1, w_tiles * p.col_tiles);
    int want = may_split ? std::max(1, std::min(kSgMaxSplits, sms * 9 / 5 / tiles)) : 1;
    // Pairs of CTAs find a place on nearly every SM, larger clusters do not: us per launch, with one slice less / this many: 20 x 6
    // tiles in 2 slices (240 CTAs) 14.1 / 11.5, 16 x 4 in 4 (256) 9.6 / 9.4, 24 x 6 in 2 (288) 10.4 / 9.2, 16 x 6 in 3 (288) 11.7 / 16.7.
    if (may_split && want == 1 && tiles <= sms - 4) want = 2;
    want = std::min(want, std::max(1, kb / 2));
    p.kb_per_split = (kb + want - 1) / want;
    p.splits = (kb + p.kb_per_split - 1) / p.kb_per_split;
    const int stage = kSgWBytes + p.n_cols * 128;
    const int own = ((parts > 1 ? 8 : p.n_cols) + p.splits - 1) / p.splits;
    const int exchange = p.splits * parts * own * kSgRows * 4;  // overlays the ring when there is one slice
    const int room = kSgSmemBudget - 1024 - (p.splits > 1 ? exchange : 0);
    p.stages = std::max(1, std::min(std::min(kSgMaxStages, p.kb_per_split), room / stage));
    p.smem = (p.splits > 1 ? p.stages * stage + exchange : std::max(p.stages * stage, exchange)) + 1024;
    return p;
}

static cudaError_t sg_configure() {
    static std::mutex mu;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0 || dev >= 64 || configured[dev]) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    for (auto k : {k_gemm_stream<false>, k_gemm_stream<true>}) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSgSmemBudget + 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    configured[dev] = e == cudaSuccess;
    return e;
}

// mw: 64-row maps of the group's matrices (unused slots repeat slot 0); mx: map of the operand rows with n_cols-row boxes
// (ignored when the operand is staged from the residual stream).
cudaError_t sg_launch(const SgPlan& plan, int epilogue, const CUtensorMap* const* mw, const CUtensorMap& mx, SgArgs a, cudaStream_t s) {
    cudaError_t e = sg_configure();
    if (e != cudaSuccess) return e;
    int halves = 0;
    for (int g = 0; g < a.n_groups; g++) { a.g[g].half0 = halves; halves += (a.g[g].M + kSgHalf - 1) / kSgHalf; }
    a.kb_per_split = plan.kb_per_split; a.n_cols = plan.n_cols; a.parts = plan.parts; a.stages = plan.stages; a.epilogue = epilogue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.col_tiles, plan.row_tiles, plan.splits);
    cfg.blockDim = dim3(kSgThreads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = plan.splits;
    cfg.attrs = attr;
    cfg.numAttrs = plan.splits > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, a.bf16 ? k_gemm_stream<true> : k_gemm_stream<false>, *mw[0], *mw[1], *mw[2], mx, a);
}

// Launch shape of a product on tiles: of SM pairs or of single SMs.
struct PgShape { bool pair; int tiles_n, splits, kb_per_split, units; float cost; };
// The work of the busiest SM or pair in K blocks of a pair (about 0.28 us); K slices of a residual product are the ones that make
// it least, a sliced unit's epilogue and its atomics counted as 8 blocks.
static PgShape pg_shape_of(bool pair, int rows, int tiles_w, int kb, bool may_split, int sms) {
    PgShape p{};
    p.pair = pair;
    p.tiles_n = (rows + (pair ? 255 : 127)) / (pair ? 256 : 128);
    const int tiles = p.tiles_n * tiles_w, lanes = pair ? sms / 2 : sms;
    p.cost = 1e30f;
    for (int want = 1; want <= (may_split ? 8 : 1); want++) {
        const int per = (kb + want - 1) / want, n = (kb + per - 1) / per;
        const float cost = (float)((tiles * n + lanes - 1) / lanes) * (float)(per + (n > 1 ? 8 : 0));
        if (cost < p.cost) { p.cost = cost; p.splits = n; p.kb_per_split = per; p.units = tiles * n; }
    }
    return p;
}
static PgShape pg_shape(int rows, int tiles_w, int kb, bool may_split, int sms) {
    const PgShape pair = pg_shape_of(true, rows, tiles_w, kb, may_split, sms), single = pg_shape_of(false, rows, tiles_w, kb, may_split, sms);
    // Fitted to the times of twelve shapes at 33 to 2048 rows (2 x 14336 x 4096: pairs 22 + 17.8 us a wave, single SMs 18 + 23.1; 2 x
    // 5632 x 2048: 10 + 9.3, 8 + 12): the better one of the two, or within 3 % of it, except for 4096 x 4096 at 1600 rows (12 %).
    return single.cost * 1.28f < pair.cost + 7.f ? single : pair;
}

// mw: 128-row maps of the group's matrices (unused slots repeat slot 0); mx: map of the operand rows with 128-row boxes.
cudaError_t pg_launch(const CUtensorMap* const* mw, const CUtensorMap& mx, PgArgs a, int sms, cudaStream_t s) {
    static std::mutex mu;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev >= 0 && dev < 64 && !configured[dev]) {
            cudaError_t e = cudaFuncSetAttribute(k_gemm_pair<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PgTile<true>::kSmemBytes);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gemm_pair<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PgTile<false>::kSmemBytes);
            for (auto k : {k_gemm_pair<true>, k_gemm_pair<false>})
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return e;
            configured[dev] = true;
        }
    }
    int halves = 0;
    const int groups = a.epilogue == PG_SWIGLU ? 1 : a.n_groups;
    for (int g = 0; g < groups; g++) { a.g[g].half0 = halves; halves += (a.g[g].M + 127) / 128; }
    a.tiles_w = a.epilogue == PG_SWIGLU ? halves : (halves + 1) / 2;
    const int kb = a.K / kTcBlockK;
    const PgShape shape = pg_shape(a.rows, a.tiles_w, kb, a.epilogue == PG_RESIDUAL, sms);
    a.tiles_n = shape.tiles_n;
    a.splits = shape.splits;
    a.kb_per_split = shape.kb_per_split;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(shape.pair ? 2 * std::min(sms / 2, shape.units) : std::min(sms, shape.units));
    cfg.blockDim = dim3(kPgThreads);
    cfg.dynamicSmemBytes = shape.pair ? PgTile<true>::kSmemBytes : PgTile<false>::kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = shape.pair ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, shape.pair ? k_gemm_pair<true> : k_gemm_pair<false>, *mw[0], *mw[1], *mw[2], mx, a);
}

__global__ void k_f32_to_16(const float* src, int64_t n, uint16_t* dst, int bf16) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (bf16) dst[i] = __bfloat16_as_ushort(__float2bfloat16_rn(src[i]));
    else dst[i] = __half_as_ushort(__float2half_rn(src[i]));
}

// Y[n][m] = sum_k W[m][k] * X16[n][k], X16 = X rounded to the weights' 16-bit type.  W, X, Y are host pointers.
int32_t gemm_tc_bench(int32_t type, const void* w, int32_t M, int32_t K, const float* x, int32_t N, float* y, int32_t warmup,
                      int32_t iterations, float* avg_ms, int32_t device) {
    if (!w || !x || !y || M < 1 || N < 1 || N > 256 || K < kTcBlockK || K % kTcBlockK != 0 || iterations < 1)
        return esp::fail(ESP_CUDA_ERR_INVALID_ARGUMENT, "gemm_tc_bench: need 1 <= N <= 256 and K a multiple of 64");
    if (type != WT_F16 && type != WT_BF16) return esp::fail(ESP_CUDA_ERR_INVALID_ARGUMENT, "gemm_tc_bench: fp16 or bf16 weights only");
    if (force_failure_enabled()) return esp::fail(ESP_CUDA_ERR_FORCED_FAILURE, "forced failure is enabled");
    ESP_CUDA_TRY(cudaSetDevice(device));
    const int alloc_rows = (N + 15) / 16 * 16;
    const int ldo = (M + 3) / 4 * 4;  // the kernel stores four weight rows at a time
    std::vector<void*> owned;
    auto cleanup = [&] { for (void* p : owned) cudaFree(p); };
    auto body = [&]() -> int32_t {
        void *dw = nullptr, *dx16 = nullptr;
        float *dx = nullptr, *dy = nullptr;
        int* derr = nullptr;
        ESP_CUDA_TRY(cudaMalloc(&dw, (size_t)M * K * 2)); owned.push_back(dw);
        ESP_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&dx), sizeof(float) * (size_t)N * K)); owned.push_back(dx);
        ESP_CUDA_TRY(cudaMalloc(&dx16, (size_t)alloc_rows * K * 2)); owned.push_back(dx16);
        ESP_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&dy), sizeof(float) * (size_t)N * ldo)); owned.push_back(dy);
        ESP_CUDA_TRY(cudaMalloc(reinterpret_cast<void**>(&derr), sizeof(int))); owned.push_back(derr);
        ESP_CUDA_TRY(cudaMemcpy(dw, w, (size_t)M * K * 2, cudaMemcpyDefault));
        ESP_CUDA_TRY(cudaMemcpy(dx, x, sizeof(float) * (size_t)N * K, cudaMemcpyDefault));
        ESP_CUDA_TRY(cudaMemset(dx16, 0, (size_t)alloc_rows * K * 2));
        ESP_CUDA_TRY(cudaMemset(derr, 0, sizeof(int)));
        const int64_t nx = (int64_t)N * K;
        k_f32_to_16<<<(unsigned)((nx + 255) / 256), 256>>>(dx, nx, static_cast<uint16_t*>(dx16), type == WT_BF16);
        ESP_CUDA_TRY(cudaGetLastError());
        CUtensorMap mw, mx;
        int32_t rc;
        if ((rc = tc_make_map(&mw, dw, type == WT_BF16, M, K, kSgHalf))) return rc;
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        // the plan the decode engine would use for a product of this shape, with the batch rows rounded to 16 bits
        const SgPlan plan = sg_plan((M + kSgRows - 1) / kSgRows, N, K / kTcBlockK, 1, true, sms);
        if ((rc = tc_make_map(&mx, dx16, type == WT_BF16, alloc_rows, K, plan.n_cols))) return rc;
        const CUtensorMap* maps[3] = {&mw, &mw, &mw};
        SgArgs a{};
        a.n_groups = 1;
        a.g[0].M = M; a.g[0].out = dy; a.g[0].ldo = ldo;
        a.K = K; a.rows = N; a.all_rows = 1; a.error = derr; a.bf16 = type == WT_BF16;
        auto launch = [&]() -> cudaError_t { return sg_launch(plan, SG_STORE, maps, mx, a, nullptr); };
        for (int i = 0; i < warmup; i++) ESP_CUDA_TRY(launch());
        cudaEvent_t e0, e1;
        ESP_CUDA_TRY(cudaEventCreate(&e0));
        ESP_CUDA_TRY(cudaEventCreate(&e1));
        ESP_CUDA_TRY(cudaDeviceSynchronize());
        ESP_CUDA_TRY(cudaEventRecord(e0));
        for (int i = 0; i < iterations; i++) ESP_CUDA_TRY(launch());
        ESP_CUDA_TRY(cudaEventRecord(e1));
        cudaError_t e = cudaEventSynchronize(e1);
        float total = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&total, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        ESP_CUDA_TRY(e);
        if (avg_ms) *avg_ms = total / iterations;
        int herr = 0;
        ESP_CUDA_TRY(cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost));
        if (herr) return esp::fail(ESP_CUDA_ERR_TIMEOUT, "tensor-core GEMM gave up waiting on a barrier");
        ESP_CUDA_TRY(cudaMemcpy2D(y, sizeof(float) * M, dy, sizeof(float) * ldo, sizeof(float) * M, N, cudaMemcpyDeviceToHost));
        return ESP_CUDA_OK;
    };
    int32_t rc = body();
    cleanup();
    return rc;
}

}  // namespace esp

extern "C" int32_t esp_cuda_gemm_tc_bench(int32_t type, const void* weights, int32_t rows, int32_t cols, const float* x, int32_t n, float* y,
                                          int32_t warmup, int32_t iterations, float* avg_ms, int32_t device) {
    return esp::gemm_tc_bench(type, weights, rows, cols, x, n, y, warmup, iterations, avg_ms, device);
}
