// Host side of pk100_gemm: argument validation, TMA tensor-map encoding and the
// dispatch table over (operand kind, tile width, swizzle, epilogue family).
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "gemm_sm100.cuh"
#include "pk100_internal.h"

namespace pk100 {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) ==
                cudaSuccess && qres == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(sym);
        }
    });
    return fn;
}

// Descriptor cache.  A tensor map is a pure function of (base, element size, extents, leading
// dimension, box, swizzle), and a host that runs the same layers on the same buffers request after
// request asks for the same few hundred maps again and again; encoding one costs a driver call.
// Direct-mapped table keyed by a hash of those fields, guarded by one mutex (launchers are
// thread-compatible, not thread-hot).  The 128-byte maps are copied out, so an evicted entry
// never invalidates a launch already issued.
struct MapKey {
    const void* base; uint64_t rows, cols, ld; int elem_bytes, box_rows, swizzle_bytes;
    bool operator==(const MapKey& o) const {
        return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld &&
               elem_bytes == o.elem_bytes && box_rows == o.box_rows && swizzle_bytes == o.swizzle_bytes;
    }
};
struct MapSlot { MapKey key; CUtensorMap map; bool used; };
constexpr int kMapSlots = 4096;
static MapSlot* g_map_slots = nullptr;
static std::mutex g_map_mutex;
static std::atomic<long long> g_map_hits{0}, g_map_misses{0};

static size_t map_hash(const MapKey& k) {
    uint64_t h = reinterpret_cast<uintptr_t>(k.base) * 0x9E3779B97F4A7C15ull;
    h ^= (k.rows * 0xC2B2AE3D27D4EB4Full) ^ (k.cols << 17) ^ (k.ld << 29);
    h ^= static_cast<uint64_t>(k.elem_bytes * 31 + k.box_rows * 7 + k.swizzle_bytes);
    h ^= h >> 29;
    return static_cast<size_t>(h * 0xBF58476D1CE4E5B9ull >> 32) % kMapSlots;
}

static int encode_map(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows,
                      uint64_t cols, uint64_t ld, int box_rows, int swizzle_bytes);

// 2-D row-major matrix [rows, cols] with `ld` elements between rows; box =
// [box_rows, swizzle_bytes / elem_bytes] elements, swizzle mode = box width.
static int make_map(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows,
                    uint64_t cols, uint64_t ld, int box_rows, int swizzle_bytes) {
    const MapKey key{base, rows, cols, ld, elem_bytes, box_rows, swizzle_bytes};
    const size_t slot = map_hash(key);
    {
        std::lock_guard<std::mutex> lock(g_map_mutex);
        if (g_map_slots == nullptr) g_map_slots = new MapSlot[kMapSlots]();
        MapSlot& s = g_map_slots[slot];
        if (s.used && s.key == key) {
            *map = s.map;
            g_map_hits.fetch_add(1, std::memory_order_relaxed);
            return PK100_OK;
        }
    }
    const int rc = encode_map(map, base, elem_bytes, rows, cols, ld, box_rows, swizzle_bytes);
    if (rc != PK100_OK) return rc;
    g_map_misses.fetch_add(1, std::memory_order_relaxed);
    std::lock_guard<std::mutex> lock(g_map_mutex);
    MapSlot& s = g_map_slots[slot];
    s.key = key; s.map = *map; s.used = true;
    return PK100_OK;
}

static int encode_map(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows,
                      uint64_t cols, uint64_t ld, int box_rows, int swizzle_bytes) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return PK100_ERR_DRIVER;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * static_cast<uint64_t>(elem_bytes)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(swizzle_bytes / elem_bytes),
                               static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem_strides[2] = {1, 1};
    const CUtensorMapDataType dtype =
        elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    const CUtensorMapSwizzle swz =
        swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    const CUresult res = fn(map, dtype, 2, const_cast<void*>(base), dims, strides, box,
                            elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return res == CUDA_SUCCESS ? PK100_OK : PK100_ERR_DRIVER;
}

// Tensor map of the output for the staged TMA store (256-column kernels, 128-column linear kernels): every epilogue
// warp owns 32 rows x (tile columns / 4); INT4 weights: 32 rows x 64 columns at a time.  Only slices with 64- or 128-byte rows leave that way
// (their swizzle modes); anything else keeps per-thread stores, and so does fp32 output, which the staging does not encode.
// Returns the row bytes or 0.
template <int Epi, int BlockN = 256, int BSrc = BSRC_TMA>
static int make_out_map(CUtensorMap* map, const GemmParams& p) {
    const int out_cols = Epi == EPI_GLU ? p.n / 2 : p.n;
    const int cols_per_warp = BSrc == BSRC_W4G128 ? 64 : (Epi == EPI_GLU ? BlockN / 2 : BlockN) / (GemmWarps<BSRC_TMA>::kEpilogue / 4);
    if (p.out_type == OUT_F32) return 0;
    const int obytes = p.out_type == OUT_F16 ? 2 : 1;
    const int row_bytes = cols_per_warp * obytes;
    if (row_bytes != 64 && row_bytes != 128) return 0;
    if (BSrc == BSRC_TMA && BlockN == 128 && row_bytes != 64) return 0;      // its staging holds 64-byte rows only
    if ((reinterpret_cast<uintptr_t>(p.out) & 15u) != 0) return 0;
    if ((static_cast<size_t>(p.ld_out) * obytes) % 16 != 0) return 0;
    if (make_map(map, p.out, obytes, p.m, out_cols, p.ld_out, 32, row_bytes) != PK100_OK) return 0;
    return row_bytes;
}

// Calls f(true or false type: the residual arrives by TMA, its tensor map).  It does where fp16 output leaves by TMA
// stores: the map has the boxes of the output slices.
template <int Epi, int BSrc, int BlockN, typename F>
static int with_residual(const GemmParams& p, const CUtensorMap& any, F&& f) {
    if constexpr (Epi == EPI_LINEAR && gemm_store_bytes<Epi, BSrc, BlockN>() > 0) {
        CUtensorMap map;
        if (p.residual != nullptr && p.store_row_bytes != 0 && p.out_type == OUT_F16 &&
            make_map(&map, p.residual, 2, p.m, p.n, p.ld_res, 32, p.store_row_bytes) == PK100_OK)
            return f(std::true_type{}, map);
    }
    return f(std::false_type{}, any);
}

// CTA pairs (cta_group::2) for the 256-column kernels.  Off by default, a validated alternative.  The pair path still
// issues both operands from one warp and its MMAs behind a branch, without a dependent launch; in that form, us at 45 056
// rows, pairs / one CTA per tile: fp16 output projection 92 / 102, FF contract 138 / 114, GLU 111 / 92.
static std::atomic<int> g_use_pairs{0};
extern "C" void pk100_set_gemm_cta_pairs(int enable) { g_use_pairs.store(enable != 0); }

// Process-wide cap on the persistent CTAs of a GEMM whose own max_ctas is <= 0 (0 = one per SM).
static std::atomic<int> g_dependent_launch{1};
static std::atomic<int> g_cta_cap{0};
extern "C" void pk100_set_gemm_cta_cap(int ctas) { g_cta_cap.store(ctas > 0 ? ctas : 0); }
static int shared_budget() {
    const int cap = g_cta_cap.load(std::memory_order_relaxed);
    return cap > 0 && cap < pk100_sm_count() ? cap : pk100_sm_count();
}
static int cta_budget(const pk100_gemm_args& a) { return a.max_ctas > 0 ? a.max_ctas : shared_budget(); }
extern "C" void pk100_set_dependent_launch(int enable) { g_dependent_launch.store(enable != 0); }
extern "C" void pk100_tensor_map_cache_stats(long long* hits, long long* misses) {
    if (hits != nullptr) *hits = g_map_hits.load(std::memory_order_relaxed);
    if (misses != nullptr) *misses = g_map_misses.load(std::memory_order_relaxed);
}

template <int Kind, int SwizzleBytes, int Epi>
static int launch_pair(const pk100_gemm_args& a, const GemmParams& p_in, cudaStream_t stream) {
    constexpr int BlockN = 256;
    using Smem = GemmSmem<BlockN / 2, SwizzleBytes, BlockN, gemm_store_bytes<Epi, BSRC_TMA, BlockN>()>;
    GemmParams p = p_in;
    constexpr int elem = Kind == KIND_F16 ? 2 : 1;
    CUtensorMap map_a, map_b;
    int rc = make_map(&map_a, a.a, elem, a.m, a.k, a.lda, kBlockM, SwizzleBytes);
    if (rc != PK100_OK) return rc;
    rc = make_map(&map_b, a.b, elem, a.n, a.k, a.ldb, BlockN / 2, SwizzleBytes);
    if (rc != PK100_OK) return rc;
    CUtensorMap map_out = map_a;
    p.store_row_bytes = make_out_map<Epi>(&map_out, p);
    const int m_groups = (a.m + 2 * kBlockM - 1) / (2 * kBlockM);
    const int n_tiles = (p.n + BlockN - 1) / BlockN;
    int pairs = cta_budget(a) / 2;
    if (pairs > m_groups * n_tiles) pairs = m_groups * n_tiles;
    if (pairs < 1) pairs = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(GemmWarps<BSRC_TMA>::kThreads);
    cfg.dynamicSmemBytes = Smem::kTotal;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return with_residual<Epi, BSRC_TMA, BlockN>(p, map_a, [&](auto res_tma, const CUtensorMap& map_res) -> int {
        constexpr auto kernel = gemm_kernel<Kind, BlockN, SwizzleBytes, Epi, BSRC_TMA, 2, decltype(res_tma)::value>;
        cudaError_t err = pk100_grant_smem<kernel>(Smem::kTotal);
        if (err != cudaSuccess) return static_cast<int>(err);
        err = cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, map_out, map_res, p);
        if (err != cudaSuccess) {
            cudaGetLastError();
            return static_cast<int>(err);
        }
        pk100_count_launch();
        return PK100_OK;
    });
}

template <int Kind, int BlockN, int SwizzleBytes, int Epi>
static int launch(const pk100_gemm_args& a, const GemmParams& p_in, cudaStream_t stream) {
    if constexpr (BlockN == 256) {
        if (g_use_pairs.load() != 0 && a.m > kBlockM) return launch_pair<Kind, SwizzleBytes, Epi>(a, p_in, stream);
    }
    using Smem = GemmSmem<BlockN, SwizzleBytes, BlockN, gemm_store_bytes<Epi, BSRC_TMA, BlockN>()>;
    GemmParams p = p_in;
    constexpr int elem = Kind == KIND_F16 ? 2 : 1;
    CUtensorMap map_a, map_b;
    int rc = make_map(&map_a, a.a, elem, a.m, a.k, a.lda, kBlockM, SwizzleBytes);
    if (rc != PK100_OK) return rc;
    // GLU: one box of values, one of gates
    rc = make_map(&map_b, a.b, elem, a.n, a.k, a.ldb, Epi == EPI_GLU ? BlockN / 2 : BlockN, SwizzleBytes);
    if (rc != PK100_OK) return rc;
    CUtensorMap map_out = map_a;
    if constexpr (gemm_store_bytes<Epi, BSRC_TMA, BlockN>() > 0) p.store_row_bytes = make_out_map<Epi, BlockN>(&map_out, p);
    const int m_tiles = (a.m + kBlockM - 1) / kBlockM;
    const int n_tiles = (p.n + BlockN - 1) / BlockN;
    int ctas = cta_budget(a);
    if (ctas > m_tiles * n_tiles) ctas = m_tiles * n_tiles;
    return with_residual<Epi, BSRC_TMA, BlockN>(p, map_a, [&](auto res_tma, const CUtensorMap& map_res) -> int {
        constexpr auto kernel = gemm_kernel<Kind, BlockN, SwizzleBytes, Epi, BSRC_TMA, 1, decltype(res_tma)::value>;
        const cudaError_t granted = pk100_grant_smem<kernel>(Smem::kTotal);
        if (granted != cudaSuccess) return static_cast<int>(granted);
        pk100_launch_chained(kernel, dim3(ctas), dim3(GemmWarps<BSRC_TMA>::kThreads), Smem::kTotal, stream, map_a, map_b, map_out, map_res, p);
        return pk100_launch_status();
    });
}

// fp16 activations x INT4 group-128 weights, dequantised in shared memory by producer warps.
static int launch_w4(const pk100_gemm_args& a, const GemmParams& p_in, cudaStream_t stream) {
    constexpr int BlockN = 128;
    constexpr int kMTiles = GemmWarps<BSRC_W4G128>::kMTiles;
    using Smem = GemmSmem<BlockN, 128, BlockN * kMTiles, gemm_store_bytes<EPI_LINEAR, BSRC_W4G128, BlockN>(), kBlockM * kMTiles,
                          gemm_code_bytes<BSRC_W4G128>()>;
    GemmParams p = p_in;
    CUtensorMap map_a, map_b;
    int rc = make_map(&map_a, a.a, 2, a.m, a.k, a.lda, kBlockM, 128);
    if (rc != PK100_OK) return rc;
    rc = make_map(&map_b, a.b, 1, a.n, a.k / 2, a.k / 2, BlockN, 128);        // the codes
    if (rc != PK100_OK) return rc;
    CUtensorMap map_out = map_a;
    p.store_row_bytes = make_out_map<EPI_LINEAR, BlockN, BSRC_W4G128>(&map_out, p);
    const int m_items = (a.m + kBlockM * kMTiles - 1) / (kBlockM * kMTiles);   // 256-row work items
    const int n_tiles = (p.n + BlockN - 1) / BlockN;
    int ctas = cta_budget(a);
    if (ctas > m_items * n_tiles) ctas = m_items * n_tiles;
    return with_residual<EPI_LINEAR, BSRC_W4G128, BlockN>(p, map_a, [&](auto res_tma, const CUtensorMap& map_res) -> int {
        constexpr auto kernel = gemm_kernel<KIND_F16, BlockN, 128, EPI_LINEAR, BSRC_W4G128, 1, decltype(res_tma)::value>;
        const cudaError_t granted = pk100_grant_smem<kernel>(Smem::kTotal);
        if (granted != cudaSuccess) return static_cast<int>(granted);
        pk100_launch_chained(kernel, dim3(ctas), dim3(GemmWarps<BSRC_W4G128>::kThreads), Smem::kTotal, stream, map_a, map_b, map_out, map_res, p);
        return pk100_launch_status();
    });
}

static bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

}  // namespace pk100

using namespace pk100;

int pk100_tensor_map_2d(void* map, const void* base, int elem_bytes, unsigned long long rows,
                        unsigned long long cols, unsigned long long ld, int box_rows, int swizzle_bytes) {
    return make_map(static_cast<CUtensorMap*>(map), base, elem_bytes, rows, cols, ld, box_rows, swizzle_bytes);
}

int pk100_cta_budget() { return pk100::shared_budget(); }

bool pk100_dependent_launch_enabled() { return pk100::g_dependent_launch.load(std::memory_order_relaxed) != 0; }

static std::atomic<long long> g_launches{0};
void pk100_count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
extern "C" long long pk100_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

extern "C" int pk100_gemm(void* stream_v, const pk100_gemm_args* a) { return pk100_gemm_chained(stream_v, a, false); }

int pk100_gemm_chained(void* stream_v, const pk100_gemm_args* a, bool b_settled) {
    if (a == nullptr || a->a == nullptr || a->b == nullptr || a->out == nullptr) return PK100_ERR_NULL;
    if (a->m < 0 || a->n <= 0 || a->k <= 0) return PK100_ERR_SHAPE;
    if (a->m == 0) return PK100_OK;
    if (a->kind < PK100_KIND_F16 || a->kind > PK100_KIND_F16_W4G128) return PK100_ERR_UNSUPPORTED;
    const bool w4 = a->kind == PK100_KIND_F16_W4G128;
    const int elem = (a->kind == PK100_KIND_F16 || w4) ? 2 : 1;
    if ((static_cast<long long>(a->k) * elem) % 16 != 0 ||
        (static_cast<long long>(a->lda) * elem) % 16 != 0 || a->lda < a->k)
        return PK100_ERR_SHAPE;
    if (!w4 && ((static_cast<long long>(a->ldb) * elem) % 16 != 0 || a->ldb < a->k)) return PK100_ERR_SHAPE;
    if (w4) {
        if (a->b_group_scales == nullptr) return PK100_ERR_NULL;
        if (a->k % 128 != 0 || a->epilogue != PK100_EPI_LINEAR || a->keep_in != nullptr)
            return PK100_ERR_SHAPE;
    }
    if (a->n % 32 != 0) return PK100_ERR_SHAPE;
    if (!aligned16(a->a) || !aligned16(a->b) || !aligned16(a->out)) return PK100_ERR_ALIGN;
    if (a->out_type < PK100_OUT_F16 || a->out_type > PK100_OUT_S8) return PK100_ERR_UNSUPPORTED;
    const int out_elem = a->out_type == PK100_OUT_F16 ? 2 : (a->out_type == PK100_OUT_F32 ? 4 : 1);
    const int out_cols = a->epilogue == PK100_EPI_GLU ? a->n / 2 : a->n;
    if (a->ld_out < out_cols || (static_cast<long long>(a->ld_out) * out_elem) % 16 != 0)
        return PK100_ERR_SHAPE;
    if (a->residual != nullptr) {
        if (!aligned16(a->residual)) return PK100_ERR_ALIGN;
        if (a->ld_res < out_cols || a->ld_res % 8 != 0) return PK100_ERR_SHAPE;
        if (a->epilogue != PK100_EPI_LINEAR) return PK100_ERR_UNSUPPORTED;
    }
    if (a->keep_in != nullptr) {
        if (elem != 1 || a->k % 64 != 0 || a->k > 4096) return PK100_ERR_SHAPE;
    }
    if (a->epilogue == PK100_EPI_GLU && (a->n % 128 != 0)) return PK100_ERR_SHAPE;
    if (a->epilogue == PK100_EPI_SPARSE_OUT) {
        if (a->keep_out == nullptr) return PK100_ERR_NULL;
        if (a->n % 64 != 0 || a->out_type != PK100_OUT_S8) return PK100_ERR_SHAPE;
    }

    GemmParams p{};
    p.m = a->m;
    p.n = a->n;
    p.k = a->k;
    p.row_scales = a->row_scales;
    p.row_scale = a->row_scale;
    p.col_scales = a->col_scales;
    p.bias = a->bias;
    p.act = a->act;
    p.residual = static_cast<const __half*>(a->residual);
    p.ld_res = a->ld_res;
    p.alpha = a->alpha;
    p.valid_rows = a->valid_rows > 0 ? a->valid_rows : a->m;
    p.out = a->out;
    p.ld_out = a->ld_out;
    p.out_type = a->out_type;
    p.out_scale = a->out_scale;
    p.tau = a->tau;
    p.keep_out = a->keep_out;
    p.stats_out = a->stats_out;
    p.keep_in = a->keep_in;
    p.w4_scales = w4 ? static_cast<const __half*>(a->b_group_scales) : nullptr;
    p.status = a->status;
    p.b_settled = b_settled ? 1 : 0;
    // Where A and the output do not share L2 (126 MB) with room to spare, walking the row tiles inside would stream
    // A from HBM once per column tile.  us at 45 056 rows, row tiles inside / column tiles inside: FF expand
    // 195 / 189, QKV 160 / 149, fp16 output projection 116 / 105, GLU 105 / 95, pointwise-2 87 / 78, INT4 1024 -> 4096
    // 555 / 520; at 6144 rows 29.2 / 29.3, 22.7 / 22.8, 21.5 / 22.0, 16.9 / 17.0, 16.7 / 17.0, 81.0 / 80.6.
    p.n_inner = static_cast<long long>(a->m) * (static_cast<long long>(a->k) * elem + static_cast<long long>(out_cols) * out_elem) > (64ll << 20) ? 1 : 0;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

    // Tile width: the one with the shorter schedule, counting whole waves over the CTAs available and a
    // 128-column tile as 0.7 of a 256-column one (measured: at 3072 x 1024 one wave of 96 wide tiles
    // takes 17.6 us against 20.3 us for two waves of 192 narrow ones; at 6144 x 1024 two wide waves
    // take 24.3 us against 28.7 us for three narrow ones; a single partial wave prefers the narrow tile).
    const int m_tiles = (a->m + kBlockM - 1) / kBlockM;
    // 64-column tiles where they still fit one wave: such a launch is bound by the round trips of its operand
    // ring (1.7 us each, the weights come from DRAM), and eight 24 KB stages hold a K of 1024 bytes whole where
    // the 128-column tile has five stages, for twice the CTAs and half the epilogue.  Encoder of a 4 s request
    // (128 rows, 24 layers, GLU rule below included) 340 us shorter, of a 60 s one (768 rows) 210 us; back to back,
    // 128-column tiles against these: FF contract with a 30 % live K 13.8 / 12.2 us at 128 rows, 12.9 / 11.0 at 512,
    // 13.6 / 12.1 at 1024; K = 1024 INT8 6.4 / 5.8, 6.6 / 5.9, 6.8 / 6.1.
    const bool tiny = a->n % 64 == 0 && static_cast<long long>(m_tiles) * (a->n / 64) <= cta_budget(*a);
    bool narrow = a->n % 256 != 0;
    if (!narrow) {
        const long long ctas = cta_budget(*a);
        const long long wide = (static_cast<long long>(m_tiles) * (a->n / 256) + ctas - 1) / ctas;
        const long long thin = (static_cast<long long>(m_tiles) * (a->n / 128) + ctas - 1) / ctas;
        narrow = thin * 7 < wide * 10;
    }

    if (w4) return launch_w4(*a, p, stream);
    switch (a->epilogue) {
    case PK100_EPI_LINEAR:
        if (tiny) {
            if (a->kind == PK100_KIND_F16) return launch<KIND_F16, 64, 128, EPI_LINEAR>(*a, p, stream);
            if (a->kind == PK100_KIND_E4M3) return launch<KIND_F8, 64, 128, EPI_LINEAR>(*a, p, stream);
            return launch<KIND_I8, 64, 128, EPI_LINEAR>(*a, p, stream);
        }
        if (a->kind == PK100_KIND_F16) {
            return narrow ? launch<KIND_F16, 128, 128, EPI_LINEAR>(*a, p, stream)
                          : launch<KIND_F16, 256, 128, EPI_LINEAR>(*a, p, stream);
        }
        if (a->kind == PK100_KIND_E4M3) {
            return narrow ? launch<KIND_F8, 128, 128, EPI_LINEAR>(*a, p, stream)
                          : launch<KIND_F8, 256, 128, EPI_LINEAR>(*a, p, stream);
        }
        // A tile-sparse A operand (keep_in) runs on the same 128-byte K blocks: a block is skipped
        // when both of its 64-wide sparsity tiles are dead (dead tiles hold zeros, so a half-dead
        // block is computed correctly).  64-byte K blocks matched the skip granularity but
        // measured 14 % slower: TMA moves rows of a box at the same rate whatever their width.
        return narrow ? launch<KIND_I8, 128, 128, EPI_LINEAR>(*a, p, stream)
                      : launch<KIND_I8, 256, 128, EPI_LINEAR>(*a, p, stream);
    case PK100_EPI_GLU: {
        // 128-column tiles (64 values and their gates) likewise only in one wave
        const bool thin_glu = a->n % 256 != 0 || static_cast<long long>(m_tiles) * (a->n / 128) <= cta_budget(*a);
        if (a->kind == PK100_KIND_E4M3) {
            return thin_glu ? launch<KIND_F8, 128, 128, EPI_GLU>(*a, p, stream)
                                     : launch<KIND_F8, 256, 128, EPI_GLU>(*a, p, stream);
        }
        if (a->kind == PK100_KIND_F16) {
            return thin_glu ? launch<KIND_F16, 128, 128, EPI_GLU>(*a, p, stream)
                                     : launch<KIND_F16, 256, 128, EPI_GLU>(*a, p, stream);
        }
        return PK100_ERR_UNSUPPORTED;
    }
    case PK100_EPI_SPARSE_OUT:
        if (a->kind == PK100_KIND_E4M3) {
            // narrower tiles where they still fit one wave, as above: 8.1 -> 6.4 us at 128 and 256 rows (64 columns
            // each), 8.2 -> 7.3 at 512 (128)
            if (static_cast<long long>(m_tiles) * (a->n / 64) <= cta_budget(*a)) return launch<KIND_F8, 64, 128, EPI_SPARSE_OUT>(*a, p, stream);
            if (a->n % 128 == 0 && static_cast<long long>(m_tiles) * (a->n / 128) <= cta_budget(*a))
                return launch<KIND_F8, 128, 128, EPI_SPARSE_OUT>(*a, p, stream);
            return launch<KIND_F8, 256, 128, EPI_SPARSE_OUT>(*a, p, stream);
        }
        if (a->kind == PK100_KIND_F16) return launch<KIND_F16, 256, 128, EPI_SPARSE_OUT>(*a, p, stream);
        return PK100_ERR_UNSUPPORTED;
    default:
        return PK100_ERR_UNSUPPORTED;
    }
}
