// Host side of the tensor-core Linear kernel (tc_kernel.cuh): tensor maps, launch plans, launch parameters.
#include "tc_kernel.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace kb {

using namespace tc;

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

std::once_flag g_encode_once;
EncodeTiledFn g_encode = nullptr;
char g_tc_reason[160] = "";

void resolve_encode()
{
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
    if (e != cudaSuccess || fn == nullptr || qres != cudaDriverEntryPointSuccess) {
        std::snprintf(g_tc_reason, sizeof(g_tc_reason), "cuTensorMapEncodeTiled is not available from the driver (%s)",
                      cudaGetErrorString(e));
        (void)cudaGetLastError();
        return;
    }
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
}

cudaError_t encode_kmajor(CUtensorMap *map, const void *base, int kind, long long rows, long long k_total,
                          long long ld_elems, int box_rows, long long batch = 1, long long batch_stride = 0)
{
    if (batch > 1) {
        // [batch][rows][k]: a box is one batch entry deep.  An operand all entries share is encoded with one entry.
        const int es3 = dtype_size(kind);
        const CUtensorMapDataType dt3 = (kind == KUDNN_B200_F32)   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                        : (kind == KUDNN_B200_F16) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                   : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const bool shared = batch_stride == 0;
        cuuint64_t dims[3] = {static_cast<cuuint64_t>(k_total), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(shared ? 1 : batch)};
        cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld_elems) * es3,
                                 static_cast<cuuint64_t>(shared ? rows * ld_elems : batch_stride) * es3};
        cuuint32_t box[3] = {static_cast<cuuint32_t>(kStageRowBytes / es3), static_cast<cuuint32_t>(box_rows), 1};
        cuuint32_t estr[3] = {1, 1, 1};
        CUresult r = g_encode(map, dt3, 3, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
    }
    const int es = dtype_size(kind);
    const CUtensorMapDataType dt = (kind == KUDNN_B200_F32)   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : (kind == KUDNN_B200_F16) ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                   : (kind == KUDNN_B200_S8)  ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                                              : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(k_total), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld_elems) * es};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(kStageRowBytes / es), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace

bool tc_available()
{
    std::call_once(g_encode_once, resolve_encode);
    return g_encode != nullptr;
}

const char *tc_unavailable_reason()
{
    return g_tc_reason;
}

cudaError_t tc_encode_kmajor(void *map128, const void *base, int kind, long long rows, long long k_total, long long ld_elems,
                             int box_rows)
{
    if (!tc_available()) {
        return cudaErrorNotSupported;
    }
    CUtensorMap m;
    cudaError_t e = encode_kmajor(&m, base, kind, rows, k_total, ld_elems, box_rows);
    if (e == cudaSuccess) {
        std::memcpy(map128, &m, sizeof(m));
    }
    return e;
}

cudaError_t tc_make_plan(const TcOperands &ops, long long m, long long n, int sm_count, bool with_staging, TcPlan *plan)
{
    static_assert(sizeof(CUtensorMap) <= 128, "tensor map storage too small");
    if (!tc_available()) {
        return cudaErrorNotSupported;
    }
    const long long tiles_m = (m + kBM - 1) / kBM;
    const long long tiles256 = ops.batch * tiles_m * ((n + 255) / 256);
    const int bn = (tiles256 >= sm_count || n > 128 * 64) ? 256 : 128;
    const long long tiles = ops.batch * tiles_m * ((n + bn - 1) / bn);  // over all batch entries
    if (tiles > (1ll << 30)) {
        return cudaErrorInvalidValue;
    }
    // CTA pairs for the large-problem shape (256-wide tiles): 256 x 256 tiles over clusters of two.  Not for launches
    // that run for many milliseconds: those are limited by the board's power cap, and the pair shape, which needs
    // fewer cycles, draws enough more power per cycle to end up slower there (bf16 n = 28672, k = 8192, ms per call,
    // pair / single CTA: 4096 rows 1.385 / 1.396, 8192 rows 2.84 / 2.85, 16384 rows 6.10 / 5.96, 32768 rows
    // 13.3 / 12.4).
    const double flops = 2.0 * static_cast<double>(m) * static_cast<double>(n) * static_cast<double>(ops.k_total);
    // batched launches use single CTAs
    bool pair = bn == 256 && m > kBM && flops < 6.0e12 && ops.batch == 1;
    if (const char *env = std::getenv("KUDNN_B200_TC_PAIR")) {
        pair = pair && std::atoi(env) != 0;
    }
    int pair_clusters = 0;
    if (pair) {
        const size_t smem = static_cast<size_t>(with_staging ? 5 : 6) * (kABytes + 128 * kStageRowBytes) + 1024 + kTailBytes +
                            (with_staging ? kStagingBytes : 0);
        pair_clusters = ops.kind == KUDNN_B200_F32   ? pair_clusters_kind<KUDNN_B200_F32>(smem)
                        : ops.kind == KUDNN_B200_F16 ? pair_clusters_kind<KUDNN_B200_F16>(smem)
                        : ops.kind == KUDNN_B200_S8  ? pair_clusters_kind<KUDNN_B200_S8>(smem)
                                                     : pair_clusters_kind<KUDNN_B200_BF16>(smem);
        pair = pair_clusters > 0;
    }
    plan->pair = pair ? 1 : 0;
    plan->narrow_from = 0;
    plan->block_n = bn;
    plan->stages = ((bn == 256 && !pair) ? 4 : 6) - (with_staging ? 1 : 0);
    // Split-K: with at most half the SMs busy and a long K, the CTAs of a cluster share a tile and cut K between
    // them (2, 4 or 8 ways: the rows of the tile are divided among the ranks for the final pass).  Each split keeps
    // at least four k-blocks so that the pipeline still fills, and no split may be empty.
    const int elems_per_row = kStageRowBytes / dtype_size(ops.kind);
    const long long num_kb = (ops.k_total + elems_per_row - 1) / elems_per_row;
    long long splits = 1;
    if (!pair && tiles * 2 <= sm_count && num_kb >= 8 && ops.kind != KUDNN_B200_S8) {
        long long want = std::min<long long>(sm_count / tiles, num_kb / 4);
        if (const char *env = std::getenv("KUDNN_B200_TC_SPLITS")) {
            const long long v = std::atoll(env);
            if (v >= 1 && v <= num_kb) {
                want = v;
            }
        }
        while (splits * 2 <= want && splits * 2 <= kMaxSplits) {
            splits *= 2;
        }
        while (splits > 1 && (num_kb + (num_kb + splits - 1) / splits - 1) / ((num_kb + splits - 1) / splits) != splits) {
            splits /= 2;
        }
    }
    plan->splits = static_cast<int>(splits);
    plan->kb_per_split = static_cast<int>((num_kb + splits - 1) / splits);
    const long long items = tiles * splits;
    plan->grid = splits > 1 ? static_cast<int>(items) : static_cast<int>(tiles < sm_count ? tiles : sm_count);
    const int b_rows = pair ? bn / 2 : bn;  // rows of the weight operand one CTA loads per k-block
    plan->smem_bytes = static_cast<size_t>(plan->stages) * (kABytes + b_rows * kStageRowBytes) + 1024 + kTailBytes +
                       (with_staging ? kStagingBytes : 0);
    if (pair) {
        const long long pair_tiles = ((m + 2 * kBM - 1) / (2 * kBM)) * ((n + bn - 1) / bn);
        plan->grid = 2 * static_cast<int>(pair_tiles < pair_clusters ? pair_tiles : pair_clusters);
        // Tiles left over after the last full wave: if they would keep at most half of the pairs busy, each of them
        // is processed as two pieces of half the width, which shortens that wave to a little more than half.
        const long long rem = pair_tiles % pair_clusters;
        bool narrow = pair_tiles > pair_clusters && rem > 0 && 2 * rem <= pair_clusters;
        plan->narrow_from = static_cast<int>(narrow ? pair_tiles - rem : pair_tiles);
    }
    CUtensorMap ta, tb;
    cudaError_t e = encode_kmajor(&ta, ops.a, ops.kind, m, ops.k_total, ops.lda, kBM, ops.batch, ops.a_bstride);
    if (e != cudaSuccess) {
        return e;
    }
    e = encode_kmajor(&tb, ops.b, ops.kind, n, ops.k_total, ops.ldb, b_rows, ops.batch, ops.b_bstride);
    if (e != cudaSuccess) {
        return e;
    }
    std::memcpy(plan->tmap_a, &ta, sizeof(ta));
    std::memcpy(plan->tmap_b, &tb, sizeof(tb));
    return cudaSuccess;
}

cudaError_t launch_tc(const TcOperands &ops, const TcPlan &plan, const EpiParams &epi, long long m, long long n,
                      DeviceStatus *status, cudaStream_t stream, long long wait_limit_cycles, int skip_kblock,
                      const BatchParams *bp)
{
    TcParams p;
    p.epi = epi;
    p.batch = static_cast<int>(ops.batch);
    p.a_bz = ops.a_bstride != 0 ? 1 : 0;
    p.b_bz = ops.b_bstride != 0 ? 1 : 0;
    std::memset(&p.bp, 0, sizeof(p.bp));
    p.bp.n1 = p.bp.n2 = 1;
    if (ops.batch > 1) {
        if (bp == nullptr || plan.pair != 0) {
            return cudaErrorInvalidValue;
        }
        p.bp = *bp;
    }
    p.wait_limit = wait_limit_cycles > 0 ? wait_limit_cycles : kDefaultWaitLimitCycles;
    // the test hook is honoured by the plain single-CTA shape only (no cluster partner is left half-signalled)
    p.skip_kb = (plan.pair == 0 && plan.splits == 1) ? skip_kblock : -1;
    {
        const bool sixteen = ops.kind == KUDNN_B200_F16 || ops.kind == KUDNN_B200_BF16;
        const bool light = sixteen && plan.splits == 1 && ops.batch == 1 && epi.n_mirrors == 0 && epi.beta == 0.0f &&
                           epi.res_op == KUDNN_B200_RES_NONE && epi.c_dtype == ops.kind &&
                           (epi.has_bias == 0 || epi.bias_dtype == ops.kind) &&
                           (epi.act == KUDNN_B200_ACT_NONE || epi.act == KUDNN_B200_ACT_RELU || epi.act == KUDNN_B200_ACT_SWISH);
        p.epi_warps = light ? 4 : kEpiWarps;
    }
    p.m = static_cast<int>(m);
    p.n = static_cast<int>(n);
    const int elems_per_row = kStageRowBytes / dtype_size(ops.kind);
    p.num_kb = static_cast<int>((ops.k_total + elems_per_row - 1) / elems_per_row);
    const int tile_rows = plan.pair ? 2 * kBM : kBM;
    p.tiles_m = static_cast<int>((m + tile_rows - 1) / tile_rows);
    p.tiles_n = static_cast<int>((n + plan.block_n - 1) / plan.block_n);
    p.num_tiles = p.tiles_m * p.tiles_n;
    p.idesc = ops.kind == KUDNN_B200_S8
                  ? make_idesc_i8(ops.a_signed != 0, ops.b_signed != 0, plan.block_n, plan.pair ? 2 * kBM : kBM)
                  : make_idesc(ops.kind, plan.block_n, plan.pair ? 2 * kBM : kBM);
    p.status = status;
    p.splits = plan.splits;
    p.kb_per_split = plan.kb_per_split;
    p.stages = plan.stages;
    {
        // The A rows of one raster group are re-read for every tile column and should stay in L2 next to the
        // streaming weights: at most about 64 MB of them (16 tile rows of 256 x 8192 bf16).  Measured on the 32768-row
        // layer, ms per call for 8 / 12 / 16 tile rows per group: 13.05 / 12.84 / 12.72; DRAM traffic is the same
        // within 3 % (the wave's working set exceeds what L2 retains either way).
        const long long tile_bytes = static_cast<long long>(tile_rows) * ops.k_total * dtype_size(ops.kind);
        long long gm = (64ll << 20) / (tile_bytes > 0 ? tile_bytes : 1);
        gm = gm < 2 ? 2 : (gm > kMaxGroupM ? kMaxGroupM : gm);
        p.group_m = static_cast<int>(gm);
    }
    p.num_items = plan.pair ? plan.narrow_from + 2 * (p.num_tiles - plan.narrow_from)
                            : p.num_tiles * plan.splits * static_cast<int>(ops.batch);
    p.narrow_from = plan.pair ? plan.narrow_from : p.num_tiles;
    p.idesc_narrow = ops.kind == KUDNN_B200_S8
                         ? make_idesc_i8(ops.a_signed != 0, ops.b_signed != 0, plan.block_n / 2, plan.pair ? 2 * kBM : kBM)
                         : make_idesc(ops.kind, plan.block_n / 2, plan.pair ? 2 * kBM : kBM);
    switch (ops.kind) {
        case KUDNN_B200_S8:
            if (plan.splits != 1 || ops.batch != 1) {
                return cudaErrorInvalidValue;
            }
            return launch_kind<KUDNN_B200_S8>(plan, p, stream);
        case KUDNN_B200_F32:
            return launch_kind<KUDNN_B200_F32>(plan, p, stream);
        case KUDNN_B200_F16:
            return launch_kind<KUDNN_B200_F16>(plan, p, stream);
        default:
            return launch_kind<KUDNN_B200_BF16>(plan, p, stream);
    }
}

}  // namespace kb
