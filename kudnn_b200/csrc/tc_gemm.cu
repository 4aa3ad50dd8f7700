// Host side of the tensor-core Linear kernel (tc_kernel.cuh): tensor maps, launch plans, launch parameters.
#include "tc_wide.cuh"

#include <algorithm>
#include <atomic>
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
                                   : (kind == KUDNN_B200_S32) ? CU_TENSOR_MAP_DATA_TYPE_INT32
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

namespace {

int env_choice(const char *name)
{
    const char *v = std::getenv(name);
    return v == nullptr || *v == '\0' ? -1 : std::atoi(v);
}

// The driver is asked once per device, kind and shared-memory size: the query takes several microseconds, and a plan is made
// for every call whose activations lie at a new address.
int pair_clusters_of(int kind, bool with_staging, size_t smem)
{
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices][8][2];  // clusters + 1; 0 = not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    std::atomic<int> *slot = dev < kDevices && kind < 8 ? &known[dev][kind][with_staging ? 1 : 0] : nullptr;
    if (slot != nullptr && slot->load() > 0) {
        return slot->load() - 1;
    }
    const int clusters = kind == KUDNN_B200_F32   ? pair_clusters_kind<KUDNN_B200_F32>(smem)
                         : kind == KUDNN_B200_F16 ? pair_clusters_kind<KUDNN_B200_F16>(smem)
                         : kind == KUDNN_B200_S8  ? pair_clusters_kind<KUDNN_B200_S8>(smem)
                                                  : pair_clusters_kind<KUDNN_B200_BF16>(smem);
    if (slot != nullptr && clusters > 0) {  // a failed query is asked again
        slot->store(clusters + 1);
    }
    return clusters;
}

}  // namespace

int tc_pair_clusters(int kind, size_t smem_bytes)
{
    return pair_clusters_of(kind, false, smem_bytes);
}

namespace {

// Estimated SM cycles of a launch of single CTAs.  A k-block of a tile costs its MMAs (2 cycles per column whatever the
// operand type) or its operand bytes (about 60 per cycle and SM), whichever is more.
double single_cta_cycles(long long tiles, int splits, long long kb, int bn, int a_rows, bool via_smem, int sm_count, double per_value = 0.35)
{
    const double per_kb = std::max(2.0 * bn, 2.1 * (a_rows + bn));
    const double area = static_cast<double>(a_rows) * bn;
    // finished from shared memory, with contiguous stores; or straight from tensor memory, under the next tile's products.
    // The other ranks' shares of a cut tile arrive at about 12 bytes per cycle.
    if (via_smem) {
        const double finish = 2500.0 + 0.04 * area + 0.2 * area / splits + (splits > 1 ? 1000.0 + area * 4 * (splits - 1) / splits / 12 : 0.0);
        const long long waves = (tiles * splits + sm_count - 1) / sm_count;
        return waves * (2500.0 + kb * per_kb + finish);
    }
    const double epilogue = 1000.0 + per_value * area;
    const long long waves = (tiles + sm_count - 1) / sm_count;
    return 2500.0 + waves * std::max(kb * per_kb, epilogue) + epilogue;
}

// Estimated SM cycles of the kernel of 256 x 512 tiles on `pairs` CTA pairs, and how its work is cut: the whole tiles of the last
// wave, which would keep only some of the pairs busy, become halves, and the halves of a last wave quarters.
double wide_cycles(bool ints, long long m, long long n, long long kb, int pairs, TcPlan *plan)
{
    // A k-block costs 1024 cycles of MMAs in a whole tile (measured 1.85 times the 640 of a pair's 256 x 256 tile in
    // tc_kernel.cuh, in launches that fill the GPU), and in a half or a quarter what six stages in flight bring in; where K is
    // short the epilogue is the longer part.
    // 8-bit integers are multiplied twice as fast, so that the copies set the pace, and 32-bit results are not drained ahead.
    const double whole_cost = ints ? kb * 850.0 + 6000.0 : std::max(kb * 1200.0, 16000.0);
    const double half_cost = ints ? kb * 560.0 + 4000.0 : std::max(kb * 740.0, 9000.0);
    const double quarter_cost = ints ? kb * 500.0 + 2500.0 : std::max(kb * 670.0, 6000.0);
    const long long tiles_m = (m + 255) / 256, columns = (n + 255) / 256;
    const long long tiles = tiles_m * (columns / 2), odd = tiles_m * (columns % 2);
    const int forced = env_choice("KUDNN_B200_TC_WIDE");
    double best = 1e300;
    for (const long long whole : {tiles, tiles / pairs * pairs, 0ll}) {
        const long long halves = 2 * (tiles - whole) + odd;
        for (const long long cut : {0ll, (whole + halves) % pairs, halves}) {
            if (cut > halves || (forced >= 1 && forced <= 3 && (whole != (forced == 1 ? tiles : 0) || cut != (forced == 3 ? halves : 0)))) {
                continue;
            }
            // item i falls to pair i modulo their number: pair j has X / pairs of the first X, and one more if j < X % pairs, so that
            // only these pairs can be the busiest
            const long long ends[3] = {whole, whole + halves - cut, whole + halves + cut};
            double longest = 0.0;
            for (const long long pair : {0ll, ends[0] % pairs, ends[1] % pairs, ends[2] % pairs}) {
                long long count[3];
                for (int i = 0; i < 3; ++i) {
                    count[i] = ends[i] / pairs + (pair < ends[i] % pairs ? 1 : 0);
                }
                longest = std::max(longest, whole_cost * count[0] + half_cost * (count[1] - count[0]) + quarter_cost * (count[2] - count[1]));
            }
            if (longest < best) {
                best = longest;
                plan->wide_whole = static_cast<int>(whole);
                plan->wide_half = static_cast<int>(halves - cut);
                plan->wide_items = static_cast<int>(whole + halves + cut);
            }
        }
    }
    return 20000.0 + best;  // start, and the last epilogue
}

}  // namespace

bool tc_wide_takes(const TcOperands &ops, const EpiParams &epi, TcRows rows)
{
    const int kind = ops.kind;
    const bool second = epi.res_op != KUDNN_B200_RES_NONE;
    if (kind == KUDNN_B200_S8) {
        // (a TMA store does not clip inside 16 bytes)
        return epi.n % 4 == 0 && ops.batch == 1 && epi.n_mirrors == 0 && epi.beta == 0.0f && !second && epi.c != nullptr && epi.c_sn == 1 && epi.c_sm % 4 == 0 &&
               (reinterpret_cast<uintptr_t>(epi.c) & 15u) == 0 && (epi.has_bias == 0 || (epi.bias_dtype == KUDNN_B200_S32 && epi.bias_sm == 0));
    }
    return (kind == KUDNN_B200_F16 || kind == KUDNN_B200_BF16) && ops.batch == 1 && rows == TcRows::kVectors && epi.n_mirrors == 0 &&
           epi.beta == 0.0f && (epi.c == nullptr) == second && epi.c_dtype == kind &&
           (epi.has_bias == 0 || (epi.bias_dtype == kind && epi.bias_sm == 0)) &&
           (!second || (epi.res_dtype == kind && epi.out_dtype == kind)) &&
           (epi.act == KUDNN_B200_ACT_NONE || epi.act == KUDNN_B200_ACT_RELU || epi.act == KUDNN_B200_ACT_SWISH ||
            epi.act == KUDNN_B200_ACT_GELU_TANH);
}

cudaError_t tc_make_plan(const TcOperands &ops, long long m, long long n, int sm_count, bool with_staging, TcRows rows,
                         bool wide_ok, TcPlan *plan)
{
    static_assert(sizeof(CUtensorMap) <= 128, "tensor map storage too small");
    if (!tc_available()) {
        return cudaErrorNotSupported;
    }
    const bool ints = ops.kind == KUDNN_B200_S8;
    const int width_step = ints ? 32 : 16;
    const long long tiles_m = (m + kBM - 1) / kBM;
    const int a_rows_single = static_cast<int>(m >= kBM ? kBM : (m + 7) / 8 * 8);
    const int elems_per_row = kStageRowBytes / dtype_size(ops.kind);
    const long long num_kb = (ops.k_total + elems_per_row - 1) / elems_per_row;
    // Single-CTA shapes: every tile width that the MMA takes, with K whole or cut between the 2, 4 or 8 CTAs of a cluster
    // (the rows of the tile are divided among them for the final pass).  Which of them is fastest follows from how the
    // tiles fill the SMs: with one work item per CTA a tile is finished from shared memory; more items than SMs run
    // persistently, the epilogue of one under the products of the next.  Kernel times: 64 x 11008 x 4096 in 86 CTAs of
    // 128 x 128 with K cut in two 39 us, in the shape chosen here 20 us; 1027 x 4096 x 11008 in two waves of 128 x 128
    // tiles 133 us, in one wave of 144 tiles of 128 x 256 71 us.
    const int forced_splits = env_choice("KUDNN_B200_TC_SPLITS");
    double best = 1e300;
    int bn = 128;
    long long splits = 1;
    bool via_smem = false;
    for (int w = width_step; w <= 256; w += width_step) {
        if (w - width_step >= n) {
            break;  // wider than the matrix
        }
        const long long tiles = ops.batch * tiles_m * ((n + w - 1) / w);
        if (tiles > (1ll << 30)) {
            continue;
        }
        for (int sp = 1; sp <= kMaxSplits; sp *= 2) {
            if (sp > 1) {
                // every split keeps at least two k-blocks and none is empty; a GPC's SMs do not divide into clusters of four
                // and eight without a rest (33 and 15 of them fit 148 SMs, cudaOccupancyMaxActiveClusters)
                const long long per = (num_kb + sp - 1) / sp;
                const int room = sp == 8 ? sm_count * 30 / 37 : sp == 4 ? sm_count * 33 / 37 : sm_count;
                if (ints || per < 2 || (num_kb + per - 1) / per != sp || (forced_splits < 0 && tiles * sp > room)) {
                    continue;
                }
            }
            if (forced_splits >= 1 && sp > forced_splits) {
                continue;
            }
            // (an output whose rows are not contiguous, column by column for one, leaves from the accumulator with a thread per row)
            const bool one_item = sp > 1 || (!ints && !with_staging && rows != TcRows::kOther &&
                                             (tiles <= sm_count || rows == TcRows::kContiguous));
            double cost = single_cta_cycles(tiles, sp, (num_kb + sp - 1) / sp, w, a_rows_single, one_item, sm_count);
            if (forced_splits >= 1 && sp * 2 <= forced_splits && sp * 2 <= kMaxSplits) {
                cost *= 1e6;  // taken only if no larger cut fits
            }
            if (cost < best) {
                best = cost;
                bn = w;
                splits = sp;
                via_smem = one_item;
            }
        }
    }
    if (best >= 1e300) {
        return cudaErrorInvalidValue;
    }
    // CTA pairs: 256 x 256 tiles over clusters of two, where that is estimated to be faster.  Not for launches
    // that run for many milliseconds: those are limited by the board's power cap, and this pair shape, which needs
    // fewer cycles, draws enough more power per cycle to end up slower there (bf16 n = 28672, k = 8192, ms per call,
    // pair / single CTA: 4096 rows 1.385 / 1.396, 8192 rows 2.84 / 2.85, 16384 rows 6.10 / 5.96, 32768 rows
    // 13.3 / 12.4).  The pairs on 256 x 512 tiles below are not held back so: in turn for seconds each, 32768 rows with
    // SiLU 12.4 to 12.5 ms at 1.10 GHz against 12.9 at 1.25 GHz of single CTAs.
    const double flops = 2.0 * static_cast<double>(m) * static_cast<double>(n) * static_cast<double>(ops.k_total);
    // Batched launches use single CTAs.
    bool pair = n > kBM && m > kBM && (flops < 6.0e12 || env_choice("KUDNN_B200_TC_PAIR") > 0) && ops.batch == 1 &&
                forced_splits <= 1 && env_choice("KUDNN_B200_TC_PAIR") != 0;
    // Cycles the epilogue takes per value: a thread's row leaves 16 bytes at a time, or value by value, rows side by side for one
    // output (column by column) or scattered.  4096 x 4603 x 2304, pair against single CTAs: bf16 379 and 130 us, fp32, whose
    // products take six times as long, 414 and 427 us.
    const double per_value = ints || rows == TcRows::kVectors || rows == TcRows::kAligned ? 0.35 : rows == TcRows::kContiguous ? 4.3 : 2.5;
    const int pair_stages = with_staging ? 5 : 6;
    plan->narrow_from = 0;
    // What the shape chosen so far is held against the kernel of 512-column tiles with: the same estimate, but with what a value
    // of its epilogue takes where K is too short to cover it (2048 rows against 1024, n = 9216, k = 256: 10 to 12 us per tile).
    // 32-bit integers leave there 16 bytes of a row at a time: about 28 000 cycles per tile of 4096 x 11008 x 4096.
    const double narrow_per_value = ints ? 0.85 : 0.55;
    double narrow_cycles = via_smem ? best : single_cta_cycles(ops.batch * tiles_m * ((n + bn - 1) / bn), 1, num_kb, bn, a_rows_single, false, sm_count, narrow_per_value);
    if (pair) {
        const long long pair_tiles = ((m + 2 * kBM - 1) / (2 * kBM)) * ((n + 255) / 256);
        const long long guess = sm_count / 2;
        const long long full = pair_tiles / guess, rem = pair_tiles % guess;
        const double waves = full + (rem == 0 ? 0.0 : (full > 0 && 2 * rem <= guess ? 0.55 : 1.0));
        const double epilogue = 1000.0 + per_value * kBM * 256;
        const double cycles = 4000.0 + waves * std::max(num_kb * 640.0, epilogue) + epilogue;
        pair = cycles < best || env_choice("KUDNN_B200_TC_PAIR") > 0;
        if (pair) {
            const double drain = narrow_per_value * kBM * 256;
            narrow_cycles = ints ? 4000.0 + num_kb * 640.0 + (waves - 1.0) * std::max(num_kb * 640.0, drain) + 0.5 * drain
                                 : 4000.0 + waves * std::max(num_kb * 640.0, drain) + drain;
        }
        int clusters = 0;
        if (pair) {
            clusters = pair_clusters_of(ops.kind, with_staging, static_cast<size_t>(pair_stages) * (kABytes + 128 * kStageRowBytes) + 1024 +
                                                      kTailBytes + (with_staging ? kStagingBytes : 0));
            pair = clusters > 0;
        }
        if (pair) {
            bn = 256;
            splits = 1;
            via_smem = false;
            plan->grid = 2 * static_cast<int>(pair_tiles < clusters ? pair_tiles : clusters);
            // Tiles left over after the last full wave: if they would keep at most half of the pairs busy, each of them
            // is processed as two pieces of half the width, which shortens that wave to a little more than half.
            const long long left = pair_tiles % clusters;
            const bool narrow = pair_tiles > clusters && left > 0 && 2 * left <= clusters;
            plan->narrow_from = static_cast<int>(narrow ? pair_tiles - left : pair_tiles);
        }
    }
    plan->wide = 0;
    const int forced_wide = env_choice("KUDNN_B200_TC_WIDE");
    if (wide_ok && m > kBM && forced_splits <= 1 && forced_wide != 0 && (env_choice("KUDNN_B200_TC_PAIR") < 0 || forced_wide > 0) &&
        m < (1ll << 31) - 512 && n < (1ll << 31) - 512 && ((m + 255) / 256) * ((n + 127) / 128) < (1ll << 30)) {
        const int clusters = pair_clusters_of(ops.kind, with_staging, WideShape<KUDNN_B200_F16>::kSmem);
        if (clusters > 0 && (wide_cycles(ints, m, n, num_kb, clusters, plan) < narrow_cycles || forced_wide > 0)) {
            plan->wide = 1;
            pair = true;
            bn = 256;
            splits = 1;
            via_smem = false;
            plan->grid = 2 * std::min(plan->wide_items, clusters);
        }
    }
    plan->pair = pair ? 1 : 0;
    plan->rows = rows;
    plan->block_n = bn;
    plan->via_smem = via_smem ? 1 : 0;
    plan->splits = static_cast<int>(splits);
    plan->kb_per_split = static_cast<int>((num_kb + splits - 1) / splits);
    plan->a_rows = pair ? kBM : a_rows_single;
    const long long tiles = ops.batch * tiles_m * ((n + bn - 1) / bn);  // over all batch entries
    if (!pair) {
        plan->grid = static_cast<int>(via_smem ? tiles * splits : std::min<long long>(tiles, sm_count));
    }
    const int b_rows = pair ? bn / 2 : bn;  // rows of the weight operand one CTA loads per k-block
    const long long stage = static_cast<long long>(plan->a_rows + b_rows) * kStageRowBytes;
    const long long fixed = 1024 + kTailBytes + (with_staging ? kStagingBytes : 0);
    plan->stages = static_cast<int>(std::min<long long>((kSmemLimit - fixed) / stage, kMaxStages));
    if (pair) {
        plan->stages = pair_stages;
    } else if (via_smem) {
        plan->stages = std::max(std::min(plan->stages, plan->kb_per_split), 2);
    }
    // the last stage's MMA reads 128 rows of A wherever the copy stopped, and a tile finished from shared memory lies
    // there as fp32 with four columns of padding
    long long ring = std::max(plan->stages * stage, (plan->stages - 1) * stage + kABytes);
    if (via_smem) {
        ring = std::max<long long>(ring, static_cast<long long>(plan->a_rows) * (bn + 4) * 4);
    }
    ring = (ring + 1023) / 1024 * 1024;
    plan->ring_bytes = static_cast<int>(ring);
    plan->smem_bytes = plan->wide ? (ints ? WideShape<KUDNN_B200_S8>::kSmem : WideShape<KUDNN_B200_F16>::kSmem) : static_cast<size_t>(ring + fixed);
    if (plan->smem_bytes > static_cast<size_t>(kSmemLimit)) {
        return cudaErrorInvalidValue;
    }
    CUtensorMap ta, tb;
    cudaError_t e = encode_kmajor(&ta, ops.a, ops.kind, m, ops.k_total, ops.lda, plan->a_rows, ops.batch, ops.a_bstride);
    if (e != cudaSuccess) {
        return e;
    }
    e = encode_kmajor(&tb, ops.b, ops.kind, n, ops.k_total, ops.ldb, b_rows, ops.batch, ops.b_bstride);
    if (e != cudaSuccess) {
        return e;
    }
    std::memcpy(plan->tmap_a, &ta, sizeof(ta));
    std::memcpy(plan->tmap_b, &tb, sizeof(tb));
    if (plan->wide) {
        e = encode_kmajor(&tb, ops.b, ops.kind, n, ops.k_total, ops.ldb, 64, ops.batch, ops.b_bstride);
        std::memcpy(plan->tmap_b64, &tb, sizeof(tb));
    }
    return e;
}

namespace {

// The A rows of one raster group are re-read for every tile column and should stay in L2 next to the
// streaming weights: at most about 64 MB of them (16 tile rows of 256 x 8192 bf16).  Measured on the 32768-row
// layer, ms per call for 8 / 12 / 16 tile rows per group: 13.05 / 12.84 / 12.72; DRAM traffic is the same
// within 3 % (the wave's working set exceeds what L2 retains either way).
int raster_group(const TcOperands &ops, int tile_rows)
{
    const long long tile_bytes = static_cast<long long>(tile_rows) * ops.k_total * dtype_size(ops.kind);
    const long long gm = (64ll << 20) / (tile_bytes > 0 ? tile_bytes : 1);
    return static_cast<int>(gm < 2 ? 2 : (gm > kMaxGroupM ? kMaxGroupM : gm));
}

cudaError_t launch_wide(const TcOperands &ops, const TcPlan &plan, const EpiParams &epi, long long m, long long n,
                        DeviceStatus *status, cudaStream_t stream, long long wait_limit_cycles, int skip_kblock)
{
    if (!tc_wide_takes(ops, epi, plan.rows)) {
        return cudaErrorInvalidValue;  // the plan was made for another epilogue
    }
    WideParams p;
    p.epi = epi;
    p.m = static_cast<int>(m);
    p.n = static_cast<int>(n);
    const int elems_per_row = kStageRowBytes / dtype_size(ops.kind);
    p.num_kb = static_cast<int>((ops.k_total + elems_per_row - 1) / elems_per_row);
    p.tiles_m = static_cast<int>((m + 255) / 256);
    p.tiles_w = static_cast<int>((n + 255) / 256 / 2);
    // Taller raster groups for launches of many milliseconds: the rows of B of a tile are then shared by more pairs at a time, although
    // a group's rows of A (134 MB there) no longer stay in L2.  The 32768-row layer in a loop of seconds under the power cap, on a
    // warmer GPU than the figures above, 8 / 16 / 32 tile rows per group: 14.3 / 13.2-13.7 / 13.0-13.2 ms.
    // Not for shorter ones: 8192 x 4096 x 4096 in one group of 32 instead of two of 16 gains nothing (1.05 against 1.07 times the
    // 256-column tiles, runs differing by 2 %).
    const bool tall = 2.0 * static_cast<double>(m) * static_cast<double>(n) * static_cast<double>(ops.k_total) >= 6.0e12;
    p.group_m = tall ? 32 : raster_group(ops, 2 * kBM);
    p.n_whole = plan.wide_whole;
    p.n_half = plan.wide_half;
    p.num_items = plan.wide_items;
    const bool ints = ops.kind == KUDNN_B200_S8;
    p.idesc = ints ? make_idesc_i8(ops.a_signed != 0, ops.b_signed != 0, 256, 2 * kBM) : make_idesc(ops.kind, 256, 2 * kBM);
    p.idesc_quarter = ints ? make_idesc_i8(ops.a_signed != 0, ops.b_signed != 0, 128, 2 * kBM) : make_idesc(ops.kind, 128, 2 * kBM);
    p.b_stable = ops.b_stable ? 1 : 0;
    p.load_kb = skip_kblock >= 0 ? std::min(skip_kblock, p.num_kb) : p.num_kb;
    p.status = status;
    p.wait_limit = wait_limit_cycles > 0 ? wait_limit_cycles : kDefaultWaitLimitCycles;
    // the output, written in boxes of 32 rows x 128 bytes
    const bool second = epi.res_op != KUDNN_B200_RES_NONE;
    CUtensorMap out;
    const cudaError_t e = encode_kmajor(&out, second ? epi.out : epi.c, ints ? KUDNN_B200_S32 : ops.kind, m, n, second ? epi.out_sm : epi.c_sm, 32);
    if (e != cudaSuccess) {
        return e;
    }
    return ints                        ? launch_wide_kind<KUDNN_B200_S8>(plan, &out, p, stream)
           : ops.kind == KUDNN_B200_F16 ? launch_wide_kind<KUDNN_B200_F16>(plan, &out, p, stream)
                                        : launch_wide_kind<KUDNN_B200_BF16>(plan, &out, p, stream);
}

}  // namespace

cudaError_t launch_tc(const TcOperands &ops, const TcPlan &plan, const EpiParams &epi, long long m, long long n,
                      DeviceStatus *status, cudaStream_t stream, long long wait_limit_cycles, int skip_kblock,
                      const BatchParams *bp, const int *run_if)
{
    if (plan.wide) {
        return run_if != nullptr ? cudaErrorInvalidValue : launch_wide(ops, plan, epi, m, n, status, stream, wait_limit_cycles, skip_kblock);
    }
    TcParams p;
    p.epi = epi;
    p.run_if = run_if;
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
        const bool light = sixteen && plan.via_smem == 0 && ops.batch == 1 && epi.n_mirrors == 0 && epi.beta == 0.0f &&
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
    p.bn = plan.block_n;
    p.b_stable = ops.b_stable ? 1 : 0;
    p.a_rows = plan.a_rows;
    p.ring_bytes = plan.ring_bytes;
    p.via_smem = plan.via_smem;
    p.rows = plan.rows;
    p.group_m = raster_group(ops, tile_rows);
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
