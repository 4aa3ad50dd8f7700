// fp32 Linear on the fp16 tensor cores, for large products: CTA pairs, cta_group::2.
//
// An fp32 matrix product is bound by the tensor pipe, which multiplies TF32 at half the rate of fp16 although both carry 11
// significant bits.  So every row is scaled by a power of two that takes its largest element to [2^14, 2^15) and written as
// x = hi + lo / 2^12 with hi = fp16(x) and lo = fp16((x - hi) 2^12) (split_half_kernel): to 2^-23 of every element down to 2^-28 of
// the row's largest, as the TF32 planes do.  The products hi.hi go to one accumulator and
// hi.lo + lo.hi to another; acc0 + acc1 / 2^12, scaled back by row and column, is the sum of the three products that the TF32
// planes add up (the fourth, lo.lo, is 2^-22 relative there and here).  Two accumulators also keep the small products out of the
// additions to the large one, and a k-block of 64 brings in each operand's planes once instead of one and a half times: 64 KiB per
// SM and 1536 cycles of MMAs.
//
// A normal distribution has one element below 2^-28 of its row's largest in 10^8.  The split leaves up to eight of them per row out
// of the planes, and the epilogue adds their products in fp32 (planes_add_rest), for up to sixteen rows of activations and weights.
// A call with lists takes 2 to 4 us more; one without 0.3 to 0.5 us more than without the code (1024 x 2048 x 1536 31.5 -> 32.0), which
// stands between the drain and the stores of every item: by 32 columns, in a function or a branch of its own it cost as much or more.
//
// Rows that this form does not carry (elements that are not finite, whose largest lies outside [2^-100, 2^64], with a nonzero
// element below 2^-60 of it, or with more than eight below 2^-28) are marked by the split; if there is any, or lists of more rows
// than that, among the activations or the weights, all CTAs leave, and the launches that follow compute the product on TF32 planes
// (tc_linear_kernel), which otherwise leave at once.  4096 x 4608 x 2304 in calls one after the other: 188 to 209 us, with one
// element of 1e-10 205 to 216, left to the TF32 planes 430 to 470, where the TF32 form by itself takes 390 to 420: the split and
// the marks in vain.
//
// Shape of one CTA: as tc_wide_kernel, a ring of three stages, tiles of 256 x 256 (both accumulators), and 256 x 128 for the tiles of
// a last wave that would keep at most half of the pairs busy.
//
// Measured against the TF32 form, kernels and splits together, in turn on one GPU: 4096 x 4608 x 2304 350 -> 185 us, 8192 x 5120 x
// 5120 1715 -> 863 us (1494 TFLOP/s of fp16 products), normwise error against 64 bits 5.4e-6 -> 2.8e-6 and 1.3e-5 -> 6.7e-6: half
// as many additions, each of which cuts the sum, and none of the small products among them.  The product kernel alone takes 174 us
// of the first, the tensor pipe busy for 81 % of its cycles, the split 19 us, the two launches that leave at once 5 each (serialised).
#pragma once

#include "tc_wide.cuh"

namespace kb {

namespace tc {

constexpr int kPlanesStages = 3;
constexpr int kPlanesStageBytes = 4 * kABytes;  // hi and lo of A, hi and lo of B
constexpr int kPlanesRing = kPlanesStages * kPlanesStageBytes;
constexpr int kPlanesSmem = kPlanesRing + kStagingBytes + 256;
static_assert(kPlanesSmem <= kSmemLimit, "shared memory of the planes kernel");

struct PlanesParams {
    EpiParams epi;
    int m, n;
    int num_kb;  // of 64 columns
    int tiles_m, tiles_n;
    int group_m;
    int n_whole, num_items;  // items [0, n_whole) are whole tiles, the rest two to a tile
    unsigned idesc, idesc_half;
    PlanesOperand a, b;
    int *fallback;  // written: whether the product is left to the launches that follow
    int load_kb;    // as in WideParams
    DeviceStatus *status;
    long long wait_limit;
};

struct PlanesItem {
    int tm, n0, width;
};

__device__ __forceinline__ PlanesItem planes_item(const PlanesParams &p, int item)
{
    PlanesItem w;
    int tile = item, half = 0;
    w.width = 256;
    if (item >= p.n_whole) {
        tile = p.n_whole + ((item - p.n_whole) >> 1);
        half = (item - p.n_whole) & 1;
        w.width = 128;
    }
    const int per_group = p.group_m * p.tiles_n;
    const int first_m = tile / per_group * p.group_m;
    const int gsize = p.tiles_m - first_m < p.group_m ? p.tiles_m - first_m : p.group_m;
    const int in_group = tile % per_group;
    w.tm = first_m + in_group % gsize;
    w.n0 = in_group / gsize * 256 + half * 128;
    return w;
}

// 32 rows (a lane each) x `columns` (128 or 64) columns: both accumulators out of tensor memory, scaled back, alpha and bias applied.
// `stage` holds the columns' scales and, 512 bytes on, their bias (-0 where there is none).
__device__ __forceinline__ void planes_drain(float alpha, float row_scale, uint32_t taddr, int columns, uint32_t stage, float (&keep)[128])
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i == 4 && columns == 64) {
            break;
        }
        uint32_t main[16], cross[16];
        tmem_load_16_issue(taddr + static_cast<uint32_t>(i * 16), main);
        tmem_load_16_issue(taddr + static_cast<uint32_t>(256 + i * 16), cross);
        tmem_load_wait16(main);
        tmem_load_wait16(cross);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            float s[4], b[4];
            const uint32_t at = stage + static_cast<uint32_t>((i * 16 + g * 4) * 4);
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(s[0]), "=f"(s[1]), "=f"(s[2]), "=f"(s[3]) : "r"(at));
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3]) : "r"(at + 512));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float v = fmaf(__uint_as_float(cross[g * 4 + j]), 0x1p-12f, __uint_as_float(main[g * 4 + j]));
                keep[i * 16 + g * 4 + j] = fmaf(v * row_scale * s[j], alpha, b[j]);
            }
        }
    }
}

__device__ __forceinline__ float planes_value(const PlanesOperand &o, long long row, int k, int num_kb)
{
    const unsigned short *at = o.planes + (row * num_kb + (k >> 6)) * 128 + (k & 63);
    return fmaf(__half2float(__ushort_as_half(at[64])), 0x1p-12f, __half2float(__ushort_as_half(at[0]))) * o.scale[row];
}

// What the planes of a row or column leave out, times the other operand's elements; where both leave out the same k, it is added
// with the column.
__device__ __forceinline__ void planes_add_rest(const PlanesParams &p, int row0, int n0, int columns, int lane, unsigned marked_rows,
                                                const unsigned (&marked_columns)[4], float (&keep)[128])
{
    const float alpha = p.epi.alpha;
    const int row = row0 + lane;
    const bool mine = (marked_rows >> lane & 1u) != 0u;
#pragma unroll 1
    for (unsigned left = marked_rows; left != 0u; left &= left - 1u) {
        const int r = __ffs(left) - 1;
        const PlanesElement *list = p.a.rest + static_cast<long long>(row0 + r) * kPlanesRest;
#pragma unroll 1
        for (int i = 0; i < kPlanesRest; ++i) {
            const PlanesElement e = list[i];
            if (e.k < 0) {
                break;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int col = n0 + q * 32 + lane;
                const float y = q * 32 < columns && col < p.n ? planes_value(p.b, col, e.k, p.num_kb) : 0.0f;
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const float t = e.x * __shfl_sync(0xffffffffu, y, j);
                    if (lane == r) {
                        keep[q * 32 + j] = fmaf(t, alpha, keep[q * 32 + j]);
                    }
                }
            }
        }
    }
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
#pragma unroll 1
        for (unsigned left = q == 0 ? marked_columns[0] : q == 1 ? marked_columns[1] : q == 2 ? marked_columns[2] : marked_columns[3]; left != 0u;
             left &= left - 1u) {
            const int c = q * 32 + __ffs(left) - 1;
            const PlanesElement *list = p.b.rest + static_cast<long long>(n0 + c) * kPlanesRest;
#pragma unroll 1
            for (int i = 0; i < kPlanesRest; ++i) {
                const PlanesElement e = list[i];
                if (e.k < 0) {
                    break;
                }
                float x = 0.0f;
                if (row < p.m) {
                    x = planes_value(p.a, row, e.k, p.num_kb);
#pragma unroll 1
                    for (int j = 0; mine && j < kPlanesRest; ++j) {
                        const PlanesElement f = p.a.rest[static_cast<long long>(row) * kPlanesRest + j];
                        if (f.k < 0) {
                            break;
                        }
                        x = f.k == e.k ? f.x : x;
                    }
                }
                const float t = x * e.x;
#pragma unroll
                for (int j = 0; j < 128; ++j) {
                    if (j == c) {
                        keep[j] = fmaf(t, alpha, keep[j]);
                    }
                }
            }
        }
    }
}

template <int kAct>
__device__ __forceinline__ void planes_finish(const PlanesParams &p, const CUtensorMap *tmap_out, int row0, int n0, int columns,
                                              uint32_t stage, int lane, float (&keep)[128])
{
    const float act_alpha = p.epi.act_alpha;
    const uint32_t my_row = stage + static_cast<uint32_t>(lane * 128);
    const uint32_t swz = static_cast<uint32_t>(lane & 7) << 4;
#pragma unroll 1
    for (int c0 = 0; c0 < columns; c0 += 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            keep[j] = activation<true>(keep[j], kAct, act_alpha);
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the copy that read this warp's box before
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(my_row + ((static_cast<uint32_t>(g) << 4) ^ swz)), "f"(keep[g * 4]),
                         "f"(keep[g * 4 + 1]), "f"(keep[g * 4 + 2]), "f"(keep[g * 4 + 3])
                         : "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && row0 < p.m && n0 + c0 < p.n) {
            tma_store_2d(tmap_out, stage, n0 + c0, row0);
        }
#pragma unroll
        for (int j = 0; j < 96; ++j) {
            keep[j] = keep[j + 32];
        }
    }
}

__global__ void __launch_bounds__(kWideThreads, 1)
    tc_planes_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_b64, const __grid_constant__ CUtensorMap tmap_out,
                     const __grid_constant__ PlanesParams p)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *staging = smem + kPlanesRing;
    uint64_t *bars = reinterpret_cast<uint64_t *>(staging + kStagingBytes);
    uint64_t *full_bar = bars;
    uint64_t *empty_bar = bars + kPlanesStages;
    uint64_t *tmem_full = bars + 2 * kPlanesStages;
    uint64_t *tmem_empty = tmem_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *marked_rows = reinterpret_cast<int *>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if ((smem_u32(smem) & 1023u) != 0) {  // never: the declaration asks for the alignment.  Both CTAs would leave here.
        if (threadIdx.x == 0) {
            atomicCAS(&p.status->code, kErrNone, kErrTimeout);
        }
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPlanesStages; ++s) {
            mbar_init(full_bar + s, 1);
            mbar_init(empty_bar + s, 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, 2 * kEpiWarps);
        *abort_flag = 0;
        *marked_rows = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the peer's barriers are initialised before anything is signalled on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t rank = cluster_rank();
    const int first_item = static_cast<int>(blockIdx.x >> 1);
    const int stride = static_cast<int>(gridDim.x >> 1);
    pdl_launch_dependents();  // only now that this CTA holds its tensor memory (see tc_linear_kernel)
    pdl_wait();
    // every CTA comes to the same answer, from the same bytes; both operands' marks are on their way at a time
    int marked = 0;
    auto count = [&](unsigned marks) {
        marked += (marks & 0x02020202u) != 0u ? kPlanesRestRows + 1 : __popc(marks & 0x01010101u);
        marked = marked < kPlanesRestRows + 1 ? marked : kPlanesRestRows + 1;
    };
    for (int i = static_cast<int>(threadIdx.x); i < (p.m + 15) / 16 || i < (p.n + 15) / 16; i += kWideThreads) {
        uint4 some[2] = {};
#pragma unroll
        for (int op = 0; op < 2; ++op) {
            const int rows = op == 0 ? p.m : p.n;
            const unsigned char *flags = (op == 0 ? p.a.flags : p.b.flags) + static_cast<long long>(i) * 16;
            if (i < (rows + 15) / 16) {
                some[op] = *reinterpret_cast<const uint4 *>(flags);
            }
        }
#pragma unroll
        for (int op = 0; op < 2; ++op) {
            if ((some[op].x | some[op].y | some[op].z | some[op].w) != 0u) {
                count(some[op].x);
                count(some[op].y);
                count(some[op].z);
                count(some[op].w);
            }
        }
    }
    if (marked != 0) {
        atomicAdd(marked_rows, marked);
    }
    __syncthreads();
    const bool fallback = *marked_rows > kPlanesRestRows, rest = *marked_rows != 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *p.fallback = fallback ? 1 : 0;
    }
    const int num_items = fallback ? 0 : p.num_items;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kWideControlRegs));
        if (warp == 0) {
            // ------------------------------------------------------------------ loads
            if (lane == 0) {
                const uint32_t ring = smem_u32(smem);
                // the barriers of the leader count both CTAs' bytes; only the leader announces them
                const uint32_t full_at = map_to_rank(smem_u32(full_bar), 0u);
                int stage = 0;
                uint32_t phase = 0;
                bool alive = true;
                for (int item = first_item; alive && item < num_items; item += stride) {
                    const PlanesItem w = planes_item(p, item);
                    const int a_row = w.tm * 256 + static_cast<int>(rank) * kBM, b_row = w.n0 + static_cast<int>(rank) * (w.width / 2);
                    const CUtensorMap *map_b = w.width == 256 ? &tmap_b : &tmap_b64;
                    const uint32_t bytes = w.width == 256 ? 8 * kABytes : 6 * kABytes;
                    for (int kb = 0; kb < p.load_kb; ++kb) {
                        if (!mbar_wait(empty_bar + stage, phase ^ 1u, abort_flag, p.status, 1, p.wait_limit)) {
                            alive = false;
                            break;
                        }
                        if (rank == 0) {
                            mbar_expect_tx(full_bar + stage, bytes);
                        }
                        const uint32_t at = ring + static_cast<uint32_t>(stage * kPlanesStageBytes), bar = full_at + static_cast<uint32_t>(stage * 8);
                        tma_load_pair_at(at, &tmap_a, bar, kb * 128, a_row);
                        tma_load_pair_at(at + kABytes, &tmap_a, bar, kb * 128 + 64, a_row);
                        tma_load_pair_at(at + 2 * kABytes, map_b, bar, kb * 128, b_row);
                        tma_load_pair_at(at + 3 * kABytes, map_b, bar, kb * 128 + 64, b_row);
                        if (++stage == kPlanesStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                }
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------------ MMAs, issued by the leader for both CTAs
            if (lane == 0 && rank == 0) {
                int stage = 0;
                uint32_t phase = 0, uses = 0;
                bool alive = true;
                for (int item = first_item; alive && item < num_items; item += stride) {
                    const PlanesItem w = planes_item(p, item);
                    const uint32_t idesc = w.width == 256 ? p.idesc : p.idesc_half;
                    alive = mbar_wait(tmem_empty, (uses & 1u) ^ 1u, abort_flag, p.status, 2, p.wait_limit);
                    ++uses;
                    tc_fence_after();
                    for (int kb = 0; alive && kb < p.num_kb; ++kb) {
                        alive = mbar_wait(full_bar + stage, phase, abort_flag, p.status, 3, p.wait_limit);
                        tc_fence_after();
                        if (!alive) {
                            break;
                        }
                        const uint32_t at = smem_u32(smem) + static_cast<uint32_t>(stage * kPlanesStageBytes);
                        const uint64_t a_hi = make_smem_desc(at), a_lo = make_smem_desc(at + kABytes);
                        const uint64_t b_hi = make_smem_desc(at + 2 * kABytes), b_lo = make_smem_desc(at + 3 * kABytes);
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            const uint32_t more = (kb != 0 || ks != 0) ? 1u : 0u;
                            const uint64_t x = static_cast<uint64_t>(2 * ks);
                            umma_pair<KUDNN_B200_F16>(tmem_base, a_hi + x, b_hi + x, idesc, more);
                            umma_pair<KUDNN_B200_F16>(tmem_base + 256u, a_hi + x, b_lo + x, idesc, more);
                            umma_pair<KUDNN_B200_F16>(tmem_base + 256u, a_lo + x, b_hi + x, idesc, 1u);
                        }
                        umma_commit_pair(empty_bar + stage);
                        if (++stage == kPlanesStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                    if (alive) {
                        umma_commit_pair(tmem_full);
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWideEpilogueRegs));
        // ------------------------------------------------------------------ epilogue: 32 rows and half of the columns per warp
        const int quarter = warp & 3;
        const int part = (warp - 4) / 4;
        const uint32_t stage = smem_u32(staging + (warp - 4) * kWarpStageBytes);
        const uint32_t drained = map_to_rank(smem_u32(tmem_empty), 0u);
        const EpiParams &e = p.epi;
        uint32_t phase = 0;
        for (int item = first_item; item < num_items; item += stride) {
            const PlanesItem w = planes_item(p, item);
            const int columns = w.width / 2;
            const int n0 = w.n0 + part * columns;
            const int row0 = w.tm * 256 + static_cast<int>(rank) * kBM + quarter * 32;
            // scales and bias wait in this warp's box, which the stores of the previous item have left
            if (lane == 0) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            __syncwarp();
            for (int c = lane; c < columns; c += 32) {
                const bool inside = n0 + c < p.n;
                const float s = inside ? p.b.scale[n0 + c] : 0.0f;
                const float b = e.has_bias == 0 ? -0.0f : inside ? static_cast<const float *>(e.bias)[(n0 + c) * e.bias_sn] : 0.0f;
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage + static_cast<uint32_t>(c * 4)), "f"(s) : "memory");
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(stage + 512u + static_cast<uint32_t>(c * 4)), "f"(b) : "memory");
            }
            __syncwarp();
            const float row_scale = row0 + lane < p.m ? p.a.scale[row0 + lane] : 0.0f;
            unsigned marked_row = 0u, marked_column[4] = {};
            if (rest) {
                marked_row = __ballot_sync(0xffffffffu, row0 + lane < p.m && p.a.flags[row0 + lane] != 0);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int c = n0 + q * 32 + lane;
                    marked_column[q] = __ballot_sync(0xffffffffu, q * 32 < columns && c < p.n && p.b.flags[c] != 0);
                }
            }
            const bool arrived = __all_sync(0xffffffffu, mbar_wait(tmem_full, phase, abort_flag, p.status, 4, p.wait_limit));
            phase ^= 1u;
            if (!arrived) {
                break;
            }
            tc_fence_after();
            float keep[128];
            planes_drain(e.alpha, row_scale, tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(part * columns),
                         columns, stage, keep);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_cluster(drained);
            }
            if ((marked_row | marked_column[0] | marked_column[1] | marked_column[2] | marked_column[3]) != 0u) {
                planes_add_rest(p, row0, n0, columns, lane, marked_row, marked_column, keep);
            }
            switch (e.act) {
                case KUDNN_B200_ACT_NONE: planes_finish<KUDNN_B200_ACT_NONE>(p, &tmap_out, row0, n0, columns, stage, lane, keep); break;
                case KUDNN_B200_ACT_RELU: planes_finish<KUDNN_B200_ACT_RELU>(p, &tmap_out, row0, n0, columns, stage, lane, keep); break;
                case KUDNN_B200_ACT_SWISH: planes_finish<KUDNN_B200_ACT_SWISH>(p, &tmap_out, row0, n0, columns, stage, lane, keep); break;
                default: planes_finish<KUDNN_B200_ACT_GELU_TANH>(p, &tmap_out, row0, n0, columns, stage, lane, keep); break;
            }
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    }

    // ---------------------------------------------------------------------- teardown, as in tc_linear_kernel
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*abort_flag != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 400000ll) {
            __nanosleep(1000);
        }
        __syncthreads();
    }
    cluster_sync_all();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

}  // namespace tc

}  // namespace kb
