// Tensor-core Linear kernel for large products: CTA pairs on 256 x 512 tiles.
//
// What bounds a large product on this GPU is not the tensor pipe but what it takes to feed it: a pair that works on 256 x 256
// (tc_kernel.cuh) brings 64 bytes per cycle into each of its SMs at the full rate of the MMAs, all that an SM takes in, and
// in launches under the board's power cap every byte that travels costs clock.  Here the pair's tile is two accumulators wide:
// a k-block of A meets 512 rows of B, 48 KiB per SM and 1024 cycles instead of 32 KiB per 512, a quarter less.  The price is
// that both accumulators belong to one tile, so nothing of tensor memory is left for the next tile while the epilogue drains
// this one.  Most of that is won back by letting the two accumulators run out of step: the first k-blocks of a tile are
// multiplied into the first accumulator, then into the second, and so are the last ones, so that the first accumulator is
// finished, drained and started again while the second is still multiplied.
//
// Shape of one CTA (384 threads, persistent, one CTA per SM, clusters of two):
//   warp 0       one lane loads a k-block: 128 rows of A, 128 rows of B per accumulator (TMA, 128-byte swizzle) into a ring of
//                four stages (halves and quarters: six; 8-bit integers: three, and four)
//   warp 1       one lane of the leader issues the cta_group::2 MMAs for both CTAs
//   warps 4..11  epilogue, four warps per accumulator, each with 32 rows of it: out of tensor memory and rounded to 16 bits at
//                once, which frees the accumulator; the rest of the chain under the next tile's products; then through 4 KiB of
//                shared memory of the warp's own, [32 rows][128 bytes], to a TMA store.  Whole 128-byte lines leave the SM,
//                and rows and columns past the output's end are clipped by the copy.
//
// Measured against the pairs on 256 x 256 tiles, in turn on one GPU, inputs from memory: 4096 x 11008 x 4096 bf16 with SiLU
// 276.5 -> 261.4 us, 8192 x 4096 x 4096 fp16 with GELU and a residual 239.6 -> 225.4, 8192 x 8192 x 8192 bf16 840 -> 735,
// 32768 x 28672 x 8192 with SiLU (single CTAs before) 12.6 -> 11.75 ms, 8192 x 8192 x 512 (epilogue) 181 -> 83.  On a warmer
// GPU, where the power cap bites sooner, the gain was 4.6, 7.4 and 4.5 % on the first, second and fourth.  All but the
// last run under the power cap: leaving out the step between the accumulators costs cycles but no time there, while every
// instruction left out of the epilogue shows.  The 16-bit instances spill (fp16 524 bytes of stores and 1380 of loads, bf16 372
// and 1388): the 128 registers of a drained accumulator beside two residual pieces and the values at work.
//
// Work items, in this order: whole tiles; halves (256 x 256, one accumulator), of which the two accumulators take turns;
// quarters (256 x 128).  The host cuts the tiles of the last wave so that all pairs end at about the same time.
#pragma once

#include "tc_kernel.cuh"

namespace kb {

namespace tc {

constexpr int kWideThreads = 128 + 32 * kEpiWarps;
// Registers per thread at launch and in the two parts of the block: 128 * 40 + 256 * 232 = 384 * 168
constexpr int kWideControlRegs = 40, kWideEpilogueRegs = 232;
constexpr int kWideStageBytes = 3 * kABytes;  // A, and B of either accumulator
constexpr int kWideSmallBytes = 2 * kABytes;  // halves and quarters, with one B each, see the same memory as a ring of their own
template <int kKind>
struct WideShape {
    // 32-bit results leave tensor memory through shared memory box by box, while the next tile waits for the accumulator: two boxes
    // per warp there, and a stage less
    static constexpr int kBoxes = kKind == KUDNN_B200_S8 ? 2 : 1;
    static constexpr int kStages = kKind == KUDNN_B200_S8 ? 3 : 4;
    static constexpr int kRing = kStages * kWideStageBytes;
    static constexpr int kSmallStages = kRing / kWideSmallBytes;
    static constexpr int kSmem = kRing + kBoxes * kStagingBytes + 256;
    static_assert(kSmem <= kSmemLimit, "shared memory of the wide kernel");
};
constexpr int kWideSkew = 2;                             // k-blocks by which the accumulators run out of step

struct WideParams {
    EpiParams epi;
    int m, n;
    int num_kb;
    int tiles_m, tiles_w;  // rows of tiles, whole tiles (512 columns) per row
    int group_m;           // tile rows per raster group
    // items [0, n_whole) are whole tiles; then n_half halves: the two of every whole tile from n_whole on, and the columns past
    // the whole tiles of every row; the last of the halves are two quarters each
    int n_whole, n_half, num_items;
    unsigned idesc, idesc_quarter;
    int b_stable;
    int load_kb;  // num_kb, or by the test hook fewer: the k-blocks of an item that are loaded
    DeviceStatus *status;
    long long wait_limit;
};

struct WideItem {
    int tm;     // 256-row tile
    int n0;     // first column
    int width;  // columns per accumulator: 256, or 128 for a quarter
    bool whole;
};

__device__ __forceinline__ WideItem wide_item(const WideParams &p, int item)
{
    WideItem w;
    int half = -1, quarter = 0;
    w.width = 256;
    w.whole = item < p.n_whole;
    if (!w.whole) {
        half = item - p.n_whole;
        if (half >= p.n_half) {
            const int q = half - p.n_half;
            half = p.n_half + (q >> 1);
            quarter = q & 1;
            w.width = 128;
        }
    }
    const int whole_tiles = p.tiles_m * p.tiles_w;
    const int tile = w.whole ? item : p.n_whole + (half >> 1);
    if (tile < whole_tiles) {
        const int per_group = p.group_m * p.tiles_w;
        const int first_m = tile / per_group * p.group_m;
        const int gsize = p.tiles_m - first_m < p.group_m ? p.tiles_m - first_m : p.group_m;
        const int in_group = tile % per_group;
        w.tm = first_m + in_group % gsize;
        w.n0 = in_group / gsize * 512 + (w.whole ? 0 : (half & 1) * 256);
    } else {
        w.tm = half - 2 * (whole_tiles - p.n_whole);
        w.n0 = p.tiles_w * 512;
    }
    w.n0 += quarter * 128;
    return w;
}

__device__ __forceinline__ void tmem_load_16_issue(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_load_wait16(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

__device__ __forceinline__ void tma_load_pair_at(uint32_t smem_dst, const CUtensorMap *tmap, uint32_t leader_bar_addr, int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
        "[%2];" ::"r"(smem_dst),
        "l"(tmap), "r"(leader_bar_addr), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *tmap, uint32_t smem_src, int x, int y)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(smem_src), "r"(x),
                 "r"(y)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// 32 columns of the residual row, as 16-bit values; groups of 8 columns past n read as zero
__device__ __forceinline__ void load_residual32(const char *row, int columns, bool sectors, uint4 (&r)[4])
{
    if (columns >= 32 && sectors) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[2 * i].x), "=r"(r[2 * i].y), "=r"(r[2 * i].z), "=r"(r[2 * i].w), "=r"(r[2 * i + 1].x),
                           "=r"(r[2 * i + 1].y), "=r"(r[2 * i + 1].z), "=r"(r[2 * i + 1].w)
                         : "l"(row + 32 * i));
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r[i] = make_uint4(0u, 0u, 0u, 0u);
        if (columns >= 8 * (i + 1)) {
            r[i] = *reinterpret_cast<const uint4 *>(row + 16 * i);
        }
    }
}

// One warp's 32 rows (a lane each) of one accumulator go through two steps; 16-bit types throughout, one output.  First all
// `columns` (256 or 128) columns come out of tensor memory at taddr and are rounded to 16 bits, which the chain does ahead of the
// activation anyway, into 128 registers, and the accumulator is handed back.  Activation, second operator and stores then run
// under the next tile's products.
//
// kChain: how the accumulator becomes a 16-bit value.  0: rounded as it is (alpha = 1, no bias); 1: alpha * acc + bias in fp32,
// rounded, where the fused form rounds like the two steps (alpha = 1, or no bias); 2: the fp16 chain, alpha * acc rounded and the
// bias added in fp16; 3: alpha * acc rounded to fp32, then the sum with the bias.  Where there is no bias `stage` holds -0, which
// changes nothing.
template <int kDt, int kChain>
__device__ __forceinline__ void wide_drain(const EpiParams &e, uint32_t taddr, int columns, uint32_t stage, uint4 (&keep)[32])
{
    const float alpha = e.alpha;
    uint32_t raw[2][16];
    tmem_load_16_issue(taddr, raw[0]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (i == 8 && columns == 128) {
            break;
        }
        tmem_load_wait16(raw[i & 1]);
        if (i != 15 && (i != 7 || columns != 128)) {
            tmem_load_16_issue(taddr + static_cast<uint32_t>((i + 1) * 16), raw[(i + 1) & 1]);
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            float v[8], side[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = __uint_as_float(raw[i & 1][g * 8 + j]);
            }
            uint4 b;
            if (kChain != 0) {
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                             : "r"(stage + static_cast<uint32_t>((i * 16 + g * 8) * 2)));
            }
            if (kChain == 1 || kChain == 3) {
                unpack8<kDt>(b, side);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] = kChain == 1 ? fmaf(v[j], alpha, side[j]) : v[j] * alpha + side[j];
                }
            } else if (kChain == 2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] *= alpha;
                }
            }
            uint4 w = pack8_rne<kDt>(v);
            if (kChain == 2) {
                w = make_uint4(add2_packed<kDt>(w.x, b.x), add2_packed<kDt>(w.y, b.y), add2_packed<kDt>(w.z, b.z), add2_packed<kDt>(w.w, b.w));
            }
            keep[i * 2 + g] = w;
        }
    }
}

template <int kAct, int kDt, bool kSecond>
__device__ __forceinline__ void wide_finish(const WideParams &p, const CUtensorMap *tmap_out, int row0, int n0, int columns,
                                            uint32_t stage, int lane, uint4 (&keep)[32])
{
    const EpiParams &e = p.epi;
    const uint32_t my_row = stage + static_cast<uint32_t>(lane * 128);
    const uint32_t swz = static_cast<uint32_t>(lane & 7) << 4;
    // rows past m read the last row's residual
    const char *res_row = static_cast<const char *>(e.res) + (static_cast<long long>(row0 + lane < p.m ? row0 + lane : p.m - 1) * e.res_sm + n0) * 2;
    const bool res_sectors = ((reinterpret_cast<uintptr_t>(e.res) | static_cast<uintptr_t>(e.res_sm * 2)) & 31u) == 0;
    uint4 res[4];
    if (kSecond) {
        load_residual32(res_row, p.n - n0, res_sectors, res);
    }
#pragma unroll 1
    for (int c0 = 0; c0 < columns; c0 += 128) {  // rolled: all 256 columns would not fit the instruction cache
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 ahead[4];
            const int next = c0 + (q + 1) * 32;
            if (kSecond && next < columns) {
                load_residual32(res_row + next * 2, p.n - (n0 + next), res_sectors, ahead);
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint4 w = act8_packed<kAct, kDt>(e, keep[q * 4 + g]);
                if (kSecond) {
                    w = combine8_packed<kDt>(e, w, res[g]);
                    res[g] = ahead[g];
                }
                keep[q * 4 + g] = w;
            }
            if ((q & 1) == 0) {
                continue;
            }
            // 64 columns are 128 bytes of every row
            if (lane == 0) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the copy that read this warp's box before
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                const uint4 w = keep[(q - 1) * 4 + g];
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(my_row + ((static_cast<uint32_t>(g) << 4) ^ swz)), "r"(w.x),
                             "r"(w.y), "r"(w.z), "r"(w.w)
                             : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            const int column = n0 + c0 + (q - 1) * 32;
            if (lane == 0 && row0 < p.m && column < p.n) {
                tma_store_2d(tmap_out, stage, column, row0);
            }
        }
#pragma unroll
        for (int g = 0; g < 16; ++g) {
            keep[g] = keep[g + 16];
        }
    }
}

// The same for 8-bit integer products: exact 32-bit sums, a bias of 32-bit integers, clamped to their range; 32 columns at a time,
// 128 bytes of every row.  `box` is the one of the warp's two boxes that the next store leaves from: only stores alternate them, so
// that all but the newest have been read when one is used again.
__device__ __forceinline__ void wide_epilogue_int(const WideParams &p, const CUtensorMap *tmap_out, uint32_t taddr, int row0, int n0,
                                                  int columns, uint32_t stage, int lane, uint32_t drained, uint32_t &box)
{
    const EpiParams &e = p.epi;
    const uint32_t swz = static_cast<uint32_t>(lane & 7) << 4;
    uint32_t next[32], cur[32];
    tmem_load_16_issue(taddr, *reinterpret_cast<uint32_t(*)[16]>(&next[0]));
    tmem_load_16_issue(taddr + 16u, *reinterpret_cast<uint32_t(*)[16]>(&next[16]));
#pragma unroll 1
    for (int c0 = 0; c0 < columns; c0 += 32) {
        tmem_load_wait16(*reinterpret_cast<uint32_t(*)[16]>(&next[0]));
        tmem_load_wait16(*reinterpret_cast<uint32_t(*)[16]>(&next[16]));
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            cur[j] = next[j];
        }
        if (c0 + 32 < columns) {
            tmem_load_16_issue(taddr + static_cast<uint32_t>(c0 + 32), *reinterpret_cast<uint32_t(*)[16]>(&next[0]));
            tmem_load_16_issue(taddr + static_cast<uint32_t>(c0 + 48), *reinterpret_cast<uint32_t(*)[16]>(&next[16]));
        } else {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_cluster(drained);
            }
        }
        if (e.has_bias != 0) {
            const int mine = n0 + c0 + lane < p.n ? static_cast<const int *>(e.bias)[(n0 + c0 + lane) * e.bias_sn] : 0;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                int sum;
                asm("add.sat.s32 %0, %1, %2;" : "=r"(sum) : "r"(static_cast<int>(cur[j])), "r"(__shfl_sync(0xffffffffu, mine, j)));
                cur[j] = static_cast<uint32_t>(sum);
            }
        }
        if (row0 >= p.m || n0 + c0 >= p.n) {
            continue;
        }
        if (lane == 0) {
            asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        }
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + box + static_cast<uint32_t>(lane * 128) + ((static_cast<uint32_t>(g) << 4) ^ swz)),
                         "r"(cur[g * 4]), "r"(cur[g * 4 + 1]), "r"(cur[g * 4 + 2]), "r"(cur[g * 4 + 3])
                         : "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(tmap_out, stage + box, n0 + c0, row0);
        }
        box ^= static_cast<uint32_t>(kWarpStageBytes);
    }
}

// kScaled: alpha != 1 and a bias outside the fp16 chain.  An instance of its own: as one more case it cost the others 0.5 %.
template <int kKind, bool kScaled>
__global__ void __launch_bounds__(kWideThreads, 1)
    tc_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                   const __grid_constant__ CUtensorMap tmap_b64, const __grid_constant__ CUtensorMap tmap_out,
                   const __grid_constant__ WideParams p)
{
    constexpr int kElemsPerRow = kKind == KUDNN_B200_S8 ? 128 : 64;  // per 128-byte k-block row
    constexpr int kWideStages = WideShape<kKind>::kStages, kWideSmallStages = WideShape<kKind>::kSmallStages;
    constexpr int kBoxBytes = WideShape<kKind>::kBoxes * kWarpStageBytes;  // per warp
    extern __shared__ __align__(1024) unsigned char smem[];          // the swizzle pattern repeats every 1024 bytes
    unsigned char *staging = smem + WideShape<kKind>::kRing;
    uint64_t *bars = reinterpret_cast<uint64_t *>(staging + kEpiWarps * kBoxBytes);
    uint64_t *full_bar = bars;
    uint64_t *empty_bar = bars + kWideStages;
    uint64_t *small_full = bars + 2 * kWideStages;
    uint64_t *small_empty = small_full + kWideSmallStages;
    uint64_t *tmem_full = small_empty + kWideSmallStages;
    uint64_t *tmem_empty = tmem_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tmem_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if ((smem_u32(smem) & 1023u) != 0) {  // never: the declaration asks for the alignment.  Both CTAs would leave here.
        if (threadIdx.x == 0) {
            atomicCAS(&p.status->code, kErrNone, kErrTimeout);
        }
        return;
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWideStages; ++s) {
            mbar_init(full_bar + s, 1);
            mbar_init(empty_bar + s, 1);
        }
        for (int s = 0; s < kWideSmallStages; ++s) {
            mbar_init(small_full + s, 1);
            mbar_init(small_empty + s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tmem_full + a, 1);
            mbar_init(tmem_empty + a, kEpiWarps);  // four warps of either CTA
        }
        *abort_flag = 0;
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

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kWideControlRegs));
        if (warp == 0) {
            // ------------------------------------------------------------------ loads
            if (lane == 0) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_b) : "memory");
                const uint32_t ring = smem_u32(smem);
                // the barriers of the leader count both CTAs' bytes; only the leader announces them
                const uint32_t large_at = map_to_rank(smem_u32(full_bar), 0u), small_at = map_to_rank(smem_u32(small_full), 0u);
                auto load_b_whole = [&](int stage, int x, int row) {
                    if (rank == 0) {
                        mbar_expect_tx(full_bar + stage, 6 * kABytes);
                    }
                    const uint32_t at = ring + static_cast<uint32_t>(stage * kWideStageBytes + kABytes);
                    tma_load_pair_at(at, &tmap_b, large_at + static_cast<uint32_t>(stage * 8), x, row);
                    tma_load_pair_at(at + kABytes, &tmap_b, large_at + static_cast<uint32_t>(stage * 8), x, row + 256);
                };
                auto load_b_small = [&](const CUtensorMap *map, uint32_t bytes, int stage, int x, int row) {
                    if (rank == 0) {
                        mbar_expect_tx(small_full + stage, bytes);
                    }
                    tma_load_pair_at(ring + static_cast<uint32_t>(stage * kWideSmallBytes + kABytes), map, small_at + static_cast<uint32_t>(stage * 8), x, row);
                };
                // weights that only pre-packing writes are on their way before the previous kernel has ended
                int early = 0;
                if (p.b_stable != 0) {
                    const WideItem w = wide_item(p, first_item);
                    const int row = w.n0 + static_cast<int>(rank) * (w.width / 2);
                    const int stages = w.whole ? kWideStages : kWideSmallStages;
                    early = p.load_kb < stages ? p.load_kb : stages;
                    for (int i = 0; i < early; ++i) {
                        if (w.whole) {
                            load_b_whole(i, i * kElemsPerRow, row);
                        } else {
                            load_b_small(w.width == 256 ? &tmap_b : &tmap_b64, w.width == 256 ? 4 * kABytes : 3 * kABytes, i, i * kElemsPerRow, row);
                        }
                    }
                }
                pdl_wait();
                int stage = 0;
                uint32_t phase = 0;
                bool alive = true;
                int item = first_item;
                for (; alive && item < p.n_whole; item += stride) {
                    const WideItem w = wide_item(p, item);
                    const int a_row = w.tm * 256 + static_cast<int>(rank) * kBM, b_row = w.n0 + static_cast<int>(rank) * 128;
                    int x = 0;
                    for (int kb = 0; kb < p.load_kb; ++kb, x += kElemsPerRow) {
                        if (!mbar_wait(empty_bar + stage, phase ^ 1u, abort_flag, p.status, 1, p.wait_limit)) {
                            alive = false;
                            break;
                        }
                        if (early == 0) {
                            load_b_whole(stage, x, b_row);
                        } else {
                            --early;
                        }
                        tma_load_pair_at(ring + static_cast<uint32_t>(stage * kWideStageBytes), &tmap_a, large_at + static_cast<uint32_t>(stage * 8), x, a_row);
                        if (++stage == kWideStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                }
                // the small ring takes over when the products that still read the large one are done
                for (int i = 0; alive && item < p.num_items && i < kWideStages; ++i) {
                    alive = mbar_wait(empty_bar + stage, phase ^ 1u, abort_flag, p.status, 1, p.wait_limit);
                    if (++stage == kWideStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                stage = 0;
                phase = 0;
                for (; alive && item < p.num_items; item += stride) {
                    const WideItem w = wide_item(p, item);
                    const int a_row = w.tm * 256 + static_cast<int>(rank) * kBM, b_row = w.n0 + static_cast<int>(rank) * (w.width / 2);
                    const CUtensorMap *map = w.width == 256 ? &tmap_b : &tmap_b64;
                    const uint32_t bytes = w.width == 256 ? 4 * kABytes : 3 * kABytes;
                    int x = 0;
                    for (int kb = 0; kb < p.load_kb; ++kb, x += kElemsPerRow) {
                        if (!mbar_wait(small_empty + stage, phase ^ 1u, abort_flag, p.status, 1, p.wait_limit)) {
                            alive = false;
                            break;
                        }
                        if (early == 0) {
                            load_b_small(map, bytes, stage, x, b_row);
                        } else {
                            --early;
                        }
                        tma_load_pair_at(ring + static_cast<uint32_t>(stage * kWideSmallBytes), &tmap_a, small_at + static_cast<uint32_t>(stage * 8), x, a_row);
                        if (++stage == kWideSmallStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                }
            }
        } else if (warp == 1) {
            // ------------------------------------------------------------------ MMAs, issued by the leader for both CTAs
            if (lane == 0 && rank == 0) {
                pdl_wait();  // the limit of the waits below counts from here
                int stage = 0;
                uint32_t phase = 0;
                uint32_t uses[2] = {0, 0};
                int turn = 0;
                bool alive = true;
                auto advance = [&](int &s, uint32_t &ph) {
                    if (++s == kWideStages) {
                        s = 0;
                        ph ^= 1u;
                    }
                };
                auto wait_full = [&](int s, uint32_t ph) {
                    const bool ok = mbar_wait(full_bar + s, ph, abort_flag, p.status, 3, p.wait_limit);
                    tc_fence_after();
                    return ok;
                };
                auto wait_drained = [&](int acc) {
                    const bool ok = mbar_wait(tmem_empty + acc, (uses[acc] & 1u) ^ 1u, abort_flag, p.status, 2, p.wait_limit);
                    ++uses[acc];
                    tc_fence_after();
                    return ok;
                };
                // the four MMAs of a k-block at `at`; part: which B of the stage
                auto multiply_at = [&](int acc, int at, int part, uint32_t idesc, bool first) {
                    const uint32_t sa = smem_u32(smem + at);
                    const uint64_t adesc = make_smem_desc(sa);
                    const uint64_t bdesc = make_smem_desc(sa + kABytes + static_cast<uint32_t>(part) * kABytes);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        umma_pair<kKind>(tmem_base + static_cast<uint32_t>(acc * 256), adesc + static_cast<uint64_t>(2 * ks),
                                         bdesc + static_cast<uint64_t>(2 * ks), idesc, (!first || ks != 0) ? 1u : 0u);
                    }
                };
                auto multiply = [&](int acc, int s, int part, uint32_t idesc, bool first) {
                    multiply_at(acc, s * kWideStageBytes, part, idesc, first);
                };
                int small_stage = 0;
                uint32_t small_phase = 0;
                for (int item = first_item; alive && item < p.num_items; item += stride) {
                    const WideItem w = wide_item(p, item);
                    if (!w.whole) {
                        const int acc = turn;
                        turn ^= 1;
                        if (!wait_drained(acc)) {
                            break;
                        }
                        const uint32_t idesc = w.width == 256 ? p.idesc : p.idesc_quarter;
                        for (int kb = 0; alive && kb < p.num_kb; ++kb) {
                            alive = mbar_wait(small_full + small_stage, small_phase, abort_flag, p.status, 3, p.wait_limit);
                            tc_fence_after();
                            if (alive) {
                                multiply_at(acc, small_stage * kWideSmallBytes, 0, idesc, kb == 0);
                                umma_commit_pair(small_empty + small_stage);
                                if (++small_stage == kWideSmallStages) {
                                    small_stage = 0;
                                    small_phase ^= 1u;
                                }
                            }
                        }
                        if (alive) {
                            umma_commit_pair(tmem_full + acc);
                        }
                        continue;
                    }
                    // whole tile: the first and the last kWideSkew k-blocks go to one accumulator after the other
                    const int skew = p.num_kb < 2 * kWideSkew ? p.num_kb / 2 : kWideSkew;
                    if (!wait_drained(0)) {
                        break;
                    }
                    int s = stage;
                    uint32_t ph = phase;
                    for (int kb = 0; alive && kb < skew; ++kb) {
                        alive = wait_full(s, ph);
                        if (alive) {
                            multiply(0, s, 0, p.idesc, kb == 0);
                            advance(s, ph);
                        }
                    }
                    if (!alive || !wait_drained(1)) {
                        break;
                    }
                    for (int kb = 0; kb < skew; ++kb) {
                        multiply(1, stage, 1, p.idesc, kb == 0);
                        umma_commit_pair(empty_bar + stage);
                        advance(stage, phase);
                    }
                    for (int kb = skew; alive && kb < p.num_kb - skew; ++kb) {
                        alive = wait_full(stage, phase);
                        if (alive) {
                            multiply(0, stage, 0, p.idesc, kb == 0);
                            multiply(1, stage, 1, p.idesc, kb == 0);
                            umma_commit_pair(empty_bar + stage);
                            advance(stage, phase);
                        }
                    }
                    s = stage;
                    ph = phase;
                    for (int kb = 0; alive && kb < skew; ++kb) {
                        alive = wait_full(s, ph);
                        if (alive) {
                            multiply(0, s, 0, p.idesc, false);
                            advance(s, ph);
                        }
                    }
                    if (!alive) {
                        break;
                    }
                    umma_commit_pair(tmem_full + 0);
                    for (int kb = 0; kb < skew; ++kb) {
                        multiply(1, stage, 1, p.idesc, false);
                        umma_commit_pair(empty_bar + stage);
                        advance(stage, phase);
                    }
                    umma_commit_pair(tmem_full + 1);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kWideEpilogueRegs));
        // ------------------------------------------------------------------ epilogue warps, four per accumulator
        pdl_launch_dependents();  // only now that this CTA holds its tensor memory (see tc_linear_kernel)
        pdl_wait();
        const int quarter = warp & 3;  // tensor-memory lanes [32 * quarter, 32 * quarter + 32)
        const int acc = (warp - 4) / 4;
        const uint32_t stage = smem_u32(staging + (warp - 4) * kBoxBytes);
        const uint32_t drained = map_to_rank(smem_u32(tmem_empty + acc), 0u);
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * 256);
        const EpiParams &e = p.epi;
        uint32_t phase = 0, box = 0;
        int turn = 0;
        for (int item = first_item; item < p.num_items; item += stride) {
            const WideItem w = wide_item(p, item);
            if (!w.whole) {
                const int whose = turn;
                turn ^= 1;
                if (whose != acc) {
                    continue;
                }
            }
            const int n0 = w.n0 + (w.whole ? acc * 256 : 0);
            const int row0 = w.tm * 256 + static_cast<int>(rank) * kBM + quarter * 32;
            if constexpr (kKind != KUDNN_B200_S8) {
                // the bias waits in this warp's box, which the stores of the previous item have left
                if (lane == 0) {
                    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                }
                __syncwarp();
                for (int c = lane; c < w.width; c += 32) {
                    const unsigned short b = e.has_bias == 0 ? static_cast<unsigned short>(0x8000)
                                             : n0 + c < p.n  ? static_cast<const unsigned short *>(e.bias)[(n0 + c) * e.bias_sn]
                                                             : static_cast<unsigned short>(0);
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(stage + static_cast<uint32_t>(c * 2)), "h"(b) : "memory");
                }
                __syncwarp();
            }
            const bool arrived = __all_sync(0xffffffffu, mbar_wait(tmem_full + acc, phase, abort_flag, p.status, 4, p.wait_limit));
            phase ^= 1u;
            if (!arrived) {
                break;
            }
            tc_fence_after();
            if constexpr (kKind == KUDNN_B200_S8) {
                wide_epilogue_int(p, &tmap_out, taddr, row0, n0, w.width, stage, lane, drained, box);
            } else {
                uint4 keep[32];
                if constexpr (kScaled) {
                    wide_drain<kKind, 3>(e, taddr, w.width, stage, keep);
                } else if (e.alpha == 1.0f && e.has_bias == 0) {
                    wide_drain<kKind, 0>(e, taddr, w.width, stage, keep);
                } else if (kKind == KUDNN_B200_F16 && e.half_chain != 0) {
                    wide_drain<kKind, 2>(e, taddr, w.width, stage, keep);
                } else {
                    wide_drain<kKind, 1>(e, taddr, w.width, stage, keep);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(drained);
                }
#define KB_WIDE(ACT)                                                                           \
        if (e.res_op != KUDNN_B200_RES_NONE) {                                                     \
            wide_finish<ACT, kKind, true>(p, &tmap_out, row0, n0, w.width, stage, lane, keep);    \
        } else {                                                                                   \
            wide_finish<ACT, kKind, false>(p, &tmap_out, row0, n0, w.width, stage, lane, keep);   \
        }
                switch (e.act) {
                    case KUDNN_B200_ACT_NONE: KB_WIDE(KUDNN_B200_ACT_NONE); break;
                    case KUDNN_B200_ACT_RELU: KB_WIDE(KUDNN_B200_ACT_RELU); break;
                    case KUDNN_B200_ACT_SWISH: KB_WIDE(KUDNN_B200_ACT_SWISH); break;
                    default: KB_WIDE(KUDNN_B200_ACT_GELU_TANH); break;
                }
#undef KB_WIDE
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

template <int kKind>
cudaError_t launch_wide_one(const TcPlan &plan, const void *tmap_out, const WideParams &p, cudaStream_t stream)
{
    auto kernel = tc_wide_kernel<kKind, false>;
    if constexpr (kKind != KUDNN_B200_S8) {
        if (p.epi.alpha != 1.0f && p.epi.has_bias != 0 && (kKind != KUDNN_B200_F16 || p.epi.half_chain == 0)) {
            kernel = tc_wide_kernel<kKind, true>;
        }
    }
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) {
        return e;
    }
    CUtensorMap ta, tb, tb64, to;
    std::memcpy(&ta, plan.tmap_a, sizeof(ta));
    std::memcpy(&tb, plan.tmap_b, sizeof(tb));
    std::memcpy(&tb64, plan.tmap_b64, sizeof(tb64));
    std::memcpy(&to, tmap_out, sizeof(to));
    return launch_chained(kernel, dim3(static_cast<unsigned>(plan.grid)), dim3(kWideThreads), WideShape<kKind>::kSmem, stream, 2u, ta, tb, tb64, to, p);
}

// One translation unit per operand kind (tc_wide_*.cu).
template <int kKind>
cudaError_t launch_wide_kind(const TcPlan &plan, const void *tmap_out, const WideParams &p, cudaStream_t stream);
#define KB_WIDE_DECLARE(KIND) \
    template <>               \
    cudaError_t launch_wide_kind<KIND>(const TcPlan &plan, const void *tmap_out, const WideParams &p, cudaStream_t stream);
KB_WIDE_DECLARE(KUDNN_B200_F16)
KB_WIDE_DECLARE(KUDNN_B200_BF16)
KB_WIDE_DECLARE(KUDNN_B200_S8)
#undef KB_WIDE_DECLARE

}  // namespace tc

}  // namespace kb
