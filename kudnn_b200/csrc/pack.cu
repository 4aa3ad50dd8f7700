// Operand packing: brings an arbitrarily strided [rows, k] operand into the K-major, 16-byte aligned form the
// tensor-core and streaming kernels read, converting the element type on the way.  fp32 operands are split
// into TF32 planes here.  The reference does the corresponding work per call and per thread inside its JIT
// GEMM (pack routines, src/dnn/src/matmul_jit/MatrixComputation/kudnn_default_impl_fp16fp16f32f32.cpp:929-962)
// and through ReorderLayer for type conversion (src/dnn/src/kudnn_gemm.cpp:36-63).
#include "kernels.cuh"

namespace kb {

namespace {

__device__ __forceinline__ void store_converted(void *dst, int dtype, long long idx, float v)
{
    if (dtype == KUDNN_B200_F32) {
        static_cast<float *>(dst)[idx] = v;
    } else if (dtype == KUDNN_B200_F16) {
        static_cast<unsigned short *>(dst)[idx] = f32_to_f16_rne_bits(v);
    } else if (dtype == KUDNN_B200_S8) {
        static_cast<signed char *>(dst)[idx] = static_cast<signed char>(static_cast<int>(v));  // 8-bit values are exact in fp32
    } else if (dtype == KUDNN_B200_U8) {
        static_cast<unsigned char *>(dst)[idx] = static_cast<unsigned char>(static_cast<int>(v));
    } else {
        static_cast<unsigned short *>(dst)[idx] = f32_to_bf16_rne_bits(v);
    }
}

// 32 x 32 tile through shared memory so both the strided read and the K-major write are coalesced
// blockIdx.z = flat batch index: the source matrix of a batch entry starts at the element offset its three batch
// strides give, the packed one at flat * dst_batch elements
__device__ __forceinline__ long long src_batch_offset(const PackBatch &pb, long long flat)
{
    const long long i2 = flat % pb.n2, r = flat / pb.n2;
    return (r / pb.n1) * pb.sb[0] + (r % pb.n1) * pb.sb[1] + i2 * pb.sb[2];
}

__global__ void __launch_bounds__(256) pack_kmajor_kernel(const void *src_base, int src_dtype, long long rows, long long k,
                                                          long long s_row, long long s_k, void *dst_base, int dst_dtype,
                                                          long long ldd, long long k_pad, const PackBatch pb)
{
    __shared__ float tile[32][33];
    const void *src = static_cast<const char *>(src_base) + src_batch_offset(pb, blockIdx.z) * dtype_size(src_dtype);
    void *dst = static_cast<char *>(dst_base) + static_cast<long long>(blockIdx.z) * pb.dst_batch * dtype_size(dst_dtype);
    const long long r0 = static_cast<long long>(blockIdx.x) * 32;
    const long long k0 = static_cast<long long>(blockIdx.y) * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const bool rows_fast = (s_row == 1 && s_k != 1);
    for (int i = ty; i < 32; i += 8) {
        // rows_fast: tx walks rows (unit stride in memory), i walks k; otherwise tx walks k
        const long long r = rows_fast ? r0 + tx : r0 + i;
        const long long kk = rows_fast ? k0 + i : k0 + tx;
        float v = 0.0f;
        if (r < rows && kk < k) {
            v = load_as_f32(src, src_dtype, r * s_row + kk * s_k);
        }
        if (rows_fast) {
            tile[tx][i] = v;
        } else {
            tile[i][tx] = v;
        }
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
        const long long r = r0 + i, kk = k0 + tx;
        if (r < rows && kk < k_pad) {
            store_converted(dst, dst_dtype, r * ldd + kk, tile[i][tx]);
        }
    }
}

__device__ __forceinline__ float to_tf32(float x)
{
    unsigned u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
    return __uint_as_float(u);
}

// dst row (pitch ldd floats) starts with three planes of k_pad floats.  Activations: [lo | hi | hi]; weights: [hi | lo | hi].
__global__ void __launch_bounds__(256) split_tf32_kernel(const float *src_base, long long rows, long long k, long long s_row,
                                                         long long s_k, float *dst_base, long long ldd, long long k_pad,
                                                         int is_weight, const PackBatch pb)
{
    __shared__ float tile[32][33];
    const float *src = src_base + src_batch_offset(pb, blockIdx.z);
    float *dst = dst_base + static_cast<long long>(blockIdx.z) * pb.dst_batch;
    const long long r0 = static_cast<long long>(blockIdx.x) * 32;
    const long long k0 = static_cast<long long>(blockIdx.y) * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const bool rows_fast = (s_row == 1 && s_k != 1);
    for (int i = ty; i < 32; i += 8) {
        const long long r = rows_fast ? r0 + tx : r0 + i;
        const long long kk = rows_fast ? k0 + i : k0 + tx;
        float v = 0.0f;
        if (r < rows && kk < k) {
            v = src[r * s_row + kk * s_k];
        }
        if (rows_fast) {
            tile[tx][i] = v;
        } else {
            tile[i][tx] = v;
        }
    }
    __syncthreads();
    for (int i = ty; i < 32; i += 8) {
        const long long r = r0 + i, kk = k0 + tx;
        if (r < rows && kk < k_pad) {
            const float v = tile[i][tx];
            const float hi = to_tf32(v);
            const float lo = to_tf32(v - hi);
            float *row = dst + r * ldd;
            if (is_weight) {
                row[kk] = hi;
                row[k_pad + kk] = lo;
            } else {
                row[kk] = lo;
                row[k_pad + kk] = hi;
            }
            row[2 * k_pad + kk] = hi;
        }
    }
}

// ---- rows that are contiguous along k already (activations, per call): no transpose, one 16-byte piece of the packed row
// per thread.  Bound by memory; the 32 x 32 transpose above reads and writes element by element and took 5 us for what
// these finish in the shadow of the next kernel's launch.
// kBytes-wide elements of one type; the source rows start anywhere.
template <int kBytes>
__global__ void __launch_bounds__(256) pack_rows_kernel(const void *src_base, long long k, long long s_row, void *dst_base, long long ldd,
                                                        long long pieces, const PackBatch pb)
{
    constexpr int kVec = 16 / kBytes;
    pdl_launch_dependents();
    pdl_wait();
    const long long piece = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    if (piece >= pieces) {
        return;
    }
    const long long row = blockIdx.y + static_cast<long long>(gridDim.y) * (blockIdx.z % pb.row_slices);
    const long long flat = blockIdx.z / pb.row_slices;
    if (row >= pb.rows) {
        return;
    }
    const unsigned char *src = static_cast<const unsigned char *>(src_base) + (src_batch_offset(pb, flat) + row * s_row + piece * kVec) * kBytes;
    const long long left = (k - piece * kVec) * kBytes;  // bytes of this piece that exist
    unsigned w[4] = {0u, 0u, 0u, 0u};
    if (left >= 16 && (reinterpret_cast<uintptr_t>(src) & 3u) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = reinterpret_cast<const unsigned *>(src)[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < kVec; ++i) {
            if (i * kBytes < left) {
                const unsigned v = kBytes == 2 ? reinterpret_cast<const unsigned short *>(src)[i] : src[i];
                w[i * kBytes / 4] |= v << (8 * (i * kBytes % 4));
            }
        }
    }
    reinterpret_cast<uint4 *>(static_cast<unsigned char *>(dst_base) + (flat * pb.dst_batch + row * ldd) * kBytes)[piece] =
        make_uint4(w[0], w[1], w[2], w[3]);
}

// fp32 rows -> TF32 planes, four columns per thread
__global__ void __launch_bounds__(256) split_rows_kernel(const float *src_base, long long k, long long s_row, float *dst_base,
                                                         long long ldd, long long k_pad, int is_weight, const PackBatch pb)
{
    pdl_launch_dependents();
    pdl_wait();
    const long long kk = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * 4;
    const long long row = blockIdx.y + static_cast<long long>(gridDim.y) * (blockIdx.z % pb.row_slices);
    const long long flat = blockIdx.z / pb.row_slices;
    if (kk >= k_pad || row >= pb.rows) {
        return;
    }
    const float *src = src_base + src_batch_offset(pb, flat) + row * s_row + kk;
    float v[4];
    if (kk + 4 <= k && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        const float4 x = *reinterpret_cast<const float4 *>(src);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = kk + i < k ? src[i] : 0.0f;
        }
    }
    float hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        hi[i] = to_tf32(v[i]);
        lo[i] = to_tf32(v[i] - hi[i]);
    }
    const float4 h = make_float4(hi[0], hi[1], hi[2], hi[3]), l = make_float4(lo[0], lo[1], lo[2], lo[3]);
    float *dst = dst_base + flat * pb.dst_batch + row * ldd + kk;
    *reinterpret_cast<float4 *>(dst) = is_weight ? h : l;
    *reinterpret_cast<float4 *>(dst + k_pad) = is_weight ? l : h;
    *reinterpret_cast<float4 *>(dst + 2 * k_pad) = h;
}

// The same split of activation rows (contiguous, on 16 bytes) by CTAs that walk over the rows, and only if *run_if is not 0: the
// launch that otherwise leaves at once has to be small.
__global__ void __launch_bounds__(256) split_rows_if_kernel(const int *run_if, const float *src_base, long long rows, long long k, long long s_row,
                                                            float *dst_base, long long ldd, long long k_pad)
{
    pdl_launch_dependents();
    pdl_wait();
    if (*run_if == 0) {
        return;
    }
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        const float *src = src_base + row * s_row;
        float *dst = dst_base + row * ldd;
        for (long long kk = threadIdx.x * 4; kk < k_pad; kk += 1024) {
            float4 v;
            if (kk + 4 <= k) {
                v = *reinterpret_cast<const float4 *>(src + kk);
            } else {
                v = make_float4(kk < k ? src[kk] : 0.0f, kk + 1 < k ? src[kk + 1] : 0.0f, kk + 2 < k ? src[kk + 2] : 0.0f, 0.0f);
            }
            const float4 h = make_float4(to_tf32(v.x), to_tf32(v.y), to_tf32(v.z), to_tf32(v.w));
            const float4 l = make_float4(to_tf32(v.x - h.x), to_tf32(v.y - h.y), to_tf32(v.z - h.z), to_tf32(v.w - h.w));
            *reinterpret_cast<float4 *>(dst + kk) = l;
            *reinterpret_cast<float4 *>(dst + k_pad + kk) = h;
            *reinterpret_cast<float4 *>(dst + 2 * k_pad + kk) = h;
        }
    }
}

// fp32 rows -> two planes of fp16 (see tc_planes.cuh): a CTA per row, eight columns per thread and step.  Bound by memory: the row
// is read once (rows of up to 8192 columns stay in registers between the search for the largest element and the conversion) and as
// many bytes are written.
//
// The low plane has all of its bits for elements from 2^-14 on after scaling: an error of 2^-37 there, 2^-23 of the element, as in
// the TF32 planes at any size.  Smaller ones would lose a bit for every factor of two, so they go to the row's list.
constexpr int kSplitThreads = 128, kSplitHeld = 8;

__global__ void __launch_bounds__(kSplitThreads, 6) split_half_kernel(const float *src_base, long long k, long long s_row, const PlanesOperand to,
                                                                   long long k_pad)
{
    __shared__ unsigned most[kSplitThreads / 32], least[kSplitThreads / 32];
    __shared__ int left_out;
    __shared__ PlanesElement rest[kPlanesRest];
    if (threadIdx.x == 0) {
        left_out = 0;
    }
    pdl_launch_dependents();
    pdl_wait();
    const long long row = blockIdx.x;
    const float *src = src_base + row * s_row;
    const int pieces = static_cast<int>(k_pad / 8);
    auto fetch = [&](int piece, float (&v)[8]) {
        const long long kk = static_cast<long long>(piece) * 8;
        if (piece < pieces && kk + 8 <= k) {
            const float4 x = *reinterpret_cast<const float4 *>(src + kk), y = *reinterpret_cast<const float4 *>(src + kk + 4);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = piece < pieces && kk + i < k ? src[kk + i] : 0.0f;
            }
        }
    };
    // the largest magnitude and the smallest that is not zero, as bit patterns
    unsigned mx = 0u, mn = 0xffffffffu;
    auto look = [&](const float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned u = __float_as_uint(v[i]) & 0x7fffffffu;
            mx = mx > u ? mx : u;
            mn = u != 0u && u < mn ? u : mn;
        }
    };
    float held[kSplitHeld][8];
    const bool holds = pieces <= kSplitThreads * kSplitHeld;
    if (holds) {
#pragma unroll
        for (int j = 0; j < kSplitHeld; ++j) {
            if (j * kSplitThreads < pieces) {
                fetch(j * kSplitThreads + static_cast<int>(threadIdx.x), held[j]);
                look(held[j]);
            }
        }
    } else {
        for (int piece = static_cast<int>(threadIdx.x); piece < pieces; piece += kSplitThreads) {
            fetch(piece, held[0]);
            look(held[0]);
        }
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    mn = __reduce_min_sync(0xffffffffu, mn);
    if ((threadIdx.x & 31) == 0) {
        most[threadIdx.x >> 5] = mx;
        least[threadIdx.x >> 5] = mn;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kSplitThreads / 32; ++w) {
        mx = most[w] > mx ? most[w] : mx;
        mn = least[w] < mn ? least[w] : mn;
    }
    const int exponent = static_cast<int>(mx >> 23) - 127;
    const bool in_range = mx == 0u || (exponent >= -100 && exponent < 64);
    // 2^(14 - exponent) and its inverse
    const float up = mx == 0u || !in_range ? 1.0f : __uint_as_float(static_cast<unsigned>(127 + 14 - exponent) << 23);
    const float down = mx == 0u || !in_range ? 1.0f : __uint_as_float(static_cast<unsigned>(127 - 14 + exponent) << 23);
    const float smallest = mn != 0xffffffffu && in_range ? __uint_as_float(mn) * up : 1.0f;
    const bool some_small = smallest < 0x1p-14f;
    unsigned short *dst = to.planes + row * 2 * k_pad;
    auto put = [&](int piece, const float (&v)[8]) {
        if (piece >= pieces) {
            return;
        }
        unsigned hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float x = v[2 * i] * up, y = v[2 * i + 1] * up;
            const __half2 h = __floats2half2_rn(x, y);
            const float2 back = __half22float2(h);
            const __half2 l = __floats2half2_rn((x - back.x) * 4096.0f, (y - back.y) * 4096.0f);
            hi[i] = *reinterpret_cast<const unsigned *>(&h);
            lo[i] = *reinterpret_cast<const unsigned *>(&l);
        }
        uint4 *at = reinterpret_cast<uint4 *>(dst + (piece >> 3) * 128 + (piece & 7) * 8);
        at[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        at[8] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    };
    if (holds) {
#pragma unroll
        for (int j = 0; j < kSplitHeld; ++j) {
            if (j * kSplitThreads < pieces) {
                put(j * kSplitThreads + static_cast<int>(threadIdx.x), held[j]);
            }
        }
    } else {
        for (int piece = static_cast<int>(threadIdx.x); piece < pieces; piece += kSplitThreads) {
            fetch(piece, held[0]);
            put(piece, held[0]);
        }
    }
    if (some_small) {
        // rare, and so a pass of its own over the row, now that its planes are written
        __syncthreads();
#pragma unroll 1
        for (int piece = static_cast<int>(threadIdx.x); piece < pieces; piece += kSplitThreads) {
            fetch(piece, held[0]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (held[0][i] != 0.0f && fabsf(held[0][i] * up) < 0x1p-14f) {
                    const int slot = atomicAdd(&left_out, 1);
                    if (slot < kPlanesRest) {
                        rest[slot] = PlanesElement{piece * 8 + i, held[0][i]};
                    }
                    unsigned short *at = dst + (piece >> 3) * 128 + (piece & 7) * 8 + i;
                    at[0] = at[64] = 0;
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        to.scale[row] = down;
        unsigned char mark = !in_range || smallest < 0x1p-46f ? kPlanesNot : 0;
        if (some_small && mark == 0) {
            const int count = left_out;
            mark = count <= kPlanesRest ? kPlanesLeft : kPlanesNot;
            PlanesElement *list = to.rest + row * kPlanesRest;
            for (int i = 0; mark == kPlanesLeft && i < count; ++i) {  // by column: the slots were taken in any order
                int at = 0;
                for (int j = 0; j < count; ++j) {
                    at += rest[j].k < rest[i].k ? 1 : 0;
                }
                list[at] = rest[i];
            }
            if (count < kPlanesRest) {
                list[count] = PlanesElement{-1, 0.0f};
            }
        }
        to.flags[row] = mark;
    }
    if (row == static_cast<long long>(gridDim.x) - 1 && threadIdx.x < static_cast<unsigned>(-gridDim.x & 15u)) {
        to.flags[row + 1 + threadIdx.x] = 0;
    }
}

// one thread per 16-byte chunk of the destination
__global__ void __launch_bounds__(256) pack_blocks_kernel(const unsigned short *src, long long rows, long long k, long long ld,
                                                          uint4 *dst, long long nkb, long long total_chunks)
{
    const long long idx = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    if (idx >= total_chunks) {
        return;
    }
    // position in the block -> (row, 16-byte chunk): byte (c & 1) * 512 + (4 r + c / 2) * 16 holds chunk c of row r
    const int pos = static_cast<int>(idx & 63);
    const int r = (pos & 31) >> 2, c = (pos & 3) * 2 + (pos >> 5);
    const long long blk = idx >> 6;
    const long long kb = blk % nkb, g = blk / nkb;
    const long long row = g * 8 + r, kk = kb * 64 + c * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows && kk < k) {  // k is a multiple of 8: a chunk is inside the row or outside of it
        v = *reinterpret_cast<const uint4 *>(src + row * ld + kk);
    }
    dst[idx] = v;
}

}  // namespace

cudaError_t launch_pack_blocks(const void *src, long long rows, long long k, long long ld, void *dst, long long k_pad,
                               cudaStream_t stream)
{
    const long long nkb = k_pad / 64;
    const long long total = (rows + 7) / 8 * nkb * 64;
    const long long blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffll) {
        return cudaErrorInvalidValue;
    }
    pack_blocks_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(static_cast<const unsigned short *>(src), rows, k, ld,
                                                                          static_cast<uint4 *>(dst), nkb, total);
    return cudaGetLastError();
}

namespace {

// Grid of the row kernels: 256 pieces x a row x (batch entry, slice of 65535 rows); false when it does not fit.
bool row_grid(long long pieces, long long rows, PackBatch *pb, dim3 *grid)
{
    const long long y = rows < 65535 ? rows : 65535;
    const long long slices = (rows + y - 1) / y;
    if (slices * pb->count > 65535) {
        return false;
    }
    pb->rows = rows;
    pb->row_slices = slices;
    *grid = dim3(static_cast<unsigned>((pieces + 255) / 256), static_cast<unsigned>(y), static_cast<unsigned>(slices * pb->count));
    return true;
}

}  // namespace

cudaError_t launch_pack_kmajor(const void *src, int src_dtype, long long rows, long long k, long long s_row,
                               long long s_k, void *dst, int dst_dtype, long long ldd, long long k_pad,
                               cudaStream_t stream, const PackBatch *batch)
{
    const PackBatch one = {1, 1, 1, {0, 0, 0}, 0};
    const PackBatch &pb = batch != nullptr ? *batch : one;
    dim3 grid;
    const int es = dtype_size(dst_dtype), vec = 16 / es;
    PackBatch by_row = pb;
    if (s_k == 1 && src_dtype == dst_dtype && es < 4 && k_pad % vec == 0 && ldd % vec == 0 && pb.dst_batch % vec == 0 &&
        (reinterpret_cast<uintptr_t>(dst) & 15u) == 0 && row_grid(k_pad / vec, rows, &by_row, &grid)) {
        return es == 2 ? launch_chained(pack_rows_kernel<2>, grid, dim3(256), 0, stream, 1, src, k, s_row, dst, ldd, k_pad / vec, by_row)
                       : launch_chained(pack_rows_kernel<1>, grid, dim3(256), 0, stream, 1, src, k, s_row, dst, ldd, k_pad / vec, by_row);
    }
    grid = dim3(static_cast<unsigned>((rows + 31) / 32), static_cast<unsigned>((k_pad + 31) / 32), static_cast<unsigned>(pb.count));
    if (grid.y > 65535 || pb.count > 65535) {
        return cudaErrorInvalidValue;
    }
    pack_kmajor_kernel<<<grid, 256, 0, stream>>>(src, src_dtype, rows, k, s_row, s_k, dst, dst_dtype, ldd, k_pad, pb);
    return cudaGetLastError();
}

cudaError_t launch_split_tf32(const void *src, long long rows, long long k, long long s_row, long long s_k, float *dst,
                              long long ldd, long long k_pad, int is_weight, cudaStream_t stream, const PackBatch *batch)
{
    const PackBatch one = {1, 1, 1, {0, 0, 0}, 0};
    const PackBatch &pb = batch != nullptr ? *batch : one;
    dim3 grid;
    PackBatch by_row = pb;
    if (s_k == 1 && k_pad % 4 == 0 && ldd % 4 == 0 && pb.dst_batch % 4 == 0 && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0 &&
        row_grid(k_pad / 4, rows, &by_row, &grid)) {
        return launch_chained(split_rows_kernel, grid, dim3(256), 0, stream, 1, static_cast<const float *>(src), k, s_row, dst, ldd, k_pad,
                              is_weight, by_row);
    }
    grid = dim3(static_cast<unsigned>((rows + 31) / 32), static_cast<unsigned>((k_pad + 31) / 32), static_cast<unsigned>(pb.count));
    if (grid.y > 65535 || pb.count > 65535) {
        return cudaErrorInvalidValue;
    }
    split_tf32_kernel<<<grid, 256, 0, stream>>>(static_cast<const float *>(src), rows, k, s_row, s_k, dst, ldd, k_pad,
                                                is_weight, pb);
    return cudaGetLastError();
}

cudaError_t launch_split_tf32_if(const int *run_if, const void *src, long long rows, long long k, long long s_row, float *dst, long long ldd,
                                 long long k_pad, int sm_count, cudaStream_t stream)
{
    const long long grid = rows < 4ll * sm_count ? rows : 4ll * sm_count;
    return launch_chained(split_rows_if_kernel, dim3(static_cast<unsigned>(grid)), dim3(256), 0, stream, 1, run_if, static_cast<const float *>(src),
                          rows, k, s_row, dst, ldd, k_pad);
}

cudaError_t launch_split_half(const void *src, long long rows, long long k, long long s_row, const PlanesOperand &dst, long long k_pad,
                              cudaStream_t stream)
{
    return launch_chained(split_half_kernel, dim3(static_cast<unsigned>(rows)), dim3(kSplitThreads), 0, stream, 1, static_cast<const float *>(src), k,
                          s_row, dst, k_pad);
}

}  // namespace kb
