// General Linear kernel: any element strides, any of the three float storage types per tensor, any size,
// leading batch dimensions with broadcast.  fp32 FMA accumulation, in ascending k (large tiles) or in four interleaved parts
// that are added in order (few tiles).  The kernel of large tiles with 32-bit integer
// accumulators is the 8-bit integer product <s8|u8, s8|u8, s32, s32> of the reference
// (src/dnn/src/kudnn_gemm.cpp:259-334): exact sums, an optional s32 bias, no post-operation.  It covers the shapes the
// tensor-core and streaming kernels decline (rows that are not 16-byte aligned, tiny problems, transposed
// activations) and serves as the on-device cross-check of the fast kernels.
//
// Work decomposition: one CTA per 64x64 output tile per batch entry, 256 threads, 4x4 outputs per thread,
// k advanced 16 at a time through shared memory; with fewer than two waves of such tiles 32x32 outputs per CTA
// (simt_small_kernel).  The role of these kernels in the reference is the batched loop around the BLAS call,
// src/dnn/src/kudnn_gemm.cpp:710-824.
#include "kernels.cuh"

namespace kb {

namespace {

constexpr int kTile = 64;
constexpr int kStepK = 16;

struct SimtParams {
    const void *a;
    const void *b;
    long long a_sm, a_sk, b_sk, b_sn;
    int a_dtype, b_dtype;
    int m, n, k;
    EpiParams epi;
    BatchParams batch;
};

__device__ __forceinline__ int load_as_int(const void *p, int dtype, long long idx)
{
    return dtype == KUDNN_B200_S8 ? static_cast<int>(static_cast<const signed char *>(p)[idx])
                                  : static_cast<int>(static_cast<const unsigned char *>(p)[idx]);
}

// c = alpha * acc + beta * c_old + bias for 32-bit integer results.  With alpha = 1 and beta = 0 or 1 (what the
// reference's callers use) everything stays in integers; other scalars go through fp64 and round to nearest.
__device__ __forceinline__ void epilogue_int(const EpiParams &p, int acc, long long mi, long long ni)
{
    int *c = static_cast<int *>(p.c);
    const long long ic = mi * p.c_sm + ni * p.c_sn;
    long long r = acc;
    if (p.alpha != 1.0f || (p.beta != 0.0f && p.beta != 1.0f)) {
        double t = static_cast<double>(p.alpha) * acc;
        if (p.beta != 0.0f) {
            t += static_cast<double>(p.beta) * c[ic];
        }
        r = llrint(t);
    } else if (p.beta == 1.0f) {
        r += c[ic];
    }
    if (p.has_bias) {
        r += static_cast<const int *>(p.bias)[mi * p.bias_sm + ni * p.bias_sn];
    }
    r = r > 2147483647ll ? 2147483647ll : (r < -2147483648ll ? -2147483648ll : r);
    c[ic] = static_cast<int>(r);
}

// ---- the same product for problems of few tiles, where latency counts: 32 x 32 outputs per CTA, and K cut between four
// groups of 64 threads.  A group advances 16 k at a time on its own (a named barrier), with the next step's operands on
// their way to registers while the current one is multiplied; the four partial sums are added in group order, and each of
// the 256 threads finishes four outputs.  Bound by the round trips to memory: one per 64 k, one for the side inputs.
constexpr int kSmallTile = 32;
constexpr int kSmallGroups = 4;
constexpr int kSmallPitch = kSmallTile + 4;

__global__ void __launch_bounds__(256) simt_small_kernel(const SimtParams p)
{
    __shared__ __align__(16) float sa[kSmallGroups][kStepK][kSmallPitch];
    __shared__ __align__(16) float sb[kSmallGroups][kStepK][kSmallPitch];
    __shared__ __align__(16) float sums[kSmallGroups][kSmallTile][kSmallPitch];

    const int tid = threadIdx.x;
    const int group = tid / 64, t = tid % 64;
    const int tx = t % 8, ty = t / 8;
    const long long m0 = static_cast<long long>(blockIdx.y) * kSmallTile;
    const long long n0 = static_cast<long long>(blockIdx.x) * kSmallTile;

    pdl_launch_dependents();
    long long bidx[3];
    batch_decompose(p.batch, blockIdx.z, bidx);
    const void *a = offset_ptr(p.a, p.a_dtype, batch_offset(p.batch.a_sb, bidx));
    const void *b = offset_ptr(p.b, p.b_dtype, batch_offset(p.batch.b_sb, bidx));
    pdl_wait();

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0.0f;
        }
    }

    // this thread's 8 elements of each operand per step: the walk order follows whichever stride is unit
    const bool a_by_k = p.a_sk == 1, b_by_k = p.b_sk == 1;
    const int a_r = a_by_k ? t / kStepK : t % kSmallTile, a_k = a_by_k ? t % kStepK : t / kSmallTile;
    const int b_r = b_by_k ? t / kStepK : t % kSmallTile, b_k = b_by_k ? t % kStepK : t / kSmallTile;
    const int a_dr = a_by_k ? 64 / kStepK : 0, a_dk = a_by_k ? 0 : 64 / kSmallTile;
    const int b_dr = b_by_k ? 64 / kStepK : 0, b_dk = b_by_k ? 0 : 64 / kSmallTile;
    float va[8], vb[8];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const long long ra = m0 + a_r + e * a_dr, ka = k0 + a_k + e * a_dk;
            const long long rb = n0 + b_r + e * b_dr, kb = k0 + b_k + e * b_dk;
            va[e] = ra < p.m && ka < p.k ? load_as_f32(a, p.a_dtype, ra * p.a_sm + ka * p.a_sk) : 0.0f;
            vb[e] = rb < p.n && kb < p.k ? load_as_f32(b, p.b_dtype, rb * p.b_sn + kb * p.b_sk) : 0.0f;
        }
    };
    int k0 = group * kStepK;
    if (k0 < p.k) {
        fetch(k0);
    }
    for (; k0 < p.k; k0 += kSmallGroups * kStepK) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            sa[group][a_k + e * a_dk][a_r + e * a_dr] = va[e];
            sb[group][b_k + e * b_dk][b_r + e * b_dr] = vb[e];
        }
        asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory");
        if (k0 + kSmallGroups * kStepK < p.k) {
            fetch(k0 + kSmallGroups * kStepK);
        }
#pragma unroll
        for (int kk = 0; kk < kStepK; ++kk) {
            const float4 av = *reinterpret_cast<const float4 *>(&sa[group][kk][ty * 4]);
            const float4 bv = *reinterpret_cast<const float4 *>(&sb[group][kk][tx * 4]);
            const float x[4] = {av.x, av.y, av.z, av.w}, y[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
                }
            }
        }
        asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory");
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<float4 *>(&sums[group][ty * 4 + i][tx * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();

    const int row = tid / 8, col = (tid % 8) * 4;
    const long long mi = m0 + row;
    if (mi >= p.m || n0 + col >= p.n) {
        return;
    }
    const EpiParams &e = p.epi;
    void *c = offset_ptr(e.c, e.c_dtype, batch_offset(p.batch.c_sb, bidx));
    const void *bias = offset_ptr(e.bias, e.bias_dtype, batch_offset(p.batch.bias_sb, bidx));
    const void *res = offset_ptr(e.res, e.res_dtype, batch_offset(p.batch.res_sb, bidx));
    void *out = offset_ptr(e.out, e.out_dtype, batch_offset(p.batch.out_sb, bidx));
    float old[4], bv[4], rv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long ni = n0 + col + j;
        old[j] = bv[j] = rv[j] = 0.0f;
        if (ni < p.n) {
            if (e.beta != 0.0f && c != nullptr) {
                old[j] = load_as_f32(c, e.c_dtype, mi * e.c_sm + ni * e.c_sn);
            }
            if (e.has_bias) {
                bv[j] = load_as_f32(bias, e.bias_dtype, mi * e.bias_sm + ni * e.bias_sn);
            }
            if (e.res_op != KUDNN_B200_RES_NONE) {
                rv[j] = load_as_f32(res, e.res_dtype, mi * e.res_sm + ni * e.res_sn);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long ni = n0 + col + j;
        if (ni < p.n) {
            float sum = 0.0f;
#pragma unroll
            for (int g = 0; g < kSmallGroups; ++g) {
                sum += sums[g][row][col + j];
            }
            const EpiResult r = finish_element(e, sum, old[j], bv[j], rv[j]);
            if (c != nullptr) {
                store_exact_mirrored(c, e.c_dtype, mi * e.c_sm + ni * e.c_sn, r.c, e.n_mirrors, e.c_delta);
            }
            if (e.res_op != KUDNN_B200_RES_NONE) {
                store_exact_mirrored(out, e.out_dtype, mi * e.out_sm + ni * e.out_sn, r.out, e.n_mirrors, e.out_delta);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) simt_linear_kernel(const SimtParams p)
{
    constexpr bool kInt = sizeof(T) == sizeof(int) && T(1) / T(2) == T(0);
    __shared__ T sa[kStepK][kTile + 4];
    __shared__ T sb[kStepK][kTile + 4];

    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const long long m0 = static_cast<long long>(blockIdx.y) * kTile;
    const long long n0 = static_cast<long long>(blockIdx.x) * kTile;

    long long bidx[3];
    batch_decompose(p.batch, blockIdx.z, bidx);
    const void *a = offset_ptr(p.a, p.a_dtype, batch_offset(p.batch.a_sb, bidx));
    const void *b = offset_ptr(p.b, p.b_dtype, batch_offset(p.batch.b_sb, bidx));
    const EpiParams epi = epi_for_batch(p.epi, p.batch, blockIdx.z);

    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = T(0);
        }
    }

    for (int k0 = 0; k0 < p.k; k0 += kStepK) {
        // 64 x 16 elements of each operand, 4 per thread; the walk order follows whichever stride is unit
        for (int e = tid; e < kTile * kStepK; e += 256) {
            int r, kk;
            if (p.a_sk == 1) {
                kk = e % kStepK;
                r = e / kStepK;
            } else {
                r = e % kTile;
                kk = e / kTile;
            }
            T v = T(0);
            if (m0 + r < p.m && k0 + kk < p.k) {
                const long long idx = (m0 + r) * p.a_sm + static_cast<long long>(k0 + kk) * p.a_sk;
                v = kInt ? static_cast<T>(load_as_int(a, p.a_dtype, idx)) : static_cast<T>(load_as_f32(a, p.a_dtype, idx));
            }
            sa[kk][r] = v;
        }
        for (int e = tid; e < kTile * kStepK; e += 256) {
            int c, kk;
            if (p.b_sk == 1) {
                kk = e % kStepK;
                c = e / kStepK;
            } else {
                c = e % kTile;
                kk = e / kTile;
            }
            T v = T(0);
            if (n0 + c < p.n && k0 + kk < p.k) {
                const long long idx = (n0 + c) * p.b_sn + static_cast<long long>(k0 + kk) * p.b_sk;
                v = kInt ? static_cast<T>(load_as_int(b, p.b_dtype, idx)) : static_cast<T>(load_as_f32(b, p.b_dtype, idx));
            }
            sb[kk][c] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kStepK; ++kk) {
            T av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                av[i] = sa[kk][ty * 4 + i];
                bv[i] = sb[kk][tx * 4 + i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = kInt ? acc[i][j] + av[i] * bv[j] : static_cast<T>(fmaf(av[i], bv[j], acc[i][j]));
                }
            }
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const long long mi = m0 + ty * 4 + i;
        if (mi >= p.m) {
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const long long ni = n0 + tx * 4 + j;
            if (ni < p.n) {
                if (kInt) {
                    epilogue_int(epi, static_cast<int>(acc[i][j]), mi, ni);
                } else {
                    epilogue_scalar(epi, static_cast<float>(acc[i][j]), mi, ni);
                }
            }
        }
    }
}

}  // namespace

static cudaError_t launch_general(const LinearProblem &pr, int sm_count, cudaStream_t stream, bool integer);

cudaError_t launch_simt(const LinearProblem &pr, int sm_count, cudaStream_t stream)
{
    return launch_general(pr, sm_count, stream, false);
}

cudaError_t launch_int_gemm(const LinearProblem &pr, int sm_count, cudaStream_t stream)
{
    return launch_general(pr, sm_count, stream, true);
}

static cudaError_t launch_general(const LinearProblem &pr, int sm_count, cudaStream_t stream, bool integer)
{
    SimtParams p;
    p.a = pr.a;
    p.b = pr.b;
    p.a_sm = pr.a_sm;
    p.a_sk = pr.a_sk;
    p.b_sk = pr.b_sk;
    p.b_sn = pr.b_sn;
    p.a_dtype = pr.a_dtype;
    p.b_dtype = pr.b_dtype;
    p.m = static_cast<int>(pr.m);
    p.n = static_cast<int>(pr.n);
    p.k = static_cast<int>(pr.k);
    p.epi = pr.epi;
    p.batch = pr.batch;
    const long long nbatch = pr.batch_count;
    // grid.z is limited to 65535 entries; larger batch counts are issued in slices
    for (long long z0 = 0; z0 < nbatch; z0 += 65535) {
        // batch slices beyond the first are not expected in practice (5-D tensors of this size do not fit memory),
        // so a slice start is folded into the outermost batch stride only when it divides evenly
        if (z0 != 0) {
            return cudaErrorInvalidValue;
        }
        // Few tiles: the small kernel (times of a call in a chain, us, small / large tiles: 113 x 198 x 246 18.5 / 60.6, 21 x 512 x 23
        // 7.4 / 24.2, both fp32 with SiLU).  From two waves of 64 x 64 tiles on, their four times lower operand traffic counts.
        const long long large_tiles = ((pr.n + kTile - 1) / kTile) * ((pr.m + kTile - 1) / kTile) * nbatch;
        const long long small_rows = (pr.m + kSmallTile - 1) / kSmallTile;
        if (!integer && large_tiles < 2 * sm_count && small_rows <= 65535) {
            const dim3 small_grid(static_cast<unsigned>((pr.n + kSmallTile - 1) / kSmallTile), static_cast<unsigned>(small_rows),
                                  static_cast<unsigned>(nbatch));
            cudaError_t e = launch_chained(simt_small_kernel, small_grid, dim3(256), 0, stream, 1, p);
            if (e != cudaSuccess) {
                return e;
            }
            continue;
        }
        dim3 grid(static_cast<unsigned>((pr.n + kTile - 1) / kTile), static_cast<unsigned>((pr.m + kTile - 1) / kTile),
                  static_cast<unsigned>(nbatch < 65535 ? nbatch : 65535));
        if (grid.y > 65535) {
            return cudaErrorInvalidValue;
        }
        if (integer) {
            simt_linear_kernel<int><<<grid, 256, 0, stream>>>(p);
        } else {
            simt_linear_kernel<float><<<grid, 256, 0, stream>>>(p);
        }
    }
    return cudaGetLastError();
}

}  // namespace kb
