// Host side of the kernel that multiplies fp32 operands as planes of fp16 (tc_planes.cuh).
#include "tc_planes.cuh"

#include <algorithm>

namespace kb {

using namespace tc;

bool planes_take(const EpiParams &epi)
{
    return epi.n_mirrors == 0 && epi.beta == 0.0f && epi.c != nullptr && epi.res_op == KUDNN_B200_RES_NONE &&
           // (a TMA store does not clip inside 16 bytes)
           epi.n % 4 == 0 && epi.c_dtype == KUDNN_B200_F32 && epi.c_sn == 1 && epi.c_sm % 4 == 0 && (reinterpret_cast<uintptr_t>(epi.c) & 15u) == 0 &&
           (epi.has_bias == 0 || (epi.bias_dtype == KUDNN_B200_F32 && epi.bias_sm == 0)) &&
           (epi.act == KUDNN_B200_ACT_NONE || epi.act == KUDNN_B200_ACT_RELU || epi.act == KUDNN_B200_ACT_SWISH ||
            epi.act == KUDNN_B200_ACT_GELU_TANH);
}

cudaError_t launch_planes(const PlanesOperand &a, const PlanesOperand &b, long long k_pad, const EpiParams &epi, long long m, long long n,
                          int *fallback, DeviceStatus *status, cudaStream_t stream, long long wait_limit_cycles, int skip_kblock)
{
    if (!tc_available() || !planes_take(epi)) {
        return cudaErrorNotSupported;
    }
    CUtensorMap ta, tb, tb64, to;
    cudaError_t e = tc_encode_kmajor(&ta, a.planes, KUDNN_B200_F16, m, 2 * k_pad, 2 * k_pad, 128);
    if (e == cudaSuccess) e = tc_encode_kmajor(&tb, b.planes, KUDNN_B200_F16, n, 2 * k_pad, 2 * k_pad, 128);
    if (e == cudaSuccess) e = tc_encode_kmajor(&tb64, b.planes, KUDNN_B200_F16, n, 2 * k_pad, 2 * k_pad, 64);
    // the output, written in boxes of 32 rows x 128 bytes
    if (e == cudaSuccess) e = tc_encode_kmajor(&to, epi.c, KUDNN_B200_F32, m, n, epi.c_sm, 32);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(tc_planes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) {
        return e;
    }
    PlanesParams p;
    p.epi = epi;
    p.m = static_cast<int>(m);
    p.n = static_cast<int>(n);
    p.num_kb = static_cast<int>(k_pad / 64);
    p.tiles_m = static_cast<int>((m + 255) / 256);
    p.tiles_n = static_cast<int>((n + 255) / 256);
    // the A rows of a raster group (4 bytes per element and row) should stay in L2, as for the other kernels
    p.group_m = static_cast<int>(std::clamp<long long>((64ll << 20) / (256 * 4 * k_pad), 2, kMaxGroupM));
    const int tiles = p.tiles_m * p.tiles_n, pairs = tc_pair_clusters(KUDNN_B200_F16, kPlanesSmem);
    if (pairs <= 0) {
        return cudaErrorNotSupported;
    }
    const int left = tiles % pairs;
    // tiles left over after the last full wave, if they would keep at most half of the pairs busy
    p.n_whole = 2 * left <= pairs ? tiles - left : tiles;
    p.num_items = p.n_whole + 2 * (tiles - p.n_whole);
    p.idesc = make_idesc(KUDNN_B200_F16, 256, 2 * kBM);
    p.idesc_half = make_idesc(KUDNN_B200_F16, 128, 2 * kBM);
    p.a = a;
    p.b = b;
    p.fallback = fallback;
    p.load_kb = skip_kblock >= 0 ? std::min(skip_kblock, p.num_kb) : p.num_kb;
    p.status = status;
    p.wait_limit = wait_limit_cycles > 0 ? wait_limit_cycles : kDefaultWaitLimitCycles;
    return launch_chained(tc_planes_kernel, dim3(static_cast<unsigned>(2 * std::min(p.num_items, pairs))), dim3(kWideThreads), kPlanesSmem, stream,
                          2u, ta, tb, tb64, to, p);
}

}  // namespace kb
