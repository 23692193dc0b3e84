// Load-time packers (see include/sal_pack.h): HBM-bound bit shuffling, one pass over the data.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sal_lutgemm.h"
#include "sal_pack.h"

namespace {

// One thread per (32-element word, row): reads the 32 x q sign bytes of its word (contiguous in
// memory) with 16-byte loads where alignment allows and writes q words.  Threads of a warp take
// consecutive rows, so the kernel-layout stores ([C/32][q][R]) are coalesced.
template <bool KERNEL_LAYOUT>
__global__ void __launch_bounds__(256) pack_planes_kernel(const int8_t *__restrict__ signs, uint32_t *__restrict__ out, int R,
                                                          int C, int q, int *bad) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (r >= R) return;
    const int8_t *src = signs + ((size_t)r * C + (size_t)j * 32) * q;
    uint32_t words[SAL_MAX_Q];
#pragma unroll
    for (int b = 0; b < SAL_MAX_Q; ++b) words[b] = 0u;
    int n_bad = 0;
    const int total = 32 * q;   // bytes of this word, element-major then plane
    const bool vec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) && (total % 16 == 0);
    int t = 0, b = 0;           // element and plane of the next byte
    const auto take = [&](int8_t v) {
        if (v == 1) {
#pragma unroll
            for (int bb = 0; bb < SAL_MAX_Q; ++bb)
                if (bb == b) words[bb] |= 1u << t;
        } else if (v != -1) {
            ++n_bad;
        }
        if (++b == q) {
            b = 0;
            ++t;
        }
    };
    if (vec) {
        for (int i = 0; i < total; i += 16) {
            const int4 chunk = *reinterpret_cast<const int4 *>(src + i);
            const int8_t *c8 = reinterpret_cast<const int8_t *>(&chunk);
#pragma unroll
            for (int k = 0; k < 16; ++k) take(c8[k]);
        }
    } else {
        for (int i = 0; i < total; ++i) take(src[i]);
    }
    const int words_per_row = C / 32;
    for (int bb = 0; bb < q; ++bb) {
        uint32_t w = 0;
#pragma unroll
        for (int k = 0; k < SAL_MAX_Q; ++k)
            if (k == bb) w = words[k];
        if (KERNEL_LAYOUT) out[((size_t)j * q + bb) * R + r] = w;
        else out[((size_t)r * words_per_row + j) * q + bb] = w;
    }
    if (n_bad && bad) atomicAdd(bad, n_bad);
}

// Bit transpose of a 32 x 32 tile held one row per lane: bit c of lane r becomes bit r of lane c.  Five exchanges of half of the
// bits with the lane 16, 8, 4, 2, 1 away.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t m = s == 16 ? 0x0000FFFFu : s == 8 ? 0x00FF00FFu : s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
        x = (lane & s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y & m) << s);
    }
    return x;
}

// Checkpoint planes [K][N/32][q] (packed along N) -> kernel planes [K/32][q][N] (packed along K), and with `alpha` the scales
// [R][G][q] -> [R][q][G] (fp32) by the CTAs behind the planes'.  Bound by memory: a CTA's 4 Q words per thread are all requested before
// the first is stored to shared memory.  A tile turned around by 32 ballots, one per column, took about five times the instructions.
// 11008 x 4096, 3 planes, with scales of 8 x 16 blocks (43 MB in all): 67.5 us for the planes' launch and the scales' operators, 19.6 us
// in this form, of which 15.7 us on the GPU (2.7 TB/s).
constexpr int TJ = 32;   // words of a row that a CTA stages
template <int Q>
__global__ void __launch_bounds__(256) repack_lat_kernel(const uint32_t *__restrict__ in, uint32_t *__restrict__ out, int K, int N, int jblocks,
                                                         const float *__restrict__ alpha, float *__restrict__ alpha_out, int G, int pairs) {
    constexpr int PITCH = TJ * Q + 1;
    __shared__ uint32_t tile[32 * PITCH];   // [32 rows][TJ words x Q planes]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int plane_ctas = (K / 32) * jblocks;
    if ((int)blockIdx.x >= plane_ctas) {
        const int i = ((int)blockIdx.x - plane_ctas) * 256 + tid;   // (row, group) of the scales
        if (i < pairs) {
            const int r = i / G, g = i % G;
            float v[Q];
#pragma unroll
            for (int b = 0; b < Q; ++b) v[b] = alpha[(size_t)i * Q + b];
#pragma unroll
            for (int b = 0; b < Q; ++b) alpha_out[((size_t)r * Q + b) * G + g] = v[b];
        }
        return;
    }
    const int kk = blockIdx.x / jblocks, j0 = (blockIdx.x % jblocks) * TJ;
    const int nw = N / 32, tj = min(TJ, nw - j0), row_words = tj * Q;
    const uint32_t *src = in + ((size_t)(32 * kk + warp) * nw + j0) * Q;
    uint32_t v[4][Q];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < Q; ++c) v[i][c] = 32 * c + lane < row_words ? src[(size_t)(8 * i) * nw * Q + 32 * c + lane] : 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < Q; ++c) tile[(warp + 8 * i) * PITCH + 32 * c + lane] = v[i][c];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4 * Q; ++i) {   // item = (word j, plane b) in the order they are stored
        const int item = warp + 8 * i, jl = item / Q, b = item % Q;
        if (item < row_words) out[((size_t)kk * Q + b) * N + (size_t)(j0 + jl) * 32 + lane] = transpose32(tile[lane * PITCH + item], lane);
    }
}

int repack(const void *in, void *out, int K, int N, int q, const void *alpha, void *alpha_out, int R, int G, void *stream) {
    if (!in || !out) return SAL_E_NULL;
    if (K < 32 || K % 32 || N < 32 || N % 32 || q < 1 || q > SAL_MAX_Q) return SAL_E_SHAPE;
    const int jblocks = (N / 32 + TJ - 1) / TJ, pairs = alpha ? R * G : 0;
    const long long ctas = (long long)(K / 32) * jblocks + (pairs + 255) / 256;
    if (jblocks > 65535 || ctas > 0x7fffffff) return SAL_E_SHAPE;
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t *ip = reinterpret_cast<const uint32_t *>(in);
    uint32_t *op = reinterpret_cast<uint32_t *>(out);
    const float *ap = reinterpret_cast<const float *>(alpha);
    float *aop = reinterpret_cast<float *>(alpha_out);
    switch (q) {
#define SAL_REPACK(Q) \
    case Q: repack_lat_kernel<Q><<<(unsigned)ctas, 256, 0, s>>>(ip, op, K, N, jblocks, ap, aop, G, pairs); break;
        SAL_REPACK(1) SAL_REPACK(2) SAL_REPACK(3) SAL_REPACK(4) SAL_REPACK(5) SAL_REPACK(6) SAL_REPACK(7) SAL_REPACK(8)
#undef SAL_REPACK
    }
    return cudaGetLastError() == cudaSuccess ? SAL_OK : SAL_E_LAUNCH;
}

}  // namespace

extern "C" {

int sal_pack_planes_i8(const void *signs, void *out, int R, int C, int q, int kernel_layout, int *bad, void *stream) {
    if (!signs || !out) return SAL_E_NULL;
    if (R < 1 || C < 32 || C % 32 || q < 1 || q > SAL_MAX_Q || C / 32 > 65535) return SAL_E_SHAPE;
    const dim3 grid((unsigned)((R + 255) / 256), (unsigned)(C / 32));
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (kernel_layout)
        pack_planes_kernel<true><<<grid, 256, 0, s>>>(reinterpret_cast<const int8_t *>(signs), reinterpret_cast<uint32_t *>(out), R,
                                                      C, q, bad);
    else
        pack_planes_kernel<false><<<grid, 256, 0, s>>>(reinterpret_cast<const int8_t *>(signs), reinterpret_cast<uint32_t *>(out), R,
                                                       C, q, bad);
    return cudaGetLastError() == cudaSuccess ? SAL_OK : SAL_E_LAUNCH;
}

int sal_repack_lat_to_kernel(const void *in, void *out, int K, int N, int q, void *stream) {
    return repack(in, out, K, N, q, nullptr, nullptr, 0, 0, stream);
}

int sal_convert_lat(const void *in, void *out, const void *alpha, void *alpha_out, int K, int N, int q, int R, int G, void *stream) {
    if (!alpha || !alpha_out) return SAL_E_NULL;
    if (R < 1 || G < 1 || (long long)R * G > 0x3fffffff) return SAL_E_SHAPE;
    return repack(in, out, K, N, q, alpha, alpha_out, R, G, stream);
}

}  // extern "C"
