// spatial.cuh -- Morton order of a set of FP64 positions, shared by the
// regular-force j set (regular.cu) and the potential (potential.cu).
#pragma once

#include "nb6_common.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>

namespace {

// ext[0..2] = min x, y, z and ext[3..5] = max (order-preserving uints).  The
// CTA reduces in shared memory before its six atomics: with one set per warp
// the kernel spent its time on atomics to the same six words (42 us for 1M
// bodies against 24 MB, 4 us, of reading).
constexpr int EXT_NT = 512;
__global__ void __launch_bounds__(EXT_NT) spatial_extent(int n, const double *__restrict__ x,
                                                        unsigned *__restrict__ ext) {
    __shared__ unsigned smn[EXT_NT / 32][3], smx[EXT_NT / 32][3];
    unsigned mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    for (int j = blockIdx.x * EXT_NT + threadIdx.x; j < n; j += gridDim.x * EXT_NT)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned o = f2ord((float)x[3 * (size_t)j + k]);
            mn[k] = min(mn[k], o);
            mx[k] = max(mx[k], o);
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = __reduce_min_sync(0xffffffffu, mn[k]);
        mx[k] = __reduce_max_sync(0xffffffffu, mx[k]);
        if (lane == 0) {
            smn[warp][k] = mn[k];
            smx[warp][k] = mx[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        unsigned a = smn[0][k], b = smx[0][k];
        for (int w = 1; w < EXT_NT / 32; ++w) {
            a = min(a, smn[w][k]);
            b = max(b, smx[w][k]);
        }
        atomicMin(&ext[k], a);
        atomicMax(&ext[3 + k], b);
    }
}

// The grid of a Morton key: 1024 cells per axis over the extent.
struct KeyGrid {
    float lo[3], sc[3];
};
NB6_DEV KeyGrid key_grid(const unsigned *__restrict__ ext) {
    KeyGrid g;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g.lo[k] = ord2f(ext[k]);
        const float w = ord2f(ext[3 + k]) - g.lo[k];
        g.sc[k] = w > 0.f ? 1023.99f / w : 0.f;
    }
    return g;
}
NB6_DEV unsigned key_of(const KeyGrid &g, const double *__restrict__ x) {
    unsigned key = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float q = ((float)x[k] - g.lo[k]) * g.sc[k];
        const unsigned c = q <= 0.f ? 0u : (q >= 1023.f ? 1023u : (unsigned)q);
        key |= spread10(c) << k;
    }
    return key;
}

// 30-bit Morton key of each body.
__global__ void spatial_keys(int n, const double *__restrict__ x, const unsigned *__restrict__ ext,
                             unsigned *__restrict__ keys, int *__restrict__ vals) {
    const KeyGrid g = key_grid(ext);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        keys[j] = key_of(g, x + 3 * (size_t)j);
        vals[j] = j;
    }
}

// Buffers of one ordering; perm[s] = the body in slot s.
struct SpatialOrder {
    DevBuf<unsigned> keys_in, keys_out, ext;
    DevBuf<int> vals_in, perm;
    DevBuf<unsigned char> tmp;

    void release() {
        keys_in.release();
        keys_out.release();
        ext.release();
        vals_in.release();
        perm.release();
        tmp.release();
    }

    void build(int n, const double *x, cudaStream_t st) {
        keys_in.reserve(n);
        keys_out.reserve(n);
        vals_in.reserve(n);
        perm.reserve(n);
        ext.reserve(6);
        NB6_CUDA_CHECK(cudaMemsetAsync(ext.ptr, 0xff, 3 * sizeof(unsigned), st));
        NB6_CUDA_CHECK(cudaMemsetAsync(ext.ptr + 3, 0, 3 * sizeof(unsigned), st));
        const int eb = std::max(1, std::min((n + EXT_NT - 1) / EXT_NT, nb6_num_sms() * 2));
        spatial_extent<<<eb, EXT_NT, 0, st>>>(n, x, ext.ptr);
        const int blocks = std::max(1, std::min((n + 255) / 256, nb6_num_sms() * 8));
        spatial_keys<<<blocks, 256, 0, st>>>(n, x, ext.ptr, keys_in.ptr, vals_in.ptr);
        NB6_CUDA_CHECK(cudaGetLastError());
        size_t need = 0;
        NB6_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, need, keys_in.ptr, keys_out.ptr, vals_in.ptr,
                                                       perm.ptr, n, 0, 30, st));
        tmp.reserve(need + 16);
        NB6_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(tmp.ptr, need, keys_in.ptr, keys_out.ptr, vals_in.ptr,
                                                       perm.ptr, n, 0, 30, st));
    }
};

}  // namespace
