// pack.cu — the flattened view's atlases into the grid's pools (wx_grid_upload).
//
// The atlases are 3-D textures with x fastest (src/render/wgpu_context.rs:119-151); a node is a block of
// D^3 texels, its slots run with z fastest. So a block is read in texture order, 32 to 128 contiguous bytes
// a row, turned round in shared memory, and written in slot order. Bound by the copy of the texels from
// host memory (104 MB of leaf texels for 200 spheres: 0.7 ms). Upload and first 720p frame of that grid:
// 1.48 ms; with the texels repacked by 16 host threads, 26.3 ms.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "wx_kernels.h"

namespace {

constexpr uint32_t kChild = 0x80000000u;

// First texel of node idx in the piece of nodes that starts at `first`: whole layers, or block rows of one.
__device__ __forceinline__ size_t block_texel(const wxk::ViewSlab &s, uint64_t idx, uint32_t log2d) {
    const uint64_t r = idx - s.first, zb = r / ((uint64_t)s.d * s.d), q = r - zb * s.d * s.d, yb = q / s.d, xb = q - yb * s.d;
    return ((size_t)(zb << log2d) * s.h + (yb << log2d)) * s.w + (xb << log2d);
}

// One CTA a node: slot word = 0 for a value, kChild | texel for a child, else the texel (a distance).
// flags: 1 a child index >= nchild, 2 a distance >= 2^31, 4 a distance >= 2^24.
template <int L>
__global__ void __launch_bounds__(256) k_pack_view_nodes(wxk::ViewSlab s, const uint32_t *__restrict__ kids,
                                                        const uint32_t *__restrict__ vals, uint32_t nchild,
                                                        uint32_t *__restrict__ slot, uint32_t *flags) {
    constexpr uint32_t D = 1u << L, N = D * D * D;
    extern __shared__ uint32_t buf[];  // N words, word i of slot i ^ (slot >> 2L): rows of x fall into different banks
    const uint64_t node = s.first + blockIdx.x;
    const uint32_t *t = s.texels + block_texel(s, node, L);
    for (uint32_t e = threadIdx.x; e < N; e += 256u) {
        const uint32_t x = e & (D - 1), y = (e >> L) & (D - 1), z = e >> (2 * L);
        const uint32_t o = (x << (2 * L)) | (y << L) | z;
        buf[o ^ x] = __ldg(t + ((size_t)z * s.h + y) * s.w + x);
    }
    __syncthreads();
    uint32_t bad = 0;
    for (uint32_t o = threadIdx.x; o < N; o += 256u) {
        const size_t w = (size_t)(node - s.first) * (N / 32) + (o >> 5);
        const uint32_t b = 1u << (o & 31u), v = buf[o ^ (o >> (2 * L))];
        uint32_t word = 0;
        if (!(vals[w] & b)) {
            if (kids[w] & b) {
                word = kChild | v;
                if (v >= nchild) bad |= 1u;
            } else {
                word = v;
                if (v >= kChild) bad |= 2u;
                else if (v >= (1u << 24)) bad |= 4u;
            }
        }
        slot[(size_t)node * N + o] = word;
    }
    if (bad) atomicOr(flags, bad);
}

// One CTA for eight leaves: voxel byte = 0 for a value, else min(texel, 255). Texels of 255 and more are counted in
// *n_ovf and, up to cap, listed in ovf.
__global__ void __launch_bounds__(256) k_pack_view_leaves(wxk::ViewSlab s, const uint32_t *__restrict__ vals,
                                                         uint8_t *__restrict__ leaf, uint2 *ovf, uint32_t cap,
                                                         unsigned long long *n_ovf) {
    __shared__ uint4 buf[8 * 512 / 16];
    const uint64_t leaf0 = s.first + (uint64_t)blockIdx.x * 8u, end = s.first + s.count;
    uint8_t *bytes = reinterpret_cast<uint8_t *>(buf);
    const uint32_t x = threadIdx.x & 7u, l = (threadIdx.x >> 3) & 7u, yb = threadIdx.x >> 6;  // rows y = yb, yb + 4
    const uint64_t n = leaf0 + l;
    if (n < end) {
        const uint32_t *t = s.texels + block_texel(s, n, 3) + x;
#pragma unroll 4
        for (uint32_t e = 0; e < 16; e++) {
            const uint32_t y = yb + (e & 1u) * 4u, z = e >> 1, o = (x << 6) | (y << 3) | z;
            const bool val = (__ldg(vals + (n - s.first) * 16u + (o >> 5)) >> (o & 31u)) & 1u;
            const uint32_t v = val ? 0u : __ldg(t + ((size_t)z * s.h + y) * s.w);
            bytes[l * 512u + o] = (uint8_t)min(v, 255u);
            if (v >= 255u) {
                const unsigned long long p = atomicAdd(n_ovf, 1ull);
                if (p < cap) ovf[p] = make_uint2((uint32_t)(n << 9) | o, v);
            }
        }
    }
    __syncthreads();
    if (leaf0 + threadIdx.x / 32u < end)
        reinterpret_cast<uint4 *>(leaf)[leaf0 * 32u + threadIdx.x] = buf[threadIdx.x];
}

}  // namespace

namespace wxk {

cudaError_t pack_view_nodes(int level, const ViewSlab &s, const uint32_t *kids, const uint32_t *vals, uint32_t nchild,
                            uint32_t *slot, uint32_t *flags, cudaStream_t st) {
    if (!s.count) return cudaSuccess;
    if (level == 5) {
        constexpr int bytes = 32768 * 4;
        const cudaError_t e = cudaFuncSetAttribute(k_pack_view_nodes<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        k_pack_view_nodes<5><<<(unsigned)s.count, 256, bytes, st>>>(s, kids, vals, nchild, slot, flags);
    } else {
        k_pack_view_nodes<4><<<(unsigned)s.count, 256, 4096 * 4, st>>>(s, kids, vals, nchild, slot, flags);
    }
    return cudaGetLastError();
}

cudaError_t pack_view_leaves(const ViewSlab &s, const uint32_t *vals, uint8_t *leaf, uint2 *ovf, uint32_t cap,
                             unsigned long long *n_ovf, cudaStream_t st) {
    if (s.count) k_pack_view_leaves<<<(unsigned)((s.count + 7) / 8), 256, 0, st>>>(s, vals, leaf, ovf, cap, n_ovf);
    return cudaGetLastError();
}

}  // namespace wxk
