// sdf.cu — compute_sdf and the slot packing on the GPU (wx_grid_build_gpu).
//
// Same result, word for word, as the host sweep in topology.cpp, which
// restates VDB345::compute_sdf (src/vdb/vdb345.rs:290-670) as three
// independent per-level chamfer sweeps. A sweep visits the containers (nodes of
// one level) in DFS order, forward and then backward; each tile slot becomes
// min(own, neighbour + 1) over its 13 "earlier" (forward) or "later"
// (backward) neighbours in slot order, updated in place; child slots, active
// leaf voxels and missing neighbours read as 0.
//
// Both sweeps are shortest paths with unit steps, so they can be computed
// breadth first instead of in the sweep's order:
//   * Forward. When a cell is visited, a neighbour cell holds its final
//     forward value if its container comes no later in DFS order, else its
//     initial value (0 or infinity). So with Z the cells that start at 0 and
//     F(k) the cells whose forward value is at most k: F(0) = Z, and a cell is
//     in F(k) if it is in F(k-1), or one of its 13 earlier neighbours is in
//     F(k-1) (container no later than its own) or in Z (container later), or
//     belongs to a missing container.
//   * Backward. A neighbour holds its final value if its container comes no
//     earlier, else its forward value. With W(k) the cells whose final value is
//     at most k: W(0) = Z, W(k) = F(k), W(k-1) and the cells one of whose 13
//     later neighbours is in W(k-1) (container no earlier), in F(k-1)
//     (container earlier) or missing.
// The final distance of a cell is the first k with the cell in W(k). No order
// is left but that of k: every container can be advanced from k-1 to k at the
// same time, on bit masks, 64 cells an instruction.
//
// k_sdf_levels advances all nodes of all three levels by one k between two
// barriers of a cooperative grid, in F and W masks that are double-buffered by
// the parity of k, and writes a cell's distance straight into the grid's pools
// when it enters W. A container is advanced only when it or one of its
// 26 neighbours changed in the previous step (act = the last such step). The
// barrier's wait is bounded; on the bound an error flag ends the kernel.
// 2000-sphere grid (476,014 leaves, ten or so steps a level): 2.14 ms, where the sweeps in the
// sweep's order (one CTA a container, a ready queue, 50 barriers a leaf) took 27.4 ms, bound by
// the chain of containers that wait for one another; the whole build and a 720p frame 34.5 -> 3.85 ms.
// Distances are small: a cell at distance k lies in a solid cube of containers
// of side k / D - 1 (every axis-aligned step toward the origin corner is
// allowed), so k < 2000 for any grid the pools can hold.
// The containers' neighbour tables come from the tree itself: a neighbour's
// origin is looked up through the root-key table and the child-index tables.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "wx_kernels.h"

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;   // no node
constexpr uint32_t kChild = 0x80000000u;

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ---------------------------------------------------------------------------
// Structure: child-index tables, derived origins, initial distances.
// ---------------------------------------------------------------------------

// cidx[node * S + s] = DFS index of the child in slot s (first[node] + rank of
// the child bit among the node's child bits), or kNone. pre[node * W + w] is
// the number of child bits in words 0..w-1 of the node (host prefix).
__global__ void k_child_table(const uint64_t *__restrict__ kid, const uint32_t *__restrict__ pre,
                              const uint32_t *__restrict__ first, uint64_t nslots, int slots_log2,
                              uint32_t *__restrict__ cidx) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslots) return;
    const uint64_t node = i >> slots_log2;
    const uint64_t w = i >> 6;
    const uint64_t word = kid[w];
    const uint32_t bit = (uint32_t)(i & 63);
    if (!((word >> bit) & 1u)) {
        cidx[i] = kNone;
        return;
    }
    const uint32_t below = __popcll(word & ((1ull << bit) - 1ull));
    cidx[i] = first[node] + pre[w] + below;
}

// Origins of the children: org_child[cidx] = org_parent + coords(s) * child_span.
__global__ void k_child_origins(const uint32_t *__restrict__ cidx, const int4 *__restrict__ org, uint64_t nslots,
                                int log2d, int child_span_log2, int4 *__restrict__ org_child) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslots) return;
    const uint32_t c = cidx[i];
    if (c == kNone) return;
    const uint64_t node = i >> (3 * log2d);
    const uint32_t s = (uint32_t)(i & ((1u << (3 * log2d)) - 1u)), dm = (1u << log2d) - 1u;
    const int4 o = org[node];
    org_child[c] = make_int4(o.x + (int)((s >> (2 * log2d)) << child_span_log2),
                             o.y + (int)(((s >> log2d) & dm) << child_span_log2),
                             o.z + (int)((s & dm) << child_span_log2), 0);
}

// *count += the clear bits of the masks (the cells without a distance yet).
__global__ void k_count_clear(const uint64_t *__restrict__ w, uint64_t n, unsigned long long *count) {
    unsigned long long c = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += 64u - __popcll(w[i]);
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(~0u, c, o);
    if ((threadIdx.x & 31u) == 0u) atomicAdd(count, c);
}

// ---------------------------------------------------------------------------
// Neighbour tables.
// ---------------------------------------------------------------------------

// N5 index of the node whose origin is exactly (x, y, z), or kNone. Origins are
// multiples of 4096 (checked on the host), so the root table applies.
__device__ __forceinline__ uint32_t find_n5(const wxk::SdfTree &t, int64_t x, int64_t y, int64_t z) {
    if (x < INT32_MIN || x > INT32_MAX || y < INT32_MIN || y > INT32_MAX || z < INT32_MIN || z > INT32_MAX)
        return kNone;
    const int xi = (int)x, yi = (int)y, zi = (int)z;
    if ((xi & 4095) || (yi & 4095) || (zi & 4095)) return kNone;
    const int4 h0 = t.root[0], h1 = t.root[1];
    if (h1.w) {
        const uint32_t ux = (uint32_t)((xi >> 12) - h0.x), uy = (uint32_t)((yi >> 12) - h0.y),
                       uz = (uint32_t)((zi >> 12) - h0.z);
        if (ux >= (uint32_t)h0.w || uy >= (uint32_t)h1.x || uz >= (uint32_t)h1.y) return kNone;
        const uint32_t *tab = reinterpret_cast<const uint32_t *>(t.root + 2 + t.n5);
        const uint32_t e = tab[(uz * (uint32_t)h1.x + uy) * (uint32_t)h0.w + ux];
        return e ? e - 1u : kNone;
    }
    for (uint32_t k = 0; k < t.n5; k++) {
        const int4 o = t.root[2 + k];
        if (o.x == xi && o.y == yi && o.z == zi) return k;
    }
    return kNone;
}

// nb[c * 27 + k] = index of the container at origin + (dx, dy, dz) * span,
// k = (dx+1)*9 + (dy+1)*3 + (dz+1); k = 13 is c itself.
template <int L>
__global__ void k_sdf_neighbours(const int4 *__restrict__ org, uint32_t nc, wxk::SdfTree t, uint32_t *__restrict__ nb) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)nc * 27) return;
    const uint32_t c = (uint32_t)(i / 27), k = (uint32_t)(i % 27);
    if (k == 13) {
        nb[i] = c;
        return;
    }
    constexpr int span_log2 = L == 5 ? 12 : L == 4 ? 7 : 3;
    const int4 o = org[c];
    const int64_t x = (int64_t)o.x + ((int)(k / 9) - 1) * (int64_t(1) << span_log2);
    const int64_t y = (int64_t)o.y + ((int)((k / 3) % 3) - 1) * (int64_t(1) << span_log2);
    const int64_t z = (int64_t)o.z + ((int)(k % 3) - 1) * (int64_t(1) << span_log2);
    uint32_t n = find_n5(t, x & ~int64_t(4095), y & ~int64_t(4095), z & ~int64_t(4095));
    if (L <= 4 && n != kNone) {
        const uint32_t s5 = ((uint32_t)((x >> 7) & 31) << 10) | ((uint32_t)((y >> 7) & 31) << 5) | (uint32_t)((z >> 7) & 31);
        n = t.c5[((size_t)n << 15) | s5];
    }
    if (L == 3 && n != kNone) {
        const uint32_t s4 = ((uint32_t)((x >> 3) & 15) << 8) | ((uint32_t)((y >> 3) & 15) << 4) | (uint32_t)((z >> 3) & 15);
        n = t.c4[((size_t)n << 12) | s4];
    }
    nb[i] = n;
}

// ---------------------------------------------------------------------------
// The levels of k.
// ---------------------------------------------------------------------------
using wxk::SdfWork;

constexpr uint64_t kZ0 = 0x0101010101010101ull;  // bit z = 0 of every row of an x slice (8 rows of 8 bits)
constexpr uint64_t kNotZ7 = 0x7F7F7F7F7F7F7F7Full;

// The cells of an x slice of a leaf within one step of the cells of the slice around it: q[3 * (dy + 1) + dz + 1]
// is the slice of the same x in the container at (dy, dz). *zd: one step in z only; *below and *above: their rows
// y - 1 and y + 1.
__device__ __forceinline__ uint64_t dilate(const uint64_t q[9], uint64_t *below, uint64_t *above) {
    const uint64_t g = q[4] | ((q[4] & kNotZ7) << 1) | ((q[4] >> 1) & kNotZ7) | ((q[3] >> 7) & kZ0) | ((q[5] & kZ0) << 7);
    const uint32_t lo = (uint32_t)(q[1] >> 56), hi = (uint32_t)q[7] & 255u;  // row -1, row 8
    const uint32_t glo = (lo | (lo << 1) | (lo >> 1) | (uint32_t)(q[0] >> 63) | ((uint32_t)(q[2] >> 49) & 128u)) & 255u;
    const uint32_t ghi = (hi | (hi << 1) | (hi >> 1) | ((uint32_t)(q[6] >> 7) & 1u) | (((uint32_t)q[8] & 1u) << 7)) & 255u;
    *below = (g << 8) | glo;
    *above = (g >> 8) | ((uint64_t)ghi << 56);
    return g;
}

// Three leaves of a warp, ten lanes each: lane j holds the slice x = j - 1 (-1 and 8 lie in the neighbours).
// Returns the lane's count of cells that got their distance.
__device__ __forceinline__ uint32_t leaf_step(const SdfWork &S, uint32_t k, uint32_t task, uint32_t lane) {
    const uint32_t grp = lane / 10u, j = lane - grp * 10u, c = task * 3u + grp;
    const wxk::SdfLevel &V = S.lv[2];
    const bool run = grp < 3u && c < V.n && V.act[c] + 1u >= k;
    if (!__any_sync(~0u, run)) return 0;
    const uint64_t *F = V.f[(k - 1u) & 1u], *W = V.w[(k - 1u) & 1u];
    const uint32_t dx = j == 0u ? 0u : j == 9u ? 2u : 1u, sx = (j - 1u) & 7u;
    uint64_t f[9], b[9];
#pragma unroll
    for (int q = 0; q < 9; q++) {
        const uint32_t n = run ? V.nb[(size_t)c * 27u + dx * 9u + q] : kNone;
        f[q] = b[q] = ~0ull;
        if (n == kNone) continue;
        const size_t i = (size_t)n * 8u + sx;
        if (n < c) f[q] = b[q] = F[i];
        else if (n > c) {
            f[q] = V.z[i];
            b[q] = W[i];
        } else {
            f[q] = F[i];
            b[q] = W[i];
        }
    }
    uint64_t dn, up;
    uint64_t g = dilate(f, &dn, &up);
    uint64_t nf = f[4] | dn | ((f[4] & kNotZ7) << 1) | ((f[3] >> 7) & kZ0);
    nf |= __shfl_up_sync(~0u, g | dn | up, 1);
    g = dilate(b, &dn, &up);
    uint64_t nw = b[4] | nf | up | ((b[4] >> 1) & kNotZ7) | ((b[5] & kZ0) << 7);
    nw |= __shfl_down_sync(~0u, g | dn | up, 1);
    const bool own = run && dx == 1u;
    const size_t i = (size_t)c * 8u + sx;
    if (own) {
        V.f[k & 1u][i] = nf;
        V.w[k & 1u][i] = nw;
    }
    const uint32_t ch = __ballot_sync(~0u, own && (nf != f[4] || nw != b[4]));
    if (run && (ch & (0x3FFu << (grp * 10u))))
        for (uint32_t q = j; q < 27u; q += 10u) {
            const uint32_t n = V.nb[(size_t)c * 27u + q];
            if (n != kNone) V.act[n] = k;
        }
    uint64_t add = own ? nw & ~b[4] : 0ull;
    const uint32_t count = __popcll(add);
    const uint64_t byte = k < 255u ? k : 255u;
    unsigned long long *out = reinterpret_cast<unsigned long long *>(S.leaf) + i * 8u;  // 64 bytes: rows y of 8 cells
    for (uint32_t y = 0; add; y++, add >>= 8) {
        const uint64_t row = add & 255u;
        if (!row) continue;
        // Bit z of the row into byte z, times the distance; a cell's byte is 0 until it is set here, once.
        const uint64_t t = (row * kZ0) & 0x8040201008040201ull;
        atomicOr(out + y, ((((t & kNotZ7) + kNotZ7) | t) >> 7 & kZ0) * byte);
        if (k >= 255u)
            for (uint32_t m = (uint32_t)row; m; m &= m - 1u) {
                const uint32_t p = atomicAdd(S.ctl + 3, 1u);
                if (p < S.ovf_cap) S.ovf[p] = make_uint2((uint32_t)(i * 64u) + y * 8u + __ffs(m) - 1u, k);
            }
    }
    return count;
}

template <int L>
struct RowOf;
template <>
struct RowOf<4> {
    using T = uint16_t;
};
template <>
struct RowOf<5> {
    using T = uint32_t;
};

// Row (x, y) of the cells around container c (x, y from -1 to D), as its cells see it: the sets kFwd ? F or Z : W or
// F by the order of the containers; *zm, *zp: the cells next to the row in z. Missing containers are all ones.
template <int L, bool kFwd>
__device__ __forceinline__ uint32_t row_of(const wxk::SdfLevel &V, uint32_t c, uint32_t par, int x, int y, uint32_t *zm,
                                           uint32_t *zp) {
    constexpr int D = 1 << L;
    using T = typename RowOf<L>::T;
    const int dx = x < 0 ? 0 : x >= D ? 2 : 1, dy = y < 0 ? 0 : y >= D ? 2 : 1;
    const size_t at = (size_t)((x & (D - 1)) * D + (y & (D - 1)));
    uint32_t r[3];
#pragma unroll
    for (int dz = 0; dz < 3; dz++) {
        const uint32_t n = V.nb[(size_t)c * 27u + dx * 9 + dy * 3 + dz];
        r[dz] = (T)~(T)0;
        if (n == kNone) continue;
        const uint64_t *src = kFwd ? (n <= c ? V.f[par] : V.z) : (n >= c ? V.w[par] : V.f[par]);
        r[dz] = reinterpret_cast<const T *>(src)[(size_t)n * (D * D) + at];
    }
    *zm = r[0] >> (D - 1);
    *zp = (r[2] & 1u) << (D - 1);
    return r[1];
}
template <int L, bool kFwd>
__device__ __forceinline__ uint32_t dilated_row(const wxk::SdfLevel &V, uint32_t c, uint32_t par, int x, int y) {
    uint32_t zm, zp;
    const uint32_t r = row_of<L, kFwd>(V, c, par, x, y, &zm, &zp);
    return r | (r << 1) | (r >> 1) | zm | zp;
}

// 32 rows (x, y) of an N4 or N5 node, one a lane.
template <int L>
__device__ __forceinline__ uint32_t node_step(const SdfWork &S, uint32_t k, uint32_t task, uint32_t lane) {
    constexpr int D = 1 << L;
    using T = typename RowOf<L>::T;
    const wxk::SdfLevel &V = S.lv[5 - L];
    const uint32_t c = task / (D * D / 32), r = (task % (D * D / 32)) * 32u + lane;
    if (V.act[c] + 1u < k) return 0;
    const uint32_t par = (k - 1u) & 1u;
    const int x = (int)(r >> L), y = (int)(r & (D - 1));
    uint32_t zm, zp;
    const uint32_t f = row_of<L, true>(V, c, par, x, y, &zm, &zp);
    uint32_t nf = f | (f << 1) | zm | dilated_row<L, true>(V, c, par, x, y - 1);
    for (int dy = -1; dy <= 1; dy++) nf |= dilated_row<L, true>(V, c, par, x - 1, y + dy);
    const uint32_t w = row_of<L, false>(V, c, par, x, y, &zm, &zp);
    uint32_t nw = w | nf | (w >> 1) | zp | dilated_row<L, false>(V, c, par, x, y + 1);
    for (int dy = -1; dy <= 1; dy++) nw |= dilated_row<L, false>(V, c, par, x + 1, y + dy);
    nf = (T)nf;
    nw = (T)nw;
    const size_t i = (size_t)c * (D * D) + r;
    reinterpret_cast<T *>(V.f[k & 1u])[i] = (T)nf;
    reinterpret_cast<T *>(V.w[k & 1u])[i] = (T)nw;
    if (__any_sync(~0u, nf != f || nw != w) && lane < 27u) {
        const uint32_t n = V.nb[(size_t)c * 27u + lane];
        if (n != kNone) V.act[n] = k;
    }
    const uint32_t add = nw & ~w, tile = add & ~(uint32_t)reinterpret_cast<const T *>(V.val)[i];  // active tiles stay 0
    for (uint32_t m = tile; m; m &= m - 1u) V.slot[i * D + (uint32_t)(__ffs(m) - 1)] = k;
    return __popc(add);
}

// Steps k0 to k1, or fewer when every cell has its distance. ctl: [0] arrivals at the barrier, [1] its release
// (2k + (1 when done)), [2] error flag, [3] overflow entries; left: cells without a distance, of all levels and of
// the leaves. A cooperative launch: the CTAs wait for one another.
__global__ void __launch_bounds__(256) k_sdf_levels(const __grid_constant__ SdfWork S, uint32_t k0, uint32_t k1,
                                                    uint32_t spin_limit) {
    __shared__ unsigned long long s_new[2];
    __shared__ uint32_t s_done;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t t5 = S.lv[0].n * 32u, t4 = t5 + S.lv[1].n * 8u, t3 = t4 + (S.lv[2].n + 2u) / 3u;
    for (uint32_t k = k0; k <= k1; k++) {
        if (threadIdx.x < 2u) s_new[threadIdx.x] = 0;
        __syncthreads();
        uint32_t upper = 0, leaf = 0;
        for (uint32_t t = blockIdx.x * 8u + (threadIdx.x >> 5); t < t3; t += gridDim.x * 8u) {
            if (t < t5) upper += node_step<5>(S, k, t, lane);
            else if (t < t4) upper += node_step<4>(S, k, t - t5, lane);
            else leaf += leaf_step(S, k, t - t4, lane);
        }
        upper = __reduce_add_sync(~0u, upper);
        leaf = __reduce_add_sync(~0u, leaf);
        if (lane == 0u && upper + leaf) {
            atomicAdd(&s_new[0], (unsigned long long)upper + leaf);
            atomicAdd(&s_new[1], (unsigned long long)leaf);
        }
        __syncthreads();
        if (threadIdx.x == 0u) {
            if (s_new[0]) atomicAdd(S.left, 0ull - s_new[0]);
            if (s_new[1]) atomicAdd(S.left + 1, 0ull - s_new[1]);
            __threadfence();
            uint32_t v;
            if (atomicAdd(S.ctl, 1u) == gridDim.x * (k - k0 + 1u) - 1u) {
                __threadfence();
                v = 2u * k + (atomicAdd(S.left, 0ull) == 0ull ? 1u : 0u);
                atomicExch(S.ctl + 1, v);
            } else {
                for (uint32_t polls = 1;; polls++) {
                    v = ld_acquire(S.ctl + 1);
                    if (v >= 2u * k) break;
                    if (polls >= spin_limit || ld_acquire(S.ctl + 2) != 0u) {  // every CTA then returns
                        atomicExch(S.ctl + 2, 1u);
                        v = 1u;
                        break;
                    }
                    __nanosleep(256);
                }
            }
            s_done = v & 1u;
            __threadfence();
        }
        __syncthreads();
        if (s_done) return;
    }
}

// ---------------------------------------------------------------------------
// Packing.
// ---------------------------------------------------------------------------

// Slot words of N5/N4: child -> flag | index, active tile -> 0; the other tiles get their distance from k_sdf_levels.
__global__ void k_pack_internal(const uint64_t *__restrict__ kid, const uint64_t *__restrict__ val,
                                const uint32_t *__restrict__ cidx, uint64_t nslots, uint32_t *__restrict__ slot) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslots) return;
    const bool k = (kid[i >> 6] >> (i & 63)) & 1u, v = (val[i >> 6] >> (i & 63)) & 1u;
    slot[i] = k && !v ? kChild | cidx[i] : 0u;
}

template <class K>
int resident_blocks(K kernel, int threads, size_t smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n > 0 ? n : 1;
}

unsigned grid_for(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

namespace wxk {

cudaError_t sdf_child_table(const uint64_t *kid, const uint32_t *pre, const uint32_t *first, uint64_t nodes,
                            int slots_log2, uint32_t *cidx, cudaStream_t st) {
    const uint64_t n = nodes << slots_log2;
    if (n) k_child_table<<<grid_for(n, 256), 256, 0, st>>>(kid, pre, first, n, slots_log2, cidx);
    return cudaGetLastError();
}

cudaError_t sdf_child_origins(const uint32_t *cidx, const int4 *org, uint64_t nodes, int log2d, int child_span_log2,
                              int4 *org_child, cudaStream_t st) {
    const uint64_t n = nodes << (3 * log2d);
    if (n) k_child_origins<<<grid_for(n, 256), 256, 0, st>>>(cidx, org, n, log2d, child_span_log2, org_child);
    return cudaGetLastError();
}

cudaError_t sdf_count_clear(const uint64_t *w, uint64_t words, unsigned long long *count, cudaStream_t st) {
    if (words) k_count_clear<<<std::min(grid_for(words, 256), 4096u), 256, 0, st>>>(w, words, count);
    return cudaGetLastError();
}

cudaError_t sdf_neighbours(int level, const int4 *org, uint32_t nc, const SdfTree &t, uint32_t *nb, cudaStream_t st) {
    const uint64_t n = (uint64_t)nc * 27;
    if (!n) return cudaSuccess;
    if (level == 5) k_sdf_neighbours<5><<<grid_for(n, 256), 256, 0, st>>>(org, nc, t, nb);
    else if (level == 4) k_sdf_neighbours<4><<<grid_for(n, 256), 256, 0, st>>>(org, nc, t, nb);
    else k_sdf_neighbours<3><<<grid_for(n, 256), 256, 0, st>>>(org, nc, t, nb);
    return cudaGetLastError();
}

cudaError_t sdf_levels(const SdfWork &w, uint32_t k0, uint32_t k1, int num_sms, uint32_t spin_limit, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(w.ctl, 0, 3 * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    const uint64_t tasks = (uint64_t)w.lv[0].n * 32 + (uint64_t)w.lv[1].n * 8 + (w.lv[2].n + 2u) / 3u;
    const uint64_t blocks = std::min<uint64_t>((uint64_t)resident_blocks(k_sdf_levels, 256, 0) * num_sms, (tasks + 7) / 8);
    SdfWork work = w;
    void *args[] = {&work, &k0, &k1, &spin_limit};
    return cudaLaunchCooperativeKernel((const void *)k_sdf_levels, dim3((unsigned)std::max<uint64_t>(blocks, 1)), dim3(256),
                                       args, 0, st);
}

cudaError_t sdf_pack_internal(const uint64_t *kid, const uint64_t *val, const uint32_t *cidx, uint64_t nslots,
                              uint32_t *slot, cudaStream_t st) {
    if (nslots) k_pack_internal<<<grid_for(nslots, 256), 256, 0, st>>>(kid, val, cidx, nslots, slot);
    return cudaGetLastError();
}

}  // namespace wxk
