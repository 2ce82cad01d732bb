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
// barriers of its running CTAs (sdf_steps.h). The first kSdfWindow steps, in which all but a
// few cells of a level set get their distance, advance every node, keep their W
// masks, and store nothing else: k_expand_* then turns the masks into pool words,
// each written once. Later steps alternate between two masks, advance a node only
// when it or one of its 26 neighbours changed in the step before (act = the last
// such step), and store a cell's distance when it enters W. The barrier's wait is
// bounded; on the bound an error flag ends the kernel.
// 2000-sphere grid (476,014 leaves, 14 steps, the leaves done after 7): 0.88 ms with k_expand_*, where the sweeps
// in the sweep's order (one CTA a container, a ready queue, 50 barriers a leaf) took 27.4 ms, bound
// by the chain of containers that wait for one another.
// Distances are small: a cell at distance k lies in a solid cube of containers
// of side k / D - 1 (every axis-aligned step toward the origin corner is
// allowed), so k < 2000 for any grid the pools can hold.
// The containers' neighbour tables come from the tree itself: a neighbour's
// origin is looked up through the root-key table and the child-index tables.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "wx_kernels.h"

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;   // no node
constexpr uint32_t kChild = 0x80000000u;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// ---------------------------------------------------------------------------
// Structure: child-index tables, derived origins, initial distances.
// ---------------------------------------------------------------------------

// pre[node * W + w] = the number of child bits in words 0..w-1 of the node; one warp a node of W (a multiple of 32) words.
__global__ void k_child_prefix(const uint64_t *__restrict__ kid, uint64_t nodes, uint32_t words, uint32_t *__restrict__ pre) {
    const uint64_t node = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if (node >= nodes) return;
    uint32_t sum = 0;
    for (uint32_t w = lane; w < words; w += 32u) {
        const uint32_t n = __popcll(kid[node * words + w]);
        uint32_t upto = n;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(~0u, upto, o);
            if ((int)lane >= o) upto += v;
        }
        pre[node * words + w] = sum + upto - n;
        sum += __shfl_sync(~0u, upto, 31);
    }
}

// cidx[node * S + s] = DFS index of the child in slot s (first[node] + rank of
// the child bit among the node's child bits), or kNone. pre: k_child_prefix.
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
    if ((threadIdx.x & 31u) == 0u && c) atomicAdd(count, c);
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
// k = (dx+1)*9 + (dy+1)*3 + (dz+1); k = 13 is c itself; nc where there is none.
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
    nb[i] = n == kNone ? nc : n;
}

// ---------------------------------------------------------------------------
// The levels of k.
// ---------------------------------------------------------------------------
using wxk::SdfLevel;
using wxk::SdfWork;

// Cells as 64-bit words of kRows rows of D cells (z); a node is D slices (x) of kSlice words (y).
template <int L>
struct Geo {
    static constexpr int D = 1 << L, kRows = 64 / D, kSlice = D / kRows, kNode = D * kSlice;
    static constexpr uint64_t kFirst = L == 3 ? 0x0101010101010101ull : L == 4 ? 0x0001000100010001ull : 0x0000000100000001ull;
    static constexpr uint64_t kNotLast = ~(kFirst << (D - 1));  // all but the last cell of each row
};

// Where the words of a set begin, for neighbours before (or at) and after the node in DFS order: the missing
// neighbour, n = V.n, comes after every node and has a word block of ones in z and w.
struct Sets {
    uint32_t before, after;
};

// The words around word yq of slice x (x from -1 to D) of node c: q[3 * (dy + 1) + dz + 1] holds the rows just before,
// at or after it in y (dy), of the node next in z (dz). No branches: all of the 9 index loads, then all 9 words are in
// flight together.
template <int L>
__device__ __forceinline__ void neighbours(const SdfLevel &V, uint32_t c, int x, int yq, uint32_t n[9]) {
    using G = Geo<L>;
    const uint32_t *nb = V.nb + (size_t)c * 27u + (x < 0 ? 0 : x >= G::D ? 18 : 9);
#pragma unroll
    for (int dy = 0; dy < 3; dy++) {
        const int y = yq + dy - 1;
#pragma unroll
        for (int dz = 0; dz < 3; dz++) n[3 * dy + dz] = nb[(y < 0 ? 0 : y >= G::kSlice ? 6 : 3) + dz];
    }
}
template <int L, bool kFwd>
__device__ __forceinline__ void around(const SdfLevel &V, Sets f, uint32_t c, int x, int yq, const uint32_t n[9], uint64_t q[9]) {
    using G = Geo<L>;
    const uint32_t sx = (uint32_t)(x & (G::D - 1)) * G::kSlice;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const uint32_t y = (uint32_t)(yq + i / 3 - 1) & (G::kSlice - 1), at = n[i] * G::kNode + sx + y;
        q[i] = V.sets[at + ((kFwd ? n[i] > c : n[i] >= c) ? f.after : f.before)];
    }
}

// The cells within one step of the words q in y and z; *below and *above: their rows y - 1 and y + 1.
template <int L>
__device__ __forceinline__ uint64_t dilate(const uint64_t q[9], uint64_t *below, uint64_t *above) {
    using G = Geo<L>;
    constexpr int R = G::D, T = 64 - R;  // bits of a row, shift of the last row
    const uint64_t g = q[4] | ((q[4] & G::kNotLast) << 1) | ((q[4] >> 1) & G::kNotLast) | ((q[3] >> (R - 1)) & G::kFirst) |
                       ((q[5] & G::kFirst) << (R - 1));
    constexpr uint64_t row = ~0ull >> T;
    const uint64_t lo = q[1] >> T, hi = q[7] & row;
    const uint64_t glo = lo | ((lo << 1) & row) | (lo >> 1) | (q[0] >> 63) | (((q[2] >> T) & 1u) << (R - 1));
    const uint64_t ghi = hi | ((hi << 1) & row) | (hi >> 1) | ((q[6] >> (R - 1)) & 1u) | ((q[8] & 1u) << (R - 1));
    *below = (g << R) | glo;
    *above = (g >> R) | (ghi << T);
    return g;
}
// Every cell of the rows y - 1, y, y + 1 within a step: what a word receives from the word beside it in x.
template <int L>
__device__ __forceinline__ uint64_t dilate_all(const uint64_t q[9]) {
    uint64_t dn, up;
    const uint64_t g = dilate<L>(q, &dn, &up);
    return g | dn | up;
}
// What a word receives from its own slice: forward the rows before it and the cell before each cell, backward those after.
template <int L, bool kFwd>
__device__ __forceinline__ uint64_t own_slice(const uint64_t q[9], uint64_t dn, uint64_t up) {
    using G = Geo<L>;
    return kFwd ? q[4] | dn | ((q[4] & G::kNotLast) << 1) | ((q[3] >> (G::D - 1)) & G::kFirst)
                : q[4] | up | ((q[4] >> 1) & G::kNotLast) | ((q[5] & G::kFirst) << (G::D - 1));
}

struct Step {
    Sets f, b;            // where the forward and the backward pass read
    uint32_t out_f, out_w;  // where F(k) and W(k) are written
};
__device__ __forceinline__ uint32_t f_set(uint32_t k) { return k == 0u ? 0u : wxk::kSdfWindow + 1u + (k & 1u); }
__device__ __forceinline__ uint32_t w_set(uint32_t k) { return k <= wxk::kSdfWindow ? k : wxk::kSdfWindow - (k & 1u); }
__device__ __forceinline__ Step step_of(const SdfLevel &V, uint32_t k) {
    const uint32_t f = f_set(k - 1u) * V.stride, w = w_set(k - 1u) * V.stride;
    return Step{{f, 0u}, {f, w}, f_set(k) * V.stride, w_set(k) * V.stride};
}

// Three leaves of a warp, ten lanes each: lane j holds the slice x = j - 1 (-1 and 8 lie in the neighbours), one word.
// Leaves that nothing changed around are left alone. Returns the lane's count of cells that got their distance.
__device__ __forceinline__ uint32_t leaf_step(const SdfWork &S, uint32_t k, uint32_t first, uint32_t active, uint32_t lane) {
    const uint32_t grp = lane / 10u, j = lane - grp * 10u;
    const SdfLevel &V = S.lv[2];
    const bool run = grp < 3u && ((active >> grp) & 1u);
    const uint32_t c = run ? first + grp : first;  // lanes without work read with the first leaf
    const Step st = step_of(V, k);
    uint64_t f[9], b[9], dn, up;
    uint32_t n[9];
    neighbours<3>(V, c, (int)j - 1, 0, n);
    around<3, true>(V, st.f, c, (int)j - 1, 0, n, f);
    around<3, false>(V, st.b, c, (int)j - 1, 0, n, b);
    uint64_t g = dilate<3>(f, &dn, &up);
    uint64_t nf = own_slice<3, true>(f, dn, up);
    nf |= __shfl_up_sync(~0u, g | dn | up, 1);
    g = dilate<3>(b, &dn, &up);
    uint64_t nw = nf | own_slice<3, false>(b, dn, up);
    nw |= __shfl_down_sync(~0u, g | dn | up, 1);
    const bool own = run && j >= 1u && j <= 8u;
    const uint32_t i = c * 8u + ((j - 1u) & 7u);
    if (own) {
        V.sets[st.out_f + i] = nf;
        V.sets[st.out_w + i] = nw;
    }
    const uint32_t ch = __ballot_sync(~0u, own && (nf != f[4] || nw != b[4]));
    uint64_t add = own ? nw & ~b[4] : 0ull;
    const uint32_t count = __popcll(add);
    if (k <= wxk::kSdfWindow) return count;
    if (run && (ch & (0x3FFu << (grp * 10u))))
        for (uint32_t q = j; q < 27u; q += 10u) V.act[V.nb[(size_t)c * 27u + q]] = k;
    const uint64_t byte = k < 255u ? k : 255u;
    unsigned long long *out = reinterpret_cast<unsigned long long *>(S.leaf) + (size_t)i * 8u;  // 64 bytes: rows y of 8 cells
    for (uint32_t y = 0; add; y++, add >>= 8) {
        const uint64_t row = add & 255u;
        if (!row) continue;
        // Bit z of the row into byte z, times the distance; a cell's byte is 0 until it is set here, once.
        constexpr uint64_t kOnes = Geo<3>::kFirst, kLow7 = Geo<3>::kNotLast;
        const uint64_t t = (row * kOnes) & 0x8040201008040201ull;
        atomicOr(out + y, ((((t & kLow7) + kLow7) | t) >> 7 & kOnes) * byte);
        if (k >= 255u)
            for (uint32_t m = (uint32_t)row; m; m &= m - 1u) {
                const uint32_t p = atomicAdd(&S.ctl->n_ovf, 1u);
                if (p < S.ovf_cap) S.ovf[p] = make_uint2(i * 64u + y * 8u + (uint32_t)__ffs(m) - 1u, k);
            }
    }
    return count;
}

// 32 words of an N4 or N5 node, one a lane.
template <int L>
__device__ __forceinline__ uint32_t node_step(const SdfWork &S, uint32_t k, uint32_t task, uint32_t lane) {
    using G = Geo<L>;
    const SdfLevel &V = S.lv[5 - L];
    const uint32_t c = task / (G::kNode / 32), r = (task % (G::kNode / 32)) * 32u + lane;
    // Other CTAs set act while it is read: the vote makes the lanes agree, as the votes below need.
    if (k > wxk::kSdfWindow + 1u && !__any_sync(~0u, V.act[c] + 1u >= k)) return 0;
    const Step st = step_of(V, k);
    const int x = (int)(r / G::kSlice), yq = (int)(r % G::kSlice);
    uint32_t n[9];
    uint64_t q[9], dn, up;
    neighbours<L>(V, c, x, yq, n);
    around<L, true>(V, st.f, c, x, yq, n, q);
    dilate<L>(q, &dn, &up);
    const uint64_t f = q[4];
    uint64_t nf = own_slice<L, true>(q, dn, up);
    around<L, false>(V, st.b, c, x, yq, n, q);
    dilate<L>(q, &dn, &up);
    const uint64_t w = q[4];
    uint64_t nw = own_slice<L, false>(q, dn, up);
    neighbours<L>(V, c, x - 1, yq, n);
    around<L, true>(V, st.f, c, x - 1, yq, n, q);
    nf |= dilate_all<L>(q);
    neighbours<L>(V, c, x + 1, yq, n);
    around<L, false>(V, st.b, c, x + 1, yq, n, q);
    nw |= nf | dilate_all<L>(q);
    const uint32_t i = c * G::kNode + r;
    V.sets[st.out_f + i] = nf;
    V.sets[st.out_w + i] = nw;
    const uint64_t add = nw & ~w;
    if (k <= wxk::kSdfWindow) return __popcll(add);
    if (__any_sync(~0u, nf != f || nw != w) && lane < 27u) V.act[V.nb[(size_t)c * 27u + lane]] = k;
    for (uint64_t m = add & ~V.val[i]; m; m &= m - 1u) V.slot[(size_t)i * 64u + (uint32_t)(__ffsll(m) - 1)] = k;  // active tiles stay 0
    return __popcll(add);
}

// The step control's memory operations (sdf_steps.h).
struct StepsMem {
    template <class T>
    __device__ __forceinline__ T add(T *p, T v) const { return atomicAdd(p, v); }
    __device__ __forceinline__ uint32_t count(uint32_t *p, uint32_t n) const { return atomicInc(p, n - 1u); }
    __device__ __forceinline__ uint32_t load(const uint32_t *p) const { return ld_relaxed(p); }
    __device__ __forceinline__ unsigned long long load(const unsigned long long *p) const {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ void store(uint32_t *p, uint32_t v) const { atomicExch(p, v); }
    __device__ __forceinline__ void fence() const { __threadfence(); }
    // Polls are relaxed: an acquire would empty the SM's L1 under the CTAs still at work (the fence after them acquires).
    __device__ __forceinline__ void pause() const { __nanosleep(256); }
};

// Steps k0 to k1, or fewer when every cell has its distance. A level takes no part once none is left in it. The CTAs
// that run share each step among them (sdf_steps.h).
constexpr uint32_t kLeafChunk = 8;  // groups of three leaves a warp takes at a time, looked over with one load
// Bound by the latency of its gathers. 2000-sphere grid, 14 steps: 0.77 ms, and k_expand_* another 0.11 ms; as
// one kernel that stored every distance by an atomic and marked the neighbours of every change from the first step on,
// 2.1 ms (of a full step's 670 us the marks took 330 and the atomics 190). 6 CTAs an SM at 40 registers: 1.96 ms for
// the whole build; 2.04 at 4 CTAs (64 registers), 2.14 at 5, 2.47 at 8 (spills).
__global__ void __launch_bounds__(256, 6) k_sdf_levels(const __grid_constant__ SdfWork S, uint32_t k0, uint32_t k1,
                                                    uint32_t spin_limit) {
    __shared__ uint32_t s_new[3], s_word, s_ticket;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n5 = S.lv[0].n * (Geo<5>::kNode / 32), n4 = S.lv[1].n * (Geo<4>::kNode / 32), n3 = S.lv[2].n;
    if (threadIdx.x == 0u) s_word = wxk::steps_enter(StepsMem{}, S.ctl, gridDim.x, k0, k1, spin_limit, &s_ticket);
    __syncthreads();
    for (;;) {
        const uint32_t word = s_word, done = wxk::steps_done(word), k = wxk::steps_k(word) + 1u;
        if (done == wxk::kStepsAllDone || k > k1) return;
        const uint32_t warp = s_ticket * 8u + (threadIdx.x >> 5), warps = wxk::steps_ctas(word) * 8u;
        if (threadIdx.x < 3u) s_new[threadIdx.x] = 0;
        __syncthreads();
        uint32_t got[3] = {0, 0, 0};
        if (!(done & 1u))
            for (uint32_t t = warp; t < n5; t += warps) got[0] += node_step<5>(S, k, t, lane);
        if (!(done & 2u))
            for (uint32_t t = warp; t < n4; t += warps) got[1] += node_step<4>(S, k, t, lane);
        if (!(done & 4u))
            for (uint32_t first = warp * (3u * kLeafChunk); first < n3; first += warps * (3u * kLeafChunk)) {
                const uint32_t c = first + lane;
                uint32_t m = __ballot_sync(~0u, lane < 3u * kLeafChunk && c < n3 && (k <= wxk::kSdfWindow + 1u || S.lv[2].act[c] + 1u >= k));
                for (uint32_t g = first; m; m >>= 3, g += 3u)
                    if (m & 7u) got[2] += leaf_step(S, k, g, m & 7u, lane);
            }
#pragma unroll
        for (int l = 0; l < 3; l++) {
            const uint32_t n = __reduce_add_sync(~0u, got[l]);
            if (lane == 0u && n) atomicAdd(&s_new[l], n);
        }
        __syncthreads();
        if (threadIdx.x == 0u) {
            for (int l = 0; l < 3; l++)
                if (s_new[l]) atomicAdd(&S.ctl->left[l], 0ull - s_new[l]);
            s_word = wxk::steps_next(StepsMem{}, S.ctl, s_ticket, word, k1, spin_limit);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Packing.
// ---------------------------------------------------------------------------

// Leaf bytes after the first kSdfWindow steps, 64 cells a thread: a cell's distance is the number of kept masks
// W(0)..W(last) that lack it (added up bit-sliced); cells not in W(last) read 0 so far.
__global__ void __launch_bounds__(256) k_expand_leaves(const __grid_constant__ SdfWork S) {
    const SdfLevel &V = S.lv[2];
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= V.n * 8u) return;
    const uint32_t last = min(S.ctl->last[2], wxk::kSdfWindow);
    uint64_t c0 = 0, c1 = 0, c2 = 0, c3 = 0, w = 0;
    for (uint32_t k = 0; k <= last; k++) {
        w = V.sets[k * V.stride + i];
        uint64_t x = ~w, t = c0 & x;
        c0 ^= x;
        x = c1 & t;
        c1 ^= t;
        t = c2 & x;
        c2 ^= x;
        c3 ^= t;
    }
    c0 &= w;
    c1 &= w;
    c2 &= w;
    c3 &= w;
    uint4 *out = reinterpret_cast<uint4 *>(S.leaf) + (size_t)i * 4u;
    // Bit b of a nibble times (1 + 2^7 + 2^14 + 2^21) has its copy at bit 8b.
    auto four = [&](uint32_t at) {
        const uint32_t n0 = (uint32_t)(c0 >> at) & 15u, n1 = (uint32_t)(c1 >> at) & 15u, n2 = (uint32_t)(c2 >> at) & 15u,
                       n3 = (uint32_t)(c3 >> at) & 15u;
        return ((n0 * 0x00204081u) & 0x01010101u) | ((n1 * 0x00408102u) & 0x02020202u) |
               ((n2 * 0x00810204u) & 0x04040404u) | ((n3 * 0x01020408u) & 0x08080808u);
    };
#pragma unroll
    for (uint32_t r = 0; r < 4; r++) out[r] = make_uint4(four(16u * r), four(16u * r + 4u), four(16u * r + 8u), four(16u * r + 12u));
}

// Slot words of N5/N4, four a thread: active tile -> 0, child -> flag | index, else the distance found in the first
// kSdfWindow steps (0 so far for a later one).
__global__ void __launch_bounds__(256) k_expand_nodes(const __grid_constant__ SdfWork S, int level,
                                                      const uint4 *__restrict__ cidx) {
    const SdfLevel &V = S.lv[level];
    const uint64_t i = (uint64_t)blockIdx.x * 256u + threadIdx.x;  // grid: exactly a quarter of the level's slots
    const uint32_t word = (uint32_t)(i >> 4), bit = (uint32_t)(i & 15u) * 4u, last = min(S.ctl->last[level], wxk::kSdfWindow);
    const uint32_t kid = (uint32_t)(V.sets[word] >> bit) & 15u, val = (uint32_t)(V.val[word] >> bit) & 15u;
    uint32_t in = kid, d = 0;  // a byte a slot
    auto bytes = [](uint32_t nibble) { return (nibble * 0x00204081u) & 0x01010101u; };
    for (uint32_t k = 1; k <= last; k++) {
        d += bytes(in ^ 15u);
        in = (uint32_t)(V.sets[k * V.stride + word] >> bit) & 15u;
    }
    d &= bytes(in & ~val) * 255u;
    uint4 w = make_uint4(d & 255u, (d >> 8) & 255u, (d >> 16) & 255u, d >> 24);
    const uint32_t child = kid & ~val;
    if (child) {
        const uint4 c = cidx[i];
        if (child & 1u) w.x = kChild | c.x;
        if (child & 2u) w.y = kChild | c.y;
        if (child & 4u) w.z = kChild | c.z;
        if (child & 8u) w.w = kChild | c.w;
    }
    reinterpret_cast<uint4 *>(V.slot)[i] = w;
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

cudaError_t sdf_child_table(const uint64_t *kid, uint32_t *pre, const uint32_t *first, uint64_t nodes,
                            int slots_log2, uint32_t *cidx, cudaStream_t st) {
    const uint64_t n = nodes << slots_log2;
    if (n) k_child_prefix<<<grid_for(nodes * 32, 256), 256, 0, st>>>(kid, nodes, 1u << (slots_log2 - 6), pre);
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
    if (words) k_count_clear<<<std::min(grid_for(words, 256), 1216u), 256, 0, st>>>(w, words, count);
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
    static_assert(kSdfMaxLevel < 4096u && offsetof(SdfCtl, error) == 16, "steps_word; the part cleared here");
    cudaError_t e = cudaMemsetAsync(w.ctl, 0, offsetof(SdfCtl, error), st);
    if (e != cudaSuccess) return e;
    const uint64_t tasks = (uint64_t)w.lv[0].n * (Geo<5>::kNode / 32) + (uint64_t)w.lv[1].n * (Geo<4>::kNode / 32) +
                           (w.lv[2].n + 3u * kLeafChunk - 1u) / (3u * kLeafChunk);
    // As many CTAs as fit the chip; fewer may run (sdf_steps.h).
    const uint64_t blocks = std::min({(uint64_t)resident_blocks(k_sdf_levels, 256, 0) * num_sms, (tasks + 7) / 8, (uint64_t)kStepsMaxCtas});
    k_sdf_levels<<<(unsigned)std::max<uint64_t>(blocks, 1), 256, 0, st>>>(w, k0, k1, spin_limit);
    return cudaGetLastError();
}

cudaError_t sdf_expand(const SdfWork &w, const uint32_t *cidx5, const uint32_t *cidx4, cudaStream_t st) {
    if (w.lv[0].n) k_expand_nodes<<<w.lv[0].n * (32768u / 1024u), 256, 0, st>>>(w, 0, reinterpret_cast<const uint4 *>(cidx5));
    if (w.lv[1].n) k_expand_nodes<<<w.lv[1].n * (4096u / 1024u), 256, 0, st>>>(w, 1, reinterpret_cast<const uint4 *>(cidx4));
    if (w.lv[2].n) k_expand_leaves<<<grid_for((uint64_t)w.lv[2].n * 8u, 256), 256, 0, st>>>(w);
    return cudaGetLastError();
}

}  // namespace wxk
