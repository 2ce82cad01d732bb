// api.cpp — the C ABI (include/woxel_gb300.h): contexts, grid upload/build,
// per-frame render, batched render (one-shot and CUDA-graph plans), tuning.
//
// Device layout of a grid (uploaded once, immutable afterwards):
//   root   2 x int4          header: {lo.x, lo.y, lo.z, dim.x}, {dim.y, dim.z, 0, use table}
//          n5 x int4         N5 origins (root keys) in DFS order
//          dim.x*dim.y*dim.z u32  dense root-key table over the box of N5 keys
//                            (origin >> 12) starting at lo: N5 index + 1, 0 = none
//   top    64^3 u32          the slot5 words of the box [-4096, 4096)^3 by position, 32 where there is no N5: just
//                            before slot5, where the kernels address it (slot5 - kTopWords)
//   slot5  n5 x 32768 u32    per N4-sized slot: child flag|N4 index, or skip distance
//   slot4  n4 x  4096 u32    per N3-sized slot: child flag|N3 index, or skip distance
//   leaf   n3 x   512 u8     per voxel: 0 for an active voxel (a hit), else the skip
//                            distance, 255 meaning "at least 255: look it up in ovf"
//   ovf    n_ovf x (u32,u32) (voxel key = leaf << 9 | offset, exact distance), sorted; in a block of its
//                            own where the build learns n_ovf after the pools (GPU build, upload)
// A slot word folds the reference's three reads per level (child-mask word,
// value-mask word, atlas texel; raycast.comp.wgsl:422-429, :453-461,
// :483-489) into one load that decides hit / descend / skip. Leaf distances
// produced by compute_sdf are small (bounded by the extent of a cluster of
// leaves), so one byte per voxel keeps the leaf pool at a quarter of the
// reference's texel bytes while the overflow table keeps any u32 exact.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "launch_ring.h"
#include "wx_alloc.h"
#include "wx_common.h"
#include "wx_kernels.h"

namespace {
// Temporary buffer of wx_grid_upload, at most. 200 spheres (104 MB of leaf texels) and the first frame: 1.34 ms at 256 and at 64 MB,
// 1.44 at 32; on a new state 2.1, 2.0 and 2.0 ms; 1000 spheres (520 MB) 3.8, 3.9, 4.1 ms and 4.6 at 16.
constexpr size_t kUploadBuffer = (size_t)64 << 20;
// What the context's pool keeps of it at a synchronisation. Pools map 32 MB at a time: with nothing kept, an upload after a
// synchronisation takes 0.49 ms for two voxels, 0.62 ms for 40 spheres and 1.27 ms for 200, so 0.34, 0.48 and 1.18 ms.
constexpr size_t kUploadKeep = (size_t)32 << 20;
constexpr uint32_t kCounterSlots = 1u << 16;  // one work counter per in-flight launch (ring)
}

struct wx_ctx {
    int device = 0;
    int num_sms = 0;
    std::string err;
    wxk::Tuning tuning;
    uint32_t *counters = nullptr;       // kCounterSlots device counters
    uint32_t next_counter = 0;
    unsigned long long *check = nullptr;  // division self-check results
    cudaMemPool_t pool = nullptr;       // for wx_grid_upload's buffer; keeps at most kUploadKeep
    void *stage = nullptr;              // device staging for host-memory outputs
    size_t stage_bytes = 0;
    wxk::Job *jobs_dev = nullptr;       // job table of the one-shot batch entry point
    size_t jobs_cap = 0;
    wxk::Job *jobs_host = nullptr;      // pinned staging for that table
    cudaEvent_t jobs_done = nullptr;    // last one-shot batch's table copy
    std::vector<uint32_t> top;          // the top table of the last host build (upload_pools)
    uint32_t top_octants = 0;           // its octants that are not 32 throughout
    uint32_t sdf_spins = wxk::kSdfSpinLimit;  // bound of the waits in the GPU SDF's step control
    uint32_t *take_counter() {
        uint32_t *c = counters + next_counter;
        next_counter = (next_counter + 1) % kCounterSlots;
        return c;
    }
};

struct wx_grid {
    int device = 0;
    void *dev = nullptr;
    size_t bytes = 0;
    float *values = nullptr;  // level-set values (zero-crossing mode), own allocation
    uint2 *ovf = nullptr;     // leaf overflow table where it is not part of dev
    wxk::DevGrid g{};
    wx_grid_info info{};
};

struct wx_batch {
    wx_ctx *ctx = nullptr;
    wxk::Job *jobs_dev = nullptr;
    uint32_t njobs = 0, total_tiles = 0;
    uint64_t rays = 0;
    uint32_t *counter = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace wx {
// Injected allocation failures (wx_inject_alloc_failures), taken one per allocation.
static std::atomic<uint32_t> g_alloc_failures{0};
bool take_injected_alloc_failure() {
    uint32_t n = g_alloc_failures.load(std::memory_order_relaxed);
    while (n != 0 && !g_alloc_failures.compare_exchange_weak(n, n - 1, std::memory_order_relaxed)) {
    }
    return n != 0;
}
}  // namespace wx

namespace {

int fail(wx_ctx *ctx, int code, const std::string &msg) {
    if (ctx) ctx->err = msg;
    wx::set_thread_error(msg);
    return code;
}
int cuda_fail(wx_ctx *ctx, cudaError_t e, const char *what) {
    return fail(ctx, e == cudaErrorMemoryAllocation ? WX_ERR_OOM : WX_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e));
}
#define WX_CUDA(ctx, call)                                       \
    do {                                                         \
        cudaError_t e_ = (call);                                 \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, #call); \
    } while (0)

// Output byte ranges [lo, hi) (rgba8, hit records) of the last k_pixel launched
// on each (device, stream). A k_pixel launch's predecessor on its stream is
// either the k_pixel recorded here (the only kernel of this library that lets
// its dependents start early) or work after which nothing overlaps; k_pixel
// itself keeps frames older than the predecessor finished (kernels.cu). So a
// frame whose outputs are disjoint from the record's need not wait before its
// stores. A stream without a record counts as overlapping.
struct PixelOutputs {
    int device;
    cudaStream_t stream;
    uintptr_t lo[2], hi[2];
};
std::mutex g_ring_mu;
wxk::LaunchRing g_ring;
constexpr size_t kPixelStreams = 256;  // records kept, oldest dropped first
std::mutex g_pixel_mu;
std::vector<PixelOutputs> g_pixel_outputs;

// Launches k_pixel for cur's outputs and records cur as its stream's last
// k_pixel, both under g_pixel_mu, so a stream's record always names the k_pixel
// enqueued on it last even when several host threads launch on one stream. The
// frame stores without waiting when its outputs are disjoint from the record's.
// cudaStreamPerThread is one handle for a different stream in every host thread,
// so no record can name its predecessor: frames on it always wait. NULL and
// cudaStreamLegacy name the same stream.
cudaError_t launch_pixel_tracked(const wxk::Job &job, const wxk::Tuning &t, int num_sms, PixelOutputs cur) {
    const uint64_t others = wxk::enter_launch(cur.device, cur.stream, job.tiles, (uint64_t)num_sms * wxk::kSplitWarps);
    const uint32_t split = wxk::pixel_split(job.tiles, others, num_sms);
    if (cur.stream == cudaStreamPerThread) return wxk::launch_pixel(job, t, false, split, cur.stream);
    if (cur.stream == cudaStreamLegacy) cur.stream = nullptr;
    auto meet = [](uintptr_t a0, uintptr_t a1, uintptr_t b0, uintptr_t b1) {
        return a0 < a1 && b0 < b1 && a0 < b1 && b0 < a1;
    };
    std::lock_guard<std::mutex> lock(g_pixel_mu);
    auto &v = g_pixel_outputs;
    bool disjoint = false;
    size_t i = 0;
    while (i < v.size() && !(v[i].device == cur.device && v[i].stream == cur.stream)) i++;
    if (i < v.size()) {
        disjoint = true;
        for (int a = 0; a < 2; a++)
            for (int b = 0; b < 2; b++)
                if (meet(cur.lo[a], cur.hi[a], v[i].lo[b], v[i].hi[b])) disjoint = false;
        v.erase(v.begin() + (long)i);
    } else if (v.size() >= kPixelStreams) {
        v.erase(v.begin());
    }
    const cudaError_t e = wxk::launch_pixel(job, t, disjoint, split, cur.stream);
    if (e == cudaSuccess) v.push_back(cur);  // after a failed launch the stream's last kernel is unknown
    return e;
}

bool device_accessible(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// The device-side address of page-locked host memory (cudaMallocHost,
// cudaHostAlloc, cudaHostRegister), through which a kernel writes to the host
// buffer directly; nullptr for pageable memory.
void *pinned_device_alias(void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

// A device allocation freed on scope exit (temporaries of wx_grid_build_gpu).
struct DevBuf {
    void *p = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    template <class T>
    T *as() const {
        return static_cast<T *>(p);
    }
};
// The same from a memory pool, in the order of the legacy stream (the temporary of wx_grid_upload): nothing waits for other
// streams.
struct StreamBuf {
    void *p = nullptr;
    StreamBuf() = default;
    StreamBuf(const StreamBuf &) = delete;
    StreamBuf &operator=(const StreamBuf &) = delete;
    ~StreamBuf() { release(); }
    void release() {
        if (p) cudaFreeAsync(p, nullptr);
        p = nullptr;
    }
};

// The root block: header, origins and the dense table of root keys, which
// replaces the linear scan of get_vdb_leaf_from_nothing
// (raycast.comp.wgsl:398-413) with one load. The scan compares
// floor(p) & ~4095 with each origin, so only origins that are multiples of
// 4096 can match; the table holds those, the first of equal origins winning as
// in the scan. Boxes of more than 2^20 keys keep the scan (use table = 0).
std::vector<int4> root_block(const std::vector<int4> &o5, uint64_t n5) {
    constexpr uint64_t kMaxKeys = 1u << 20;
    int lo[3] = {0, 0, 0}, hi[3] = {-1, -1, -1};
    bool any = false;
    for (uint64_t i = 0; i < n5; i++) {
        const int v[3] = {o5[i].x, o5[i].y, o5[i].z};
        if ((v[0] & 4095) || (v[1] & 4095) || (v[2] & 4095)) continue;
        for (int a = 0; a < 3; a++) {
            const int k = v[a] >> 12;
            lo[a] = any ? std::min(lo[a], k) : k;
            hi[a] = any ? std::max(hi[a], k) : k;
        }
        any = true;
    }
    uint64_t dim[3], keys = 1;
    for (int a = 0; a < 3; a++) {
        dim[a] = any ? (uint64_t)((int64_t)hi[a] - lo[a] + 1) : 0;
        keys *= dim[a];
    }
    const bool use = keys <= kMaxKeys;
    const uint64_t tab = use ? keys : 0;
    std::vector<int4> b(2 + n5 + (tab + 3) / 4, make_int4(0, 0, 0, 0));
    b[0] = make_int4(lo[0], lo[1], lo[2], (int)(use ? dim[0] : 0));
    b[1] = make_int4((int)(use ? dim[1] : 0), (int)(use ? dim[2] : 0), 0, use ? 1 : 0);
    for (uint64_t i = 0; i < n5; i++) b[2 + i] = o5[i];
    auto *t = reinterpret_cast<uint32_t *>(b.data() + 2 + n5);
    for (uint64_t i = 0; use && i < n5; i++) {
        const int v[3] = {o5[i].x, o5[i].y, o5[i].z};
        if ((v[0] & 4095) || (v[1] & 4095) || (v[2] & 4095)) continue;
        const uint64_t e = ((uint64_t)((v[2] >> 12) - lo[2]) * dim[1] + (uint64_t)((v[1] >> 12) - lo[1])) * dim[0] +
                           (uint64_t)((v[0] >> 12) - lo[0]);
        if (!t[e]) t[e] = (uint32_t)i + 1u;
    }
    return b;
}

// The kernels address each pool with a 32-bit element index (node << log2 slots | slot).
int check_pool_limits(wx_ctx *ctx, uint64_t n5, uint64_t n4, uint64_t n3) {
    if (n5 > (1u << 17) || n4 > (1u << 20) || n3 > (1u << 23))
        return fail(ctx, WX_ERR_UNSUPPORTED,
                    "grid too large: at most 131072 N5, 1048576 N4 and 8388608 N3 nodes");
    return WX_OK;
}

// One device block for all pools of a grid (layout at the top of this file);
// the root block is copied in, the other pools are left for the caller.
int alloc_grid(wx_ctx *ctx, const std::vector<int4> &o5, uint64_t n5, uint64_t n4, uint64_t n3, uint64_t n_ovf,
               wx_grid **out) {
    auto *gr = new (std::nothrow) wx_grid();
    if (!gr) return fail(ctx, WX_ERR_OOM, "host allocation failed");
    std::vector<int4> root;
    try {
        root = root_block(o5, n5);
    } catch (...) {
        delete gr;
        return fail(ctx, WX_ERR_OOM, "host allocation failed");
    }
    auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t b_top = wxk::kTopWords * sizeof(uint32_t), b_o5 = align(root.size() * 16) + b_top, b5 = align(n5 * 32768ull * 4),
                 b4 = align(n4 * 4096ull * 4), b3 = align(n3 * 512ull), bo = align(n_ovf * 8);
    gr->bytes = b_o5 + b5 + b4 + b3 + bo;
    gr->device = ctx->device;
    cudaError_t e = wx::dev_alloc(&gr->dev, gr->bytes);
    if (e != cudaSuccess) {
        delete gr;
        return cuda_fail(ctx, e, "cudaMalloc(node pools)");
    }
    char *b = static_cast<char *>(gr->dev);
    gr->g.root = reinterpret_cast<const int4 *>(b);
    gr->g.slot5 = reinterpret_cast<const uint32_t *>(b + b_o5);
    gr->g.slot4 = reinterpret_cast<const uint32_t *>(b + b_o5 + b5);
    gr->g.leaf = reinterpret_cast<const uint8_t *>(b + b_o5 + b5 + b4);
    gr->g.ovf = reinterpret_cast<const uint2 *>(b + b_o5 + b5 + b4 + b3);
    gr->g.n5 = (uint32_t)n5;
    gr->g.n4 = (uint32_t)n4;
    gr->g.n3 = (uint32_t)n3;
    gr->g.n_ovf = (uint32_t)n_ovf;
    gr->g.inside = 1u;
    for (uint64_t i = 0; i < n5; i++)
        for (int c : {o5[i].x, o5[i].y, o5[i].z})
            if (c != -4096 && c != 0) gr->g.inside = 0u;
    gr->info.n5 = n5;
    gr->info.n4 = n4;
    gr->info.n3 = n3;
    gr->info.device_bytes = gr->bytes;
    e = cudaMemcpy((void *)gr->g.root, root.data(), root.size() * 16, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(gr->dev);
        delete gr;
        return cuda_fail(ctx, e, "cudaMemcpy(root block)");
    }
    *out = gr;
    return WX_OK;
}

void free_grid(wx_grid *gr) {
    if (!gr) return;
    cudaFree(gr->dev);
    if (gr->values) cudaFree(gr->values);
    if (gr->ovf) cudaFree(gr->ovf);
    delete gr;
}

// Frees a grid under construction on scope exit.
struct GridGuard {
    wx_grid *g;
    ~GridGuard() { free_grid(g); }
};

// The leaf overflow table of n entries in a block of its own, for builds that learn n after alloc_grid.
int alloc_overflow(wx_ctx *ctx, wx_grid *gr, uint64_t n) {
    if (n > UINT32_MAX) return fail(ctx, WX_ERR_UNSUPPORTED, "leaf overflow table of 2^32 entries or more");
    WX_CUDA(ctx, wx::dev_alloc(&gr->ovf, n * 8));
    gr->g.ovf = gr->ovf;
    gr->g.n_ovf = (uint32_t)n;
    gr->bytes += (n * 8 + 255) & ~(size_t)255;
    gr->info.device_bytes = gr->bytes;
    return WX_OK;
}

// The kernels list overflow entries in any order; the march binary-searches them by key.
int sort_overflow(wx_ctx *ctx, wx_grid *gr) {
    std::vector<uint2> ov(gr->g.n_ovf);
    WX_CUDA(ctx, cudaMemcpy(ov.data(), gr->ovf, ov.size() * 8, cudaMemcpyDeviceToHost));
    std::sort(ov.begin(), ov.end(), [](const uint2 &a, const uint2 &b) { return a.x < b.x; });
    WX_CUDA(ctx, cudaMemcpy(gr->ovf, ov.data(), ov.size() * 8, cudaMemcpyHostToDevice));
    return WX_OK;
}

// Pack the per-voxel u32 leaf distances into bytes plus the overflow table,
// allocate one device block for all pools and upload them. The distances are
// compute_sdf's, far below 2^24 (the side of the largest cube of nodes that a grid can hold).
int upload_pools(wx_ctx *ctx, const std::vector<int4> &o5, const uint32_t *s5, const uint32_t *s4, const uint32_t *s3,
                 uint64_t n5, uint64_t n4, uint64_t n3, wx_grid **out) {
    int rc = check_pool_limits(ctx, n5, n4, n3);
    if (rc != WX_OK) return rc;
    std::vector<uint8_t> leaf;
    std::vector<uint2> ovf;
    try {
        if (ctx->top.empty()) ctx->top.assign(wxk::kTopWords, 32u);
        leaf.resize(n3 * wx::kN3Slots);
        const unsigned np = n3 < 4096 ? 1u : std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
        std::vector<std::vector<uint2>> parts(np);
        const size_t chunk = (n3 + np - 1) / np;
        auto pack = [&](unsigned p) {
            for (size_t k = p * chunk; k < std::min<size_t>(n3, (p + 1) * chunk); k++)
                for (uint32_t s = 0; s < wx::kN3Slots; s++) {
                    const uint32_t d = s3[k * wx::kN3Slots + s];
                    leaf[k * wx::kN3Slots + s] = (uint8_t)std::min<uint32_t>(d, 255u);
                    if (d >= 255u) parts[p].push_back(make_uint2((uint32_t)(k << 9) | s, d));
                }
        };
        std::vector<std::thread> th;
        for (unsigned p = 1; p < np; p++) th.emplace_back(pack, p);
        pack(0);
        for (auto &t : th) t.join();
        for (auto &p : parts) ovf.insert(ovf.end(), p.begin(), p.end());  // ascending keys
    } catch (...) {
        return fail(ctx, WX_ERR_OOM, "host allocation failed while packing leaves");
    }
    wx_grid *gr = nullptr;
    if ((rc = alloc_grid(ctx, o5, n5, n4, n3, ovf.size(), &gr)) != WX_OK) return rc;
    cudaError_t e = cudaSuccess;
    if (n5) e = cudaMemcpy((void *)gr->g.slot5, s5, n5 * 32768ull * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n4) e = cudaMemcpy((void *)gr->g.slot4, s4, n4 * 4096ull * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && n3) e = cudaMemcpy((void *)gr->g.leaf, leaf.data(), leaf.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !ovf.empty())
        e = cudaMemcpy((void *)gr->g.ovf, ovf.data(), ovf.size() * 8, cudaMemcpyHostToDevice);
    // The top table is made here, not by build_top_table: no kernel to wait for behind renders on other streams.
    for (uint32_t oct = 0; oct < 8u; oct++) {
        const uint32_t ox = oct >> 2, oy = (oct >> 1) & 1u, oz = oct & 1u;
        uint64_t i = 0;  // the first N5 there, as root_find gives it
        while (i < n5 && !(o5[i].x == (int)ox * 4096 - 4096 && o5[i].y == (int)oy * 4096 - 4096 && o5[i].z == (int)oz * 4096 - 4096)) i++;
        if (i == n5 && !((ctx->top_octants >> oct) & 1u)) continue;
        ctx->top_octants = (ctx->top_octants & ~(1u << oct)) | (i < n5 ? 1u << oct : 0u);
        for (uint32_t xy = 0; xy < 1024u; xy++) {
            uint32_t *row = &ctx->top[((ox * 32u + (xy >> 5)) << 12) | ((oy * 32u + (xy & 31u)) << 6) | (oz * 32u)];
            if (i < n5) memcpy(row, s5 + i * wx::kN5Slots + xy * 32u, 32 * sizeof(uint32_t));
            else std::fill(row, row + 32, 32u);
        }
    }
    if (e == cudaSuccess)
        e = cudaMemcpy((void *)(gr->g.slot5 - wxk::kTopWords), ctx->top.data(), ctx->top.size() * 4, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        free_grid(gr);
        return cuda_fail(ctx, e, "cudaMemcpy(node pools)");
    }
    *out = gr;
    return WX_OK;
}

// Tiles of tile_w x (32 / tile_w) pixels over the dispatched region
// 8*floor(w/8) x 4*floor(h/4) (wgpu_context.rs:281).
wxk::Job make_job(const wx_grid *grid, const wx_state_uniform &s, uint32_t width, uint32_t height, uint32_t *rgba,
                  wx_hit *hits, uint32_t tile_begin, const wxk::Tuning &t) {
    wxk::Job j;
    memset(&j, 0, sizeof j);
    j.g = grid->g;
    j.width = width;
    j.height = height;
    j.tile_w = (uint16_t)t.tile_w;
    j.order = (uint32_t)t.order;
    j.tile_h = (uint16_t)(32u / j.tile_w);
    const uint32_t wd = width & ~7u, hd = height & ~3u;
    j.tiles_x = (wd + j.tile_w - 1) / j.tile_w;
    j.tiles = j.tiles_x * ((hd + j.tile_h - 1) / j.tile_h);
    j.tile_begin = tile_begin;
    j.rgba = rgba;
    j.hits = hits;
    j.s = s;
    return j;
}

}  // namespace

uint64_t wxk::enter_launch(int device, cudaStream_t st, uint64_t tiles, uint64_t enough) {
    static thread_local char thread;
    if (st == cudaStreamLegacy) st = nullptr;
    std::lock_guard<std::mutex> lock(g_ring_mu);
    return g_ring.enter(device, reinterpret_cast<uintptr_t>(st),
                        st == cudaStreamPerThread ? reinterpret_cast<uintptr_t>(&thread) : 0, tiles, enough);
}

void wxk::ctx_device_info(const wx_ctx *ctx, int *device, int *num_sms) {
    *device = ctx->device;
    *num_sms = ctx->num_sms;
}

bool wxk::grid_device_view(const wx_grid *grid, wxk::DevGrid *out, int *device) {
    if (!grid) return false;
    *out = grid->g;
    *device = grid->device;
    return true;
}

extern "C" {

const char *wx_status_string(int status) {
    switch (status) {
        case WX_OK: return "ok";
        case WX_ERR_INVALID: return "invalid argument";
        case WX_ERR_CUDA: return "CUDA error";
        case WX_ERR_OOM: return "out of memory";
        case WX_ERR_UNSUPPORTED: return "unsupported";
        case WX_ERR_BUDGET: return "over memory budget";
        case WX_ERR_TIMEOUT: return "timed out";
        case WX_ERR_CANCELLED: return "cancelled";
        default: return "unknown status";
    }
}

int wx_ctx_create(int device, wx_ctx **out) {
    return wx::guard("wx_ctx_create", [&]() -> int {
        if (!out) return fail(nullptr, WX_ERR_INVALID, "wx_ctx_create: out is NULL");
        int n = 0;
        cudaError_t e = cudaGetDeviceCount(&n);
        if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDeviceCount");
        if (device < 0 || device >= n) return fail(nullptr, WX_ERR_INVALID, "wx_ctx_create: no such device");
        WX_CUDA(nullptr, cudaSetDevice(device));
        auto *c = new (std::nothrow) wx_ctx();
        if (!c) return fail(nullptr, WX_ERR_OOM, "host allocation failed");
        c->device = device;
        auto cleanup = [&](cudaError_t err, const char *what) {
            wx_ctx_destroy(c);
            return cuda_fail(nullptr, err, what);
        };
        if ((e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess)
            return cleanup(e, "cudaDeviceGetAttribute");
        if ((e = wxk::init_device_tables()) != cudaSuccess) return cleanup(e, "init_device_tables");
        if ((e = wx::dev_alloc(&c->counters, kCounterSlots * sizeof(uint32_t))) != cudaSuccess)
            return cleanup(e, "cudaMalloc(counters)");
        if ((e = cudaMemset(c->counters, 0, kCounterSlots * sizeof(uint32_t))) != cudaSuccess)
            return cleanup(e, "cudaMemset(counters)");
        if ((e = wx::dev_alloc(&c->check, 4 * sizeof(unsigned long long))) != cudaSuccess)
            return cleanup(e, "cudaMalloc(check)");
        if ((e = cudaEventCreateWithFlags(&c->jobs_done, cudaEventDisableTiming)) != cudaSuccess)
            return cleanup(e, "cudaEventCreate");
        *out = c;
        return WX_OK;
    });
}

int wx_ctx_destroy(wx_ctx *ctx) {
    return wx::guard("wx_ctx_destroy", [&]() -> int {
        if (!ctx) return WX_OK;
        cudaSetDevice(ctx->device);
        if (ctx->jobs_done) {
            cudaEventSynchronize(ctx->jobs_done);
            cudaEventDestroy(ctx->jobs_done);
        }
        if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
        if (ctx->stage) cudaFree(ctx->stage);
        if (ctx->counters) cudaFree(ctx->counters);
        if (ctx->check) cudaFree(ctx->check);
        if (ctx->jobs_dev) cudaFree(ctx->jobs_dev);
        if (ctx->jobs_host) cudaFreeHost(ctx->jobs_host);
        delete ctx;
        return WX_OK;
    });
}

const char *wx_last_error(const wx_ctx *ctx) { return ctx ? ctx->err.c_str() : wx_thread_last_error(); }

int wx_ctx_set_tuning(wx_ctx *ctx, const wx_tuning *t) {
    return wx::guard("wx_ctx_set_tuning", [&]() -> int {
        if (!ctx || !t) return fail(ctx, WX_ERR_INVALID, "wx_ctx_set_tuning: null argument");
        const bool tw_ok = t->tile_width == 4 || t->tile_width == 8 || t->tile_width == 16 || t->tile_width == 32;
        if (t->kernel < 0 || t->kernel > 1 || t->warps_per_block < 1 || t->warps_per_block > 8 || t->blocks_per_sm < 0 ||
            t->blocks_per_sm > 64 || !tw_ok || t->tile_order < 0 || t->tile_order > 1 ||
            !(t->rays_per_lane == 1 || t->rays_per_lane == 2 || t->rays_per_lane == 4 || t->rays_per_lane == 8))
            return fail(ctx, WX_ERR_INVALID, "wx_ctx_set_tuning: value out of range");
        ctx->tuning.kernel = t->kernel;
        ctx->tuning.warps_per_block = t->warps_per_block;
        ctx->tuning.blocks_per_sm = t->blocks_per_sm;
        ctx->tuning.tile_w = t->tile_width;
        ctx->tuning.order = t->tile_order;
        ctx->tuning.rays = t->rays_per_lane;
        return WX_OK;
    });
}

int wx_inject_alloc_failures(uint32_t count) {
    return wx::guard("wx_inject_alloc_failures", [&]() -> int {
        wx::g_alloc_failures.store(count, std::memory_order_relaxed);
        return WX_OK;
    });
}

int wx_ctx_set_sdf_wait_limit(wx_ctx *ctx, uint32_t polls) {
    return wx::guard("wx_ctx_set_sdf_wait_limit", [&]() -> int {
        if (!ctx) return WX_ERR_INVALID;
        ctx->sdf_spins = polls ? polls : wxk::kSdfSpinLimit;
        return WX_OK;
    });
}

int wx_ctx_get_tuning(const wx_ctx *ctx, wx_tuning *t) {
    return wx::guard("wx_ctx_get_tuning", [&]() -> int {
        if (!ctx || !t) return WX_ERR_INVALID;
        t->kernel = ctx->tuning.kernel;
        t->warps_per_block = ctx->tuning.warps_per_block;
        t->blocks_per_sm = ctx->tuning.blocks_per_sm;
        t->tile_width = ctx->tuning.tile_w;
        t->tile_order = ctx->tuning.order;
        t->rays_per_lane = ctx->tuning.rays;
        return WX_OK;
    });
}

int wx_autotune(wx_ctx *ctx, const wx_frame *frames, uint32_t n, const wx_tuning *candidates, uint32_t ncand,
                uint32_t reps, wx_tuning *best, double *times_ms) {
    return wx::guard("wx_autotune", [&]() -> int {
        if (!ctx || !frames || n == 0 || !best) return fail(ctx, WX_ERR_INVALID, "wx_autotune: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        std::vector<wx_tuning> cand;
        if (candidates) {
            cand.assign(candidates, candidates + ncand);
        } else {
            for (int order : {1, 0}) {
                for (int kernel : {0, 1})
                    for (int tw : {4, 8, 16})
                        for (int wpb : {2, 4, 8}) cand.push_back(wx_tuning{kernel, wpb, 0, tw, order, 1});
                // Occupancy of the persistent kernel: fewer resident warps than fit (16 per SM).
                for (int tw : {4, 8}) cand.push_back(wx_tuning{0, 4, 4, tw, order, 1});
                // Rays per lane: warps of several tiles whose lanes refill.
                for (int rays : {2, 4, 8})
                    for (int tw : {4, 8})
                        for (int wpb : {2, 4}) cand.push_back(wx_tuning{1, wpb, 0, tw, order, rays});
            }
            if (cand.size() != WX_AUTOTUNE_BUILTIN) return fail(ctx, WX_ERR_INVALID, "wx_autotune: built-in set size");
        }
        if (cand.empty()) return fail(ctx, WX_ERR_INVALID, "wx_autotune: no candidates");
        for (uint32_t i = 0; i < n; i++)
            if (!frames[i].grid || !frames[i].rgba8 || !device_accessible(frames[i].rgba8))
                return fail(ctx, WX_ERR_INVALID, "wx_autotune: frames need a grid and device rgba8");
        const wxk::Tuning saved = ctx->tuning;
        cudaEvent_t e0, e1;
        WX_CUDA(ctx, cudaEventCreate(&e0));
        WX_CUDA(ctx, cudaEventCreate(&e1));
        cudaStream_t st;
        WX_CUDA(ctx, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        double best_ms = 1e300;
        size_t best_i = 0;
        int rc = WX_OK;
        for (size_t c = 0; c < cand.size() && rc == WX_OK; c++) {
            rc = wx_ctx_set_tuning(ctx, &cand[c]);
            if (rc != WX_OK) break;
            double total = 0;
            for (uint32_t rep = 0; rep <= reps && rc == WX_OK; rep++) {  // pass 0 warms up
                cudaEventRecord(e0, st);
                for (uint32_t i = 0; i < n && rc == WX_OK; i++)
                    rc = wx_render(ctx, frames[i].grid, &frames[i].state, frames[i].width, frames[i].height,
                                   frames[i].rgba8, frames[i].hits, st);
                cudaEventRecord(e1, st);
                cudaEventSynchronize(e1);
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                if (rep > 0) total += ms;
            }
            const double mean = total / (reps ? reps : 1);
            if (times_ms) times_ms[c] = mean;
            if (rc == WX_OK && mean < best_ms) {
                best_ms = mean;
                best_i = c;
            }
        }
        cudaStreamDestroy(st);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (rc != WX_OK) {
            ctx->tuning = saved;
            return rc;
        }
        *best = cand[best_i];
        return wx_ctx_set_tuning(ctx, best);
    });
}

int wx_check_division(wx_ctx *ctx, uint32_t max_m, uint64_t out[3]) {
    return wx::guard("wx_check_division", [&]() -> int {
        if (!ctx || !out) return fail(ctx, WX_ERR_INVALID, "wx_check_division: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        WX_CUDA(ctx, wxk::check_division(max_m, ctx->check, nullptr));
        unsigned long long h[3];
        WX_CUDA(ctx, cudaMemcpy(h, ctx->check, sizeof h, cudaMemcpyDeviceToHost));
        for (int i = 0; i < 3; i++) out[i] = h[i];
        return WX_OK;
    });
}

int wx_bounds_violations(wx_ctx *ctx, uint64_t *count) {
    return wx::guard("wx_bounds_violations", [&]() -> int {
        if (!ctx || !count) return fail(ctx, WX_ERR_INVALID, "wx_bounds_violations: null argument");
    #ifdef WX_BOUNDS_CHECK
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        WX_CUDA(ctx, cudaDeviceSynchronize());
        unsigned long long n = 0;
        WX_CUDA(ctx, wxk::take_bounds_violations(&n));
        *count = n;
        return WX_OK;
    #else
        *count = 0;
        return fail(ctx, WX_ERR_UNSUPPORTED, "wx_bounds_violations: not a bounds-checked build");
    #endif
    });
}

int wx_grid_build(wx_ctx *ctx, wx_topology *t, wx_grid **out) {
    return wx::guard("wx_grid_build", [&]() -> int {
        if (!ctx || !t || !out) return fail(ctx, WX_ERR_INVALID, "wx_grid_build: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        int rc = wx_topology_sdf(t, 0);
        if (rc != WX_OK) return fail(ctx, rc, wx_thread_last_error());
        const uint64_t n5 = t->n5(), n4 = t->n4(), n3 = t->n3();
        if (n4 >= wx::kChildFlag || n3 >= wx::kChildFlag)
            return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_build: more than 2^31 nodes in a level");
        std::vector<uint32_t> s5, s4;
        std::vector<int4> o5(std::max<uint64_t>(n5, 1));
        try {
            s5.resize(n5 * wx::kN5Slots);
            s4.resize(n4 * wx::kN4Slots);
        } catch (...) {
            return fail(ctx, WX_ERR_OOM, "wx_grid_build: host allocation failed");
        }
        bool too_far = false;
        for (uint64_t i = 0; i < n5; i++) {
            o5[i] = make_int4(t->o5[i][0], t->o5[i][1], t->o5[i][2], 0);
            uint32_t next = t->first4[i];
            for (uint32_t s = 0; s < wx::kN5Slots; s++) {
                const bool kid = wx::test_bit(&t->kid5[i * wx::kN5Words], s);
                const bool val = wx::test_bit(&t->val5[i * wx::kN5Words], s);
                const uint32_t d = t->d5[i * wx::kN5Slots + s];
                if (kid) {
                    const uint32_t c = next++;
                    s5[i * wx::kN5Slots + s] = val ? 0u : (wx::kChildFlag | c);
                } else {
                    too_far |= !val && d >= wx::kChildFlag;
                    s5[i * wx::kN5Slots + s] = val ? 0u : d;
                }
            }
        }
        for (uint64_t j = 0; j < n4; j++) {
            uint32_t next = t->first3[j];
            for (uint32_t s = 0; s < wx::kN4Slots; s++) {
                const bool kid = wx::test_bit(&t->kid4[j * wx::kN4Words], s);
                const bool val = wx::test_bit(&t->val4[j * wx::kN4Words], s);
                const uint32_t d = t->d4[j * wx::kN4Slots + s];
                if (kid) {
                    const uint32_t c = next++;
                    s4[j * wx::kN4Slots + s] = val ? 0u : (wx::kChildFlag | c);
                } else {
                    too_far |= !val && d >= wx::kChildFlag;
                    s4[j * wx::kN4Slots + s] = val ? 0u : d;
                }
            }
        }
        if (too_far) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_build: tile distance >= 2^31");
        wx_grid *gr = nullptr;
        rc = upload_pools(ctx, o5, s5.data(), s4.data(), t->slot3.data(), n5, n4, n3, &gr);
        if (rc != WX_OK) return rc;
        gr->info.active_voxels = wx_topology_active_voxels(t);
        *out = gr;
        return WX_OK;
    });
}

// The same pools as wx_grid_build, with compute_sdf and the packing on the
// GPU (sdf.cu). The host uploads only the masks and the N5 origins; child
// tables, child origins, neighbour tables, the distances and the packing run on
// the device.
int wx_grid_build_gpu(wx_ctx *ctx, const wx_topology *t, wx_grid **out) {
    return wx::guard("wx_grid_build_gpu", [&]() -> int {
        if (!ctx || !t || !out) return fail(ctx, WX_ERR_INVALID, "wx_grid_build_gpu: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        using namespace wx;
        const uint64_t n5 = t->n5(), n4 = t->n4(), n3 = t->n3();
        int rc = check_pool_limits(ctx, n5, n4, n3);
        if (rc != WX_OK) return rc;
        if (t->kid5.size() != n5 * kN5Words || t->val5.size() != n5 * kN5Words || t->kid4.size() != n4 * kN4Words ||
            t->val4.size() != n4 * kN4Words || t->val3.size() != n3 * kN3Words || t->first4.size() != n5 ||
            t->first3.size() != n4)
            return fail(ctx, WX_ERR_INVALID, "wx_grid_build_gpu: masks and node counts disagree");
        std::vector<int4> o5(std::max<uint64_t>(n5, 1));
        for (uint64_t i = 0; i < n5; i++) {
            o5[i] = make_int4(t->o5[i][0], t->o5[i][1], t->o5[i][2], 0);
            if ((o5[i].x & 4095) || (o5[i].y & 4095) || (o5[i].z & 4095))
                return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_build_gpu: N5 origins must be multiples of 4096");
        }
        std::vector<int4> root;
        try {
            root = root_block(o5, n5);
        } catch (...) {
            return fail(ctx, WX_ERR_OOM, "wx_grid_build_gpu: host allocation failed");
        }

        // Temporaries, carved from one allocation: masks, child tables, origins, neighbours and the sets of the
        // distance computation.
        DevBuf tmp;
        size_t need = 0;
        auto carve = [&](size_t bytes) {
            const size_t at = need;
            need += (bytes + 255) & ~(size_t)255;
            return at;
        };
        const uint64_t nodes[3] = {n5, n4, n3}, words[3] = {n5 * kN5Words, n4 * kN4Words, n3 * kN3Words};
        size_t z[3], val[2], org[3], nb[3], act[3], pre[2], first[2], cidx[2];
        const uint64_t node_words[3] = {kN5Words, kN4Words, kN3Words};
        for (int l = 0; l < 3; l++) {
            z[l] = carve((words[l] + node_words[l]) * (wxk::kSdfWindow + 3) * 8);
            org[l] = carve(nodes[l] * 16);
            nb[l] = carve(nodes[l] * 27 * 4);
            act[l] = carve((nodes[l] + 1) * 4);
            if (l == 2) break;
            val[l] = carve(words[l] * 8);
            pre[l] = carve(words[l] * 4);
            first[l] = carve(nodes[l] * 4);
            cidx[l] = carve(words[l] * 64 * 4);
        }
        const size_t at_root = carve(root.size() * 16), at_ctl = carve(sizeof(wxk::SdfCtl));
        WX_CUDA(ctx, wx::dev_alloc(&tmp.p, need));
        char *const base = static_cast<char *>(tmp.p);
        auto u64 = [&](size_t at) { return reinterpret_cast<uint64_t *>(base + at); };
        auto u32 = [&](size_t at) { return reinterpret_cast<uint32_t *>(base + at); };
        auto i4 = [&](size_t at) { return reinterpret_cast<int4 *>(base + at); };
        // The grid's pools; the overflow table, rarely needed, follows in a block of its own.
        wx_grid *gr = nullptr;
        if ((rc = alloc_grid(ctx, o5, n5, n4, n3, 0, &gr)) != WX_OK) return rc;
        GridGuard guard{gr};
        struct Up {
            size_t at;
            const void *src;
            size_t bytes;
        } ups[] = {{z[0], t->kid5.data(), words[0] * 8},  {val[0], t->val5.data(), words[0] * 8},
                   {z[1], t->kid4.data(), words[1] * 8},  {val[1], t->val4.data(), words[1] * 8},
                   {z[2], t->val3.data(), words[2] * 8},  {first[0], t->first4.data(), n5 * 4},
                   {first[1], t->first3.data(), n4 * 4},  {at_root, root.data(), root.size() * 16},
                   {org[0], o5.data(), n5 * 16}};
        for (auto &u : ups)
            if (u.bytes) WX_CUDA(ctx, cudaMemcpy(base + u.at, u.src, u.bytes, cudaMemcpyHostToDevice));
        const cudaStream_t st = nullptr;
        auto *const ctl = reinterpret_cast<wxk::SdfCtl *>(base + at_ctl);
        WX_CUDA(ctx, cudaMemsetAsync(ctl, 0, sizeof *ctl, st));
        WX_CUDA(ctx, wxk::sdf_child_table(u64(z[0]), u32(pre[0]), u32(first[0]), n5, 15, u32(cidx[0]), st));
        WX_CUDA(ctx, wxk::sdf_child_table(u64(z[1]), u32(pre[1]), u32(first[1]), n4, 12, u32(cidx[1]), st));
        WX_CUDA(ctx, wxk::sdf_child_origins(u32(cidx[0]), i4(org[0]), n5, 5, 7, i4(org[1]), st));
        WX_CUDA(ctx, wxk::sdf_child_origins(u32(cidx[1]), i4(org[1]), n4, 4, 3, i4(org[2]), st));
        const wxk::SdfTree tree{i4(at_root), (uint32_t)n5, u32(cidx[0]), u32(cidx[1])};
        uint32_t *const slots[2] = {const_cast<uint32_t *>(gr->g.slot5), const_cast<uint32_t *>(gr->g.slot4)};
        wxk::SdfWork work{};
        for (int l = 0; l < 3; l++) {
            WX_CUDA(ctx, wxk::sdf_neighbours(5 - l, i4(org[l]), (uint32_t)nodes[l], tree, u32(nb[l]), st));
            const size_t set = (words[l] + node_words[l]) * 8, real = words[l] * 8;
            if (nodes[l]) {
                WX_CUDA(ctx, cudaMemsetAsync(base + act[l], 0, (nodes[l] + 1) * 4, st));
                // The missing neighbour's ones, in z and the W sets.
                WX_CUDA(ctx, cudaMemset2DAsync(base + z[l] + real, set, 0xFF, set - real, wxk::kSdfWindow + 1, st));
            }
            WX_CUDA(ctx, wxk::sdf_count_clear(u64(z[l]), words[l], &ctl->left[l], st));
            work.lv[l] = wxk::SdfLevel{u64(z[l]), (uint32_t)(set / 8), l < 2 ? u64(val[l]) : nullptr, u32(nb[l]), u32(act[l]),
                                       l < 2 ? slots[l] : nullptr, (uint32_t)nodes[l]};
        }
        WX_CUDA(ctx, cudaMemcpyAsync(&ctl->inactive, &ctl->left[2], 8, cudaMemcpyDeviceToDevice, st));
        work.leaf = const_cast<uint8_t *>(gr->g.leaf);
        work.ctl = ctl;
        // Distances below 255 first; the leaf cells then left are the overflow entries.
        wxk::SdfCtl h;
        WX_CUDA(ctx, wxk::sdf_levels(work, 1, wxk::kSdfWindow, ctx->num_sms, ctx->sdf_spins, st));
        WX_CUDA(ctx, wxk::sdf_expand(work, u32(cidx[0]), u32(cidx[1]), st));
        WX_CUDA(ctx, wxk::sdf_levels(work, wxk::kSdfWindow + 1, 254, ctx->num_sms, ctx->sdf_spins, st));
        WX_CUDA(ctx, wxk::build_top_table(gr->g, st));
        WX_CUDA(ctx, cudaMemcpy(&h, ctl, sizeof h, cudaMemcpyDeviceToHost));
        if (!h.error && (h.left[0] | h.left[1] | h.left[2])) {
            const uint64_t n_ovf = h.left[2];
            if (n_ovf && (rc = alloc_overflow(ctx, gr, n_ovf)) != WX_OK) return rc;
            work.ovf = gr->ovf;
            work.ovf_cap = (uint32_t)n_ovf;
            WX_CUDA(ctx, wxk::sdf_levels(work, 255, wxk::kSdfMaxLevel, ctx->num_sms, ctx->sdf_spins, st));
            WX_CUDA(ctx, wxk::build_top_table(gr->g, st));
            WX_CUDA(ctx, cudaMemcpy(&h, ctl, sizeof h, cudaMemcpyDeviceToHost));
            if (n_ovf && !h.error && (rc = sort_overflow(ctx, gr)) != WX_OK) return rc;
        }
        if (h.error) return fail(ctx, WX_ERR_TIMEOUT, "wx_grid_build_gpu: the distance steps' barrier wait hit its bound");
        if (h.left[0] | h.left[1] | h.left[2]) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_build_gpu: distances above 4095");
        gr->info.active_voxels = n3 * kN3Slots - h.inactive;
        guard.g = nullptr;
        *out = gr;
        return WX_OK;
    });
}

int wx_grid_read_pools(wx_ctx *ctx, const wx_grid *grid, uint32_t *slot5, uint32_t *slot4, uint8_t *leaf,
                       uint32_t *ovf, uint64_t *n_ovf) {
    return wx::guard("wx_grid_read_pools", [&]() -> int {
        if (!ctx || !grid) return fail(ctx, WX_ERR_INVALID, "wx_grid_read_pools: null argument");
        WX_CUDA(ctx, cudaSetDevice(grid->device));
        if (n_ovf) *n_ovf = grid->g.n_ovf;
        const uint64_t n5 = grid->info.n5, n4 = grid->info.n4, n3 = grid->info.n3;
        if (slot5 && n5) WX_CUDA(ctx, cudaMemcpy(slot5, grid->g.slot5, n5 * wx::kN5Slots * 4, cudaMemcpyDeviceToHost));
        if (slot4 && n4) WX_CUDA(ctx, cudaMemcpy(slot4, grid->g.slot4, n4 * wx::kN4Slots * 4, cudaMemcpyDeviceToHost));
        if (leaf && n3) WX_CUDA(ctx, cudaMemcpy(leaf, grid->g.leaf, n3 * wx::kN3Slots, cudaMemcpyDeviceToHost));
        if (ovf && grid->g.n_ovf)
            WX_CUDA(ctx, cudaMemcpy(ovf, grid->g.ovf, (size_t)grid->g.n_ovf * 8, cudaMemcpyDeviceToHost));
        return WX_OK;
    });
}

int wx_grid_upload(wx_ctx *ctx, const wx_vdb345_view *v, wx_grid **out) {
    return wx::guard("wx_grid_upload", [&]() -> int {
        if (!ctx || !v || !out) return fail(ctx, WX_ERR_INVALID, "wx_grid_upload: null argument");
        if (v->origin_stride < 3) return fail(ctx, WX_ERR_INVALID, "wx_grid_upload: origin_stride < 3");
        const uint64_t n5 = v->n5, n4 = v->n4, n3 = v->n3;
        if ((n5 && (!v->kids5 || !v->vals5 || !v->origins || !v->atlas[0])) ||
            (n4 && (!v->kids4 || !v->vals4 || !v->atlas[1])) || (n3 && (!v->vals3 || !v->atlas[2])))
            return fail(ctx, WX_ERR_INVALID, "wx_grid_upload: missing mask/atlas arrays");
        if (n4 >= wx::kChildFlag || n3 >= wx::kChildFlag || n5 >= wx::kChildFlag)
            return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_upload: more than 2^31 nodes in a level");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        // Atlas block placement as the shader computes it: dim = textureDimensions
        // (.y for N5, .x for N4/N3) >> log2(node dim); block (idx%d, (idx/d)%d, idx/d^2).
        const uint32_t d5 = v->dims[0][1] >> 5, d4 = v->dims[1][0] >> 4, d3 = v->dims[2][0] >> 3;
        auto block_ok = [&](int lvl, uint64_t n, uint32_t d, uint32_t nd) {
            if (n == 0) return true;
            if (d == 0) return false;
            const uint64_t dd = (uint64_t)d * d;
            const uint64_t need_x = nd * std::min<uint64_t>(n, d), need_y = nd * std::min<uint64_t>((n + d - 1) / d, d),
                           need_z = nd * ((n + dd - 1) / dd);
            return need_x <= v->dims[lvl][0] && need_y <= v->dims[lvl][1] && need_z <= v->dims[lvl][2];
        };
        if (!block_ok(0, n5, d5, 32) || !block_ok(1, n4, d4, 16) || !block_ok(2, n3, d3, 8))
            return fail(ctx, WX_ERR_INVALID, "wx_grid_upload: atlas dimensions too small for the node counts");
        int rc = check_pool_limits(ctx, n5, n4, n3);
        if (rc != WX_OK) return rc;
        std::vector<int4> o5(std::max<uint64_t>(n5, 1));
        for (uint64_t i = 0; i < n5; i++) {
            const int32_t *o = v->origins + i * v->origin_stride;
            o5[i] = make_int4(o[0], o[1], o[2], 0);
        }
        // Piece by piece, an atlas and its nodes' masks are copied to the device and packed there (pack.cu). A piece is whole
        // layers of d * d nodes, or block rows (d nodes) of one layer: as many as fit the buffer, 64 MB where the
        // device has that beside the grid, less where it has not, down to one block row.
        const uint32_t *const kids[3] = {v->kids5, v->kids4, nullptr}, *const vals[3] = {v->vals5, v->vals4, v->vals3};
        struct Atlas {
            uint64_t n, rows;
            uint32_t d, log2, words;          // mask words of a node
            size_t texel_row, slice, row;     // bytes: texels of a block row; one texel layer; a block row with its masks
        } atlas[3] = {{n5, 0, d5, 5, 1024, 0, 0, 0}, {n4, 0, d4, 4, 128, 0, 0, 0}, {n3, 0, d3, 3, 16, 0, 0, 0}};
        constexpr size_t kFixed = 1024;  // counters and alignment
        size_t least = kFixed, most = kFixed;
        for (int l = 0; l < 3; l++) {
            Atlas &a = atlas[l];
            if (!a.n) continue;
            a.rows = (a.n + a.d - 1) / a.d;
            a.texel_row = (size_t)v->dims[l][0] << (2 * a.log2 + 2);
            a.slice = (size_t)v->dims[l][0] * v->dims[l][1] * 4;
            a.row = a.texel_row + std::min<uint64_t>(a.n, a.d) * a.words * (kids[l] ? 8 : 4);
            least = std::max(least, kFixed + a.row);
            most = std::max(most, kFixed + a.row * (a.rows < a.d ? a.rows : (a.rows + a.d - 1) / a.d * a.d));
        }
        if (!ctx->pool) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.location = {cudaMemLocationTypeDevice, ctx->device};
            WX_CUDA(ctx, cudaMemPoolCreate(&ctx->pool, &props));
            uint64_t keep = kUploadKeep;
            WX_CUDA(ctx, cudaMemPoolSetAttribute(ctx->pool, cudaMemPoolAttrReleaseThreshold, &keep));
        }
        wx_grid *gr = nullptr;
        StreamBuf tmp;
        size_t bytes = std::max(least, std::min(most, kUploadBuffer));
        for (;; bytes = std::max(least, bytes / 2)) {
            const cudaError_t e = wx::dev_alloc_async(&tmp.p, bytes, ctx->pool, nullptr);
            rc = e == cudaSuccess ? alloc_grid(ctx, o5, n5, n4, n3, 0, &gr) : cuda_fail(ctx, e, "cudaMalloc(upload buffer)");
            if (rc == WX_OK) break;
            tmp.release();
            if (rc != WX_ERR_OOM || bytes == least) return rc;
            cudaStreamSynchronize(nullptr);
            cudaMemPoolTrimTo(ctx->pool, 0);
            cudaGetLastError();
        }
        GridGuard guard{gr};
        char *const base = static_cast<char *>(tmp.p);
        const cudaStream_t st = nullptr;
        struct Counts {
            unsigned long long n_ovf, clear;
            uint32_t flags;
        } h{}, *const dev = reinterpret_cast<Counts *>(base);
        WX_CUDA(ctx, cudaMemsetAsync(dev, 0, sizeof(Counts), st));
        auto pack = [&](int l) -> cudaError_t {
            const Atlas &a = atlas[l];
            if (!a.n) return cudaSuccess;
            const uint64_t fit = (bytes - kFixed) / a.row;
            for (uint64_t at = 0, step; at < a.rows; at += step) {
                const uint64_t z = at / a.d, r = at % a.d, left = a.rows - at;
                uint64_t layers = 1, rows = std::min({left, a.d - r, fit});  // block rows of a layer
                if (r == 0 && rows == a.d) {
                    layers = std::min(fit, left) / a.d;
                    if (left > layers * a.d && (layers + 1) * a.d <= fit) layers++;  // the last one, partly filled
                }
                step = layers * rows;
                const uint64_t first = at * a.d, count = std::min(step * a.d, a.n - first);
                const size_t width = rows * a.texel_row >> a.log2;  // bytes of a texel layer of the piece
                char *to = base + 256;
                const char *from = reinterpret_cast<const char *>(v->atlas[l]) + (z << a.log2) * a.slice + r * (a.texel_row >> a.log2);
                const size_t slices = layers << a.log2;
                cudaError_t e = cudaSuccess;
                if (width == a.slice) e = cudaMemcpy(to, from, slices * width, cudaMemcpyHostToDevice);
                else if (a.slice <= INT32_MAX) e = cudaMemcpy2D(to, width, from, a.slice, width, slices, cudaMemcpyHostToDevice);
                else  // beyond the largest pitch of a copy
                    for (size_t k = 0; k < slices && e == cudaSuccess; k++)
                        e = cudaMemcpy(to + k * width, from + k * a.slice, width, cudaMemcpyHostToDevice);
                const wxk::ViewSlab s{reinterpret_cast<const uint32_t *>(to), v->dims[l][0], (uint32_t)(rows << a.log2), a.d, first, count};
                to += step * a.texel_row;
                const uint32_t *mask[2] = {nullptr, nullptr};
                for (int m = 0; m < 2 && e == cudaSuccess; m++) {
                    const uint32_t *src = m ? vals[l] : kids[l];
                    if (!src) continue;
                    to = base + (((size_t)(to - base) + 255) & ~(size_t)255);
                    mask[m] = reinterpret_cast<const uint32_t *>(to);
                    e = cudaMemcpy(to, src + first * a.words, count * a.words * 4, cudaMemcpyHostToDevice);
                    to += count * a.words * 4;
                }
                if (e != cudaSuccess) return e;
                if (l < 2) {
                    e = wxk::pack_view_nodes((int)a.log2, s, mask[0], mask[1], (uint32_t)(l == 0 ? n4 : n3),
                                             const_cast<uint32_t *>(l == 0 ? gr->g.slot5 : gr->g.slot4), &dev->flags, st);
                } else {
                    e = wxk::sdf_count_clear(reinterpret_cast<const uint64_t *>(mask[1]), count * 8, &dev->clear, st);
                    if (e == cudaSuccess)
                        e = wxk::pack_view_leaves(s, mask[1], const_cast<uint8_t *>(gr->g.leaf), gr->ovf, gr->g.n_ovf,
                                                  &dev->n_ovf, st);
                }
                if (e != cudaSuccess) return e;
            }
            return cudaSuccess;
        };
        for (int l = 0; l < 3; l++) WX_CUDA(ctx, pack(l));
        WX_CUDA(ctx, wxk::build_top_table(gr->g, st));
        WX_CUDA(ctx, cudaMemcpy(&h, dev, sizeof h, cudaMemcpyDeviceToHost));
        if (h.flags & 1u) return fail(ctx, WX_ERR_INVALID, "wx_grid_upload: child index in atlas out of range");
        if (h.flags & 2u) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_grid_upload: internal tile distance >= 2^31");
        if (h.flags & 4u) gr->g.inside |= 2u;
        if (h.n_ovf) {  // rare (hand-made views): the leaves once more, now with the overflow table
            rc = alloc_overflow(ctx, gr, h.n_ovf);
            if (rc != WX_OK) return rc;
            WX_CUDA(ctx, cudaMemsetAsync(dev, 0, sizeof(Counts), st));
            WX_CUDA(ctx, pack(2));
            if ((rc = sort_overflow(ctx, gr)) != WX_OK) return rc;
        }
        gr->info.active_voxels = n3 * wx::kN3Slots - h.clear;
        guard.g = nullptr;
        *out = gr;
        return WX_OK;
    });
}

int wx_grid_release(wx_ctx *ctx, wx_grid *grid) {
    return wx::guard("wx_grid_release", [&]() -> int {
        if (!grid) return WX_OK;
        cudaSetDevice(grid->device);
        cudaError_t e = cudaFree(grid->dev);
        if (grid->values) {
            const cudaError_t e2 = cudaFree(grid->values);
            if (e == cudaSuccess) e = e2;
        }
        if (grid->ovf) {
            const cudaError_t e2 = cudaFree(grid->ovf);
            if (e == cudaSuccess) e = e2;
        }
        delete grid;
        if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaFree(node pools)");
        return WX_OK;
    });
}

int wx_grid_set_values(wx_ctx *ctx, wx_grid *grid, const float *values, float band) {
    return wx::guard("wx_grid_set_values", [&]() -> int {
        if (!ctx || !grid || !values) return fail(ctx, WX_ERR_INVALID, "wx_grid_set_values: null argument");
        if (!(band > 0.0f) || !(band < 3.0e38f))
            return fail(ctx, WX_ERR_INVALID, "wx_grid_set_values: band must be positive and finite");
        WX_CUDA(ctx, cudaSetDevice(grid->device));
        const size_t bytes = (size_t)grid->info.n3 * wx::kN3Slots * sizeof(float);
        if (!grid->values && bytes) WX_CUDA(ctx, wx::dev_alloc(&grid->values, bytes));
        if (bytes) WX_CUDA(ctx, cudaMemcpy(grid->values, values, bytes, cudaMemcpyHostToDevice));
        grid->g.values = grid->values;
        grid->g.band = band;
        return WX_OK;
    });
}

int wx_grid_get_info(const wx_grid *grid, wx_grid_info *out) {
    return wx::guard("wx_grid_get_info", [&]() -> int {
        if (!grid || !out) return WX_ERR_INVALID;
        *out = grid->info;
        return WX_OK;
    });
}

int wx_render(wx_ctx *ctx, const wx_grid *grid, const wx_state_uniform *state, uint32_t width, uint32_t height,
              uint8_t *rgba8, wx_hit *hits, void *stream) {
    return wx::guard("wx_render", [&]() -> int {
        if (!ctx || !grid || !state || !rgba8) return fail(ctx, WX_ERR_INVALID, "wx_render: null argument");
        if (grid->device != ctx->device) return fail(ctx, WX_ERR_INVALID, "wx_render: grid is on another device");
        if (((uintptr_t)rgba8 & 3) || ((uintptr_t)hits & 15))
            return fail(ctx, WX_ERR_INVALID, "wx_render: rgba8 must be 4-byte and hits 16-byte aligned");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        const uint32_t tiles_x = width / 8, tiles_y = height / 4;
        const uint64_t ntiles = (uint64_t)tiles_x * tiles_y;
        if (ntiles == 0) return WX_OK;
        if ((uint64_t)width * height >= (1ull << 32)) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_render: frame too large");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        // Device memory and page-locked host memory are written by the kernel itself
        // (page-locked memory through its device alias, over the host link while the
        // march runs); pageable host memory goes through the context's staging buffer.
        uint32_t *out_rgba = reinterpret_cast<uint32_t *>(rgba8);
        wx_hit *out_hits = hits;
        bool dev_rgba = device_accessible(rgba8);
        bool dev_hits = hits ? device_accessible(hits) : true;
        if (!dev_rgba) {
            if (void *d = pinned_device_alias(rgba8)) {
                out_rgba = static_cast<uint32_t *>(d);
                dev_rgba = true;
            }
        }
        if (!dev_hits) {
            if (void *d = pinned_device_alias(hits)) {
                out_hits = static_cast<wx_hit *>(d);
                dev_hits = true;
            }
        }
        const size_t npix = (size_t)width * height;
        if (!dev_rgba || !dev_hits) {
            const size_t need = npix * 4 + (hits ? npix * sizeof(wx_hit) + 256 : 0);
            if (need > ctx->stage_bytes) {
                if (ctx->stage) {
                    WX_CUDA(ctx, cudaStreamSynchronize(st));
                    cudaFree(ctx->stage);
                }
                ctx->stage = nullptr;
                ctx->stage_bytes = 0;
                WX_CUDA(ctx, wx::dev_alloc(&ctx->stage, need));
                ctx->stage_bytes = need;
            }
            char *b = static_cast<char *>(ctx->stage);
            if (!dev_rgba) out_rgba = reinterpret_cast<uint32_t *>(b);
            if (hits && !dev_hits) out_hits = reinterpret_cast<wx_hit *>(b + ((npix * 4 + 255) & ~(size_t)255));
        }
        const wxk::Job job = make_job(grid, *state, width, height, out_rgba, out_hits, 0, ctx->tuning);
        if (ctx->tuning.kernel == 1) {
            PixelOutputs cur{ctx->device, st, {0, 0}, {0, 0}};
            cur.lo[0] = reinterpret_cast<uintptr_t>(out_rgba);
            cur.hi[0] = cur.lo[0] + npix * 4;
            if (hits) {
                cur.lo[1] = reinterpret_cast<uintptr_t>(out_hits);
                cur.hi[1] = cur.lo[1] + npix * sizeof(wx_hit);
            }
            const cudaError_t e = launch_pixel_tracked(job, ctx->tuning, ctx->num_sms, cur);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "wxk::launch_pixel");
        } else {
            wxk::enter_launch(ctx->device, st, job.tiles);
            WX_CUDA(ctx, wxk::launch_persistent(job, ctx->take_counter(), ctx->tuning, ctx->num_sms, st));
        }
        // Copy back only the dispatched region; the rest of a host buffer is untouched.
        if (!dev_rgba)
            WX_CUDA(ctx, cudaMemcpy2DAsync(rgba8, (size_t)width * 4, out_rgba, (size_t)width * 4, (size_t)tiles_x * 32,
                                           (size_t)tiles_y * 4, cudaMemcpyDeviceToHost, st));
        if (hits && !dev_hits)
            WX_CUDA(ctx, cudaMemcpy2DAsync(hits, (size_t)width * sizeof(wx_hit), out_hits, (size_t)width * sizeof(wx_hit),
                                           (size_t)tiles_x * 8 * sizeof(wx_hit), (size_t)tiles_y * 4,
                                           cudaMemcpyDeviceToHost, st));
        return WX_OK;
    });
}

// ---- batched rendering: many frames of several grids in one persistent launch ----
static int build_jobs(wx_ctx *ctx, const wx_frame *frames, uint32_t n, std::vector<wxk::Job> &jobs,
                      wxk::GridTable &tab, uint32_t *total_tiles, uint64_t *rays) {
    jobs.clear();
    tab.n = 0;
    uint64_t tiles = 0, r = 0;
    for (uint32_t i = 0; i < n; i++) {
        const wx_frame &f = frames[i];
        if (!f.grid || !f.rgba8) return fail(ctx, WX_ERR_INVALID, "wx_frame: null grid or rgba8");
        if (((uintptr_t)f.rgba8 & 3) || ((uintptr_t)f.hits & 15))
            return fail(ctx, WX_ERR_INVALID, "wx_frame: rgba8 must be 4-byte and hits 16-byte aligned");
        if (f.grid->device != ctx->device) return fail(ctx, WX_ERR_INVALID, "wx_frame: grid is on another device");
        if (!device_accessible(f.rgba8) || (f.hits && !device_accessible(f.hits)))
            return fail(ctx, WX_ERR_INVALID, "wx_frame: batched outputs must be device memory");
        if ((uint64_t)f.width * f.height >= (1ull << 32)) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_frame: too large");
        wxk::Job j = make_job(f.grid, f.state, f.width, f.height, reinterpret_cast<uint32_t *>(f.rgba8), f.hits,
                              (uint32_t)tiles, ctx->tuning);
        if (j.tiles == 0) continue;
        wxk::index_grid(j, tab);
        jobs.push_back(j);
        tiles += j.tiles;
        r += (uint64_t)(f.width & ~7u) * (f.height & ~3u);
        if (tiles >= (1ull << 31)) return fail(ctx, WX_ERR_UNSUPPORTED, "wx_render_batch: more than 2^31 tiles");
    }
    *total_tiles = (uint32_t)tiles;
    *rays = r;
    return WX_OK;
}

int wx_render_batch(wx_ctx *ctx, const wx_frame *frames, uint32_t n, void *stream) {
    return wx::guard("wx_render_batch", [&]() -> int {
        if (!ctx || (n && !frames)) return fail(ctx, WX_ERR_INVALID, "wx_render_batch: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        std::vector<wxk::Job> jobs;
        uint32_t total = 0;
        uint64_t rays = 0;
        wxk::GridTable tab;
        int rc = build_jobs(ctx, frames, n, jobs, tab, &total, &rays);
        if (rc != WX_OK) return rc;
        if (jobs.empty()) return WX_OK;
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        // The pinned staging table is reused: wait for the previous batch's copy.
        WX_CUDA(ctx, cudaEventSynchronize(ctx->jobs_done));
        if (jobs.size() > ctx->jobs_cap) {
            if (ctx->jobs_dev) {
                WX_CUDA(ctx, cudaDeviceSynchronize());
                cudaFree(ctx->jobs_dev);
                cudaFreeHost(ctx->jobs_host);
            }
            ctx->jobs_dev = nullptr;
            ctx->jobs_host = nullptr;
            ctx->jobs_cap = 0;
            const size_t cap = std::max<size_t>(jobs.size(), 256);
            WX_CUDA(ctx, wx::dev_alloc(&ctx->jobs_dev, cap * sizeof(wxk::Job)));
            WX_CUDA(ctx, wx::pinned_alloc(&ctx->jobs_host, cap * sizeof(wxk::Job)));
            ctx->jobs_cap = cap;
        }
        memcpy(ctx->jobs_host, jobs.data(), jobs.size() * sizeof(wxk::Job));
        WX_CUDA(ctx, cudaMemcpyAsync(ctx->jobs_dev, ctx->jobs_host, jobs.size() * sizeof(wxk::Job),
                                     cudaMemcpyHostToDevice, st));
        WX_CUDA(ctx, cudaEventRecord(ctx->jobs_done, st));
        wxk::enter_launch(ctx->device, st, total);
        WX_CUDA(ctx, wxk::launch_batched(ctx->jobs_dev, (uint32_t)jobs.size(), tab, total, ctx->take_counter(), ctx->tuning,
                                         ctx->num_sms, wxk::all_modes(jobs.data(), jobs.size()), st));
        return WX_OK;
    });
}

int wx_batch_create(wx_ctx *ctx, const wx_frame *frames, uint32_t n, wx_batch **out) {
    return wx::guard("wx_batch_create", [&]() -> int {
        if (!ctx || !out || (n && !frames)) return fail(ctx, WX_ERR_INVALID, "wx_batch_create: null argument");
        WX_CUDA(ctx, cudaSetDevice(ctx->device));
        std::vector<wxk::Job> jobs;
        uint32_t total = 0;
        uint64_t rays = 0;
        wxk::GridTable tab;
        int rc = build_jobs(ctx, frames, n, jobs, tab, &total, &rays);
        if (rc != WX_OK) return rc;
        auto *b = new (std::nothrow) wx_batch();
        if (!b) return fail(ctx, WX_ERR_OOM, "host allocation failed");
        b->ctx = ctx;
        b->njobs = (uint32_t)jobs.size();
        b->total_tiles = total;
        b->rays = rays;
        auto bail = [&](cudaError_t e, const char *what) {
            wx_batch_destroy(b);
            return cuda_fail(ctx, e, what);
        };
        cudaError_t e;
        if ((e = wx::dev_alloc(&b->jobs_dev, std::max<size_t>(jobs.size(), 1) * sizeof(wxk::Job))) != cudaSuccess)
            return bail(e, "cudaMalloc(job table)");
        if (!jobs.empty() &&
            (e = cudaMemcpy(b->jobs_dev, jobs.data(), jobs.size() * sizeof(wxk::Job), cudaMemcpyHostToDevice)) != cudaSuccess)
            return bail(e, "cudaMemcpy(job table)");
        if ((e = wx::dev_alloc(&b->counter, sizeof(uint32_t))) != cudaSuccess) return bail(e, "cudaMalloc(counter)");
        // Capture counter reset + persistent launch into a graph, replayed by wx_batch_launch.
        cudaStream_t cs;
        if ((e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) != cudaSuccess) return bail(e, "cudaStreamCreate");
        if ((e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) {
            cudaStreamDestroy(cs);
            return bail(e, "cudaStreamBeginCapture");
        }
        cudaError_t le = b->njobs ? wxk::launch_batched(b->jobs_dev, b->njobs, tab, total, b->counter, ctx->tuning,
                                                        ctx->num_sms, wxk::all_modes(jobs.data(), jobs.size()), cs)
                                  : cudaMemsetAsync(b->counter, 0, sizeof(uint32_t), cs);
        e = cudaStreamEndCapture(cs, &b->graph);
        cudaStreamDestroy(cs);
        if (le != cudaSuccess) return bail(le, "capture launch_batched");
        if (e != cudaSuccess) return bail(e, "cudaStreamEndCapture");
        if ((e = cudaGraphInstantiate(&b->exec, b->graph, 0)) != cudaSuccess) return bail(e, "cudaGraphInstantiate");
        *out = b;
        return WX_OK;
    });
}

int wx_batch_launch(wx_batch *b, void *stream) {
    return wx::guard("wx_batch_launch", [&]() -> int {
        if (!b) return WX_ERR_INVALID;
        WX_CUDA(b->ctx, cudaSetDevice(b->ctx->device));
        wxk::enter_launch(b->ctx->device, static_cast<cudaStream_t>(stream), b->total_tiles);
        WX_CUDA(b->ctx, cudaGraphLaunch(b->exec, static_cast<cudaStream_t>(stream)));
        return WX_OK;
    });
}

int wx_batch_info(const wx_batch *b, uint32_t *frames, uint32_t *tiles, uint64_t *rays) {
    return wx::guard("wx_batch_info", [&]() -> int {
        if (!b) return WX_ERR_INVALID;
        if (frames) *frames = b->njobs;
        if (tiles) *tiles = b->total_tiles;
        if (rays) *rays = b->rays;
        return WX_OK;
    });
}

int wx_batch_destroy(wx_batch *b) {
    return wx::guard("wx_batch_destroy", [&]() -> int {
        if (!b) return WX_OK;
        cudaSetDevice(b->ctx->device);
        if (b->exec) cudaGraphExecDestroy(b->exec);
        if (b->graph) cudaGraphDestroy(b->graph);
        if (b->jobs_dev) cudaFree(b->jobs_dev);
        if (b->counter) cudaFree(b->counter);
        delete b;
        return WX_OK;
    });
}

}  // extern "C"
