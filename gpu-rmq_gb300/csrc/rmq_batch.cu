// rmq_batch.cu — batched build and queries over many independent arrays
// (include/rmq_gb300_batch.h).
//
// Packed layout: every array keeps its values where the caller put them
// (d_values + value_offsets[a]); the window tables of all arrays
// (rmq_window.cuh) live in one buffer, array a's at its descriptor's win_off.
//
// Work lists: each build kernel runs one CTA per tile of any array, the query
// kernel one CTA per run of queries of one array.  Build + queries can be
// captured as one CUDA graph.  384 arrays of 2^10 .. 2^20 values, 1.4e8
// queries of lognormal(sqrt(size), 1) lengths, build and queries: 4125 us with
// the block-minimum levels, 1949 us with the tables.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/rmq_gb300_batch.h"
#include "rmq_internal.h"
#include "rmq_window_build.cuh"

namespace rmq {

// The build's work lists: entry u of a list is one tile of one array, owner[u]
// (filled on the device by fill_owner_kernel when the batch is laid out) names
// the array, so a CTA starts with two dependent loads.
struct TileList {
    const uint64_t* off;    // first tile of each array (num_arrays + 1)
    const uint32_t* owner;  // array of each tile
};

__device__ __forceinline__ uint64_t batch_tile(const ArrayDesc* descs, const TileList& l, const float* values,
                                               char* tables, WinOut& w) {
    const uint32_t a = __ldg(l.owner + blockIdx.x);
    w = win_out(descs[a], values, tables);
    return blockIdx.x - __ldg(reinterpret_cast<const unsigned long long*>(l.off) + a);
}

__global__ void __launch_bounds__(kBlockThreads)
batch_block_kernel(const float* __restrict__ values, const ArrayDesc* __restrict__ descs, TileList l, char* tables) {
    WinOut w;
    const uint64_t tile = batch_tile(descs, l, values, tables, w);
    win_block_tile<false>(w, tile);
}

__global__ void __launch_bounds__(kLowThreads)
batch_low_kernel(const ArrayDesc* __restrict__ descs, TileList l, char* tables) {
    __shared__ uint2 sa[kSpan + kHaloLow], sb[kSpan + kHaloLow];
    WinOut w;
    const uint64_t tile = batch_tile(descs, l, nullptr, tables, w);
    win_low_tile<false>(w, tile, sa, sb);
}

__global__ void __launch_bounds__(kMidThreads)
batch_mid_kernel(const ArrayDesc* __restrict__ descs, TileList l, char* tables) {
    __shared__ uint2 sa[kSpan + kHaloMid], sb[(kSpan + kHaloMid) / 2];
    WinOut w;
    const uint64_t tile = batch_tile(descs, l, nullptr, tables, w);
    win_mid_tile(w, tile, sa, sb);
}

__global__ void __launch_bounds__(kMidThreads)
batch_top_kernel(const ArrayDesc* __restrict__ descs, TileList l, char* tables) {
    __shared__ uint2 sa[kTopEntries], sb[kTopEntries / 2];
    WinOut w;
    batch_tile(descs, l, nullptr, tables, w);
    win_top(w, win_mid_log(w), sa, sb);
}

// Work unit of the query kernels: consecutive queries of one array, answered by
// one CTA (of one request, by one warp, in the served form).  unit_owner[u]
// (filled on the device by fill_owner_kernel) names the array; one thread
// unpacks its descriptor into a shared view.
constexpr uint32_t kMaxQueryThreads = 512;

__global__ void fill_owner_kernel(const uint64_t* __restrict__ unit_off, uint32_t* __restrict__ owner) {
    const uint32_t a = blockIdx.x;
    const uint64_t u0 = unit_off[a], u1 = unit_off[a + 1];
    for (uint64_t u = u0 + threadIdx.x; u < u1; u += blockDim.x) owner[u] = a;
}

template <bool ARGMIN>
__global__ void __launch_bounds__(kMaxQueryThreads)
batch_query_kernel(const float* __restrict__ values, const ArrayDesc* __restrict__ descs,
                   const uint32_t* __restrict__ unit_owner, const uint64_t* __restrict__ unit_off,
                   const uint64_t* __restrict__ q_off, const char* __restrict__ tables,
                   const uint2* __restrict__ qs, float* __restrict__ out_min, uint32_t* __restrict__ out_idx) {
    extern __shared__ __align__(16) unsigned char batch_smem[];
    __shared__ WinView view;
    const uint32_t a = __ldg(unit_owner + blockIdx.x);
    if (threadIdx.x == 0) win_load_view(descs[a], values, tables, view);
    const uint32_t cap = blockDim.x * kBatchLaneQueries;
    const uint64_t at = q_off[a] + (blockIdx.x - unit_off[a]) * cap;
    const uint64_t left = q_off[a + 1] - at;
    const WinLists<uint32_t> sm = win_lists<uint32_t>(batch_smem, cap);
    __syncthreads();
    // One instantiation for all arrays.  Those beyond 2^24 entries would have
    // one of their own for short queries, as single handles do: 4 arrays of 2^26,
    // 2^26 queries of lognormal(32, 0.7) 1.82 ms (descending levels 2.86).
    win_block<ARGMIN, false, false, kBatchLaneQueries>(view, sm, blockDim.x, qs + at, left < cap ? uint32_t(left) : cap,
                                                out_min != nullptr ? out_min + at : nullptr,
                                                ARGMIN ? out_idx + at : nullptr);
}

// The same with results outside device memory: a thread per query (a unit is
// gridDim.y blocks), so that a warp writes whole 128-byte lines, which the CPU-GPU link wants.  54,306,557
// queries of 384 arrays, lognormal(32, 0.7), us: 3.62 ms with batch_one_kernel,
// 10.07 with batch_query_kernel; minima only 1.82 and 5.07.
template <bool ARGMIN>
__global__ void __launch_bounds__(kMaxQueryThreads)
batch_one_kernel(const float* __restrict__ values, const ArrayDesc* __restrict__ descs,
                 const uint32_t* __restrict__ unit_owner, const uint64_t* __restrict__ unit_off,
                 const uint64_t* __restrict__ q_off, const char* __restrict__ tables,
                 const uint2* __restrict__ qs, float* __restrict__ out_min, uint32_t* __restrict__ out_idx) {
    __shared__ WinView view;
    const uint32_t a = __ldg(unit_owner + blockIdx.x);
    if (threadIdx.x == 0) win_load_view(descs[a], values, tables, view);
    const uint64_t i = q_off[a] + (blockIdx.x - unit_off[a]) * (blockDim.x * kBatchLaneQueries) + blockDim.x * blockIdx.y +
                       threadIdx.x;
    __syncthreads();
    if (i >= q_off[a + 1]) return;
    const uint2 Q = ld_query(qs + i);
    const bool valid = Q.x <= Q.y && Q.y < view.n;
    WinBest<uint32_t> c{f_nan(), kNoPos, false};
    if (valid) c = win_one<false>(view, Q.x, Q.y);
    if (out_min != nullptr) st_stream(out_min + i, c.v);
    if (ARGMIN) st_stream(out_idx + i, win_place(view, c, valid ? Q.x : kNoPos));
}

// The served batch's kernel: as batch_query_kernel, but every entry (a
// request) reads its queries and writes its results through its own ServeIO
// (staging buffers or the request's page-locked host buffers), and counts
// its invalid queries so the host needs no pass over the results.
__global__ void __launch_bounds__(kMaxQueryThreads)
serve_query_kernel(const float* __restrict__ values, const ArrayDesc* __restrict__ descs,
                   const uint32_t* __restrict__ unit_owner, const uint64_t* __restrict__ unit_off,
                   const uint64_t* __restrict__ q_off, uint64_t total_units, const char* __restrict__ tables,
                   const ServeIO* __restrict__ io, uint32_t* __restrict__ bad) {
    __shared__ WinView views[kMaxQueryThreads / 32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint64_t unit = uint64_t(blockIdx.x) * (blockDim.x >> 5) + warp;
    if (unit >= total_units) return;  // the whole warp leaves
    const uint32_t a = __ldg(unit_owner + unit);
    if (lane == 0) win_load_view(descs[a], values, tables, views[warp]);
    const ServeIO r = io[a];
    const uint64_t at = (unit - unit_off[a]) * kServeUnit + lane;  // local to the request
    const bool in_range = at < q_off[a + 1] - q_off[a];
    uint2 Q = make_uint2(1u, 0u);
    if (in_range) Q = ld_query(r.qs + at);
    __syncwarp();
    const WinView& w = views[warp];
    const bool valid = in_range && Q.x <= Q.y && Q.y < w.n;
    WinBest<uint32_t> c{f_nan(), kNoPos, false};
    if (valid) c = win_one<false>(w, Q.x, Q.y);
    if (in_range) {
        if (r.out_min != nullptr) st_stream(r.out_min + at, c.v);
        if (r.out_idx != nullptr) st_stream(r.out_idx + at, win_place(w, c, valid ? Q.x : kNoPos));
    }
    const uint32_t nbad = __popc(__ballot_sync(0xffffffffu, in_range && !valid));
    if (lane == 0 && nbad != 0) atomicAdd(bad + a, nbad);
}

cudaError_t launch_serve_query(const ServeQueryArgs& a, cudaStream_t s) {
    if (a.total_units == 0) return cudaSuccess;
    const uint32_t warps = a.threads / 32u;
    const uint32_t grid = uint32_t((a.total_units + warps - 1) / warps);
    serve_query_kernel<<<grid, a.threads, 0, s>>>(a.values, a.descs, a.owner, a.unit_off, a.q_off, a.total_units,
                                                  a.tables, a.io, a.bad);
    return cudaGetLastError();
}

cudaError_t launch_fill_owner(const uint64_t* unit_off, uint32_t num, uint32_t* owner, cudaStream_t s) {
    if (num == 0) return cudaSuccess;
    fill_owner_kernel<<<num, 256, 0, s>>>(unit_off, owner);
    return cudaGetLastError();
}

#if RMQ_DEBUG_BOUNDS
RMQ_BOUNDS_COUNTER_READER(bounds_bad_batch)
#endif

cudaError_t launch_batch_query(const BatchQueryArgs& a, cudaStream_t s) {
    if (a.total_units == 0) return cudaSuccess;
    const uint32_t grid = uint32_t(a.total_units), smem = win_lists_bytes<uint32_t>(a.threads * kBatchLaneQueries);
    if (off_device(a.out_min) || off_device(a.out_idx)) {
        (a.out_idx != nullptr ? batch_one_kernel<true> : batch_one_kernel<false>)<<<dim3(grid, kBatchLaneQueries), a.threads, 0, s>>>(
            a.values, a.descs, a.owner, a.unit_off, a.q_off, a.tables, a.qs, a.out_min, a.out_idx);
        return cudaGetLastError();
    }
    if (a.out_idx != nullptr) {
        batch_query_kernel<true><<<grid, a.threads, smem, s>>>(a.values, a.descs, a.owner, a.unit_off, a.q_off,
                                                            a.tables, a.qs, a.out_min, a.out_idx);
    } else {
        batch_query_kernel<false><<<grid, a.threads, smem, s>>>(a.values, a.descs, a.owner, a.unit_off, a.q_off,
                                                             a.tables, a.qs, a.out_min, nullptr);
    }
    return cudaGetLastError();
}

}  // namespace rmq

using rmq::ArrayDesc;

// One build kernel's tiles: the first of each array and the array of each.
struct TileWork {
    uint64_t* d_off = nullptr;
    uint32_t* d_owner = nullptr;
    uint64_t total = 0;
};

struct rmq_batch {
    const float* d_values = nullptr;
    uint32_t num_arrays = 0;
    std::vector<uint64_t> val_off, sizes;
    uint64_t t = 64;        // scan threshold of the largest size class (the batch-wide t when uniform)
    uint64_t tc[3] = {64, 64, 64};  // scan threshold per size class (rmq_batch_info.class_upper)
    uint32_t qblock = 128;  // threads per CTA of the query kernel (untuned default)
    int with_index = 1;
    int device = 0;
    // tables, and after them the descriptors and lists below (one allocation)
    char* tables = nullptr;
    uint64_t lvl_capacity = 0;  // entries of the deepest plan that set_tuning accepts (nothing is built of a plan)
    uint64_t table_bytes = 0;   // of all arrays
    uint32_t max_levels = 1;
    ArrayDesc* d_descs = nullptr;
    TileWork work[4];  // tiles of the block, low, mid and top kernels
    // queries
    std::vector<uint64_t> q_off;
    uint64_t* d_q_off = nullptr;
    uint64_t* d_blk_off = nullptr;  // work-unit offsets per array
    uint32_t* d_owner = nullptr;    // array of every work unit
    uint64_t owner_capacity = 0;
    uint64_t total_blocks = 0;      // work units
    const uint32_t* d_lr = nullptr;
    uint32_t* d_argmin = nullptr;
    float* d_min = nullptr;
    bool queries_set = false;
    std::vector<ArrayDesc> h_descs;  // host copy of the descriptors (per-array loop)
    // graph + timing
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    bool build_timed = false;
    float build_ms = 0.f, query_ms = 0.f;

    // Many arrays' tables take no more than levels did, so no blocks of eight.
    uint32_t form() const { return with_index ? rmq::kFormArgmin : rmq::kFormMin; }
};

namespace {

constexpr uint64_t kBatchDefaultT = 64;
constexpr uint64_t kTuneT[] = {16, 32, 64, 256, 1024};
// Size classes of the per-class thresholds: arrays below 2^14 entries, below
// 2^18, and the rest.
constexpr int kClasses = 3;
constexpr uint64_t kClassUpper[kClasses] = {uint64_t(1) << 14, uint64_t(1) << 18, ~uint64_t(0)};

int size_class(uint64_t n) {
    int c = 0;
    while (c + 1 < kClasses && n >= kClassUpper[c]) ++c;
    return c;
}
constexpr uint32_t kTuneBlock[] = {64, 128, 256, 512};  // threads per CTA of the query kernel

int status_of(cudaError_t e) {
    if (e == cudaSuccess) return RMQ_OK;
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? RMQ_ERR_OOM : RMQ_ERR_CUDA;
}

uint64_t layout_entries(uint64_t n, uint64_t t) {
    const rmq::Layout lay = rmq::plan_layout(n, t, 3);
    return lay.num_levels > 1 ? lay.total : 0;
}

void drop_graph(rmq_batch* b) {
    if (b->graph != nullptr) {
        cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    }
}

// Plans every array's levels with its size class's threshold tc[class] (the
// plan that rmq_batch_info reports; the tables do not depend on it).
int plan(rmq_batch* b, const uint64_t (&tc)[kClasses]) {
    uint64_t base = 0;
    uint32_t max_levels = 1;
    for (uint32_t a = 0; a < b->num_arrays; ++a) {
        const rmq::Layout lay = rmq::plan_layout(b->sizes[a], tc[size_class(b->sizes[a])], 3);
        if (lay.num_levels > 1) base += lay.total;
        max_levels = std::max(max_levels, lay.num_levels);
    }
    if (base > b->lvl_capacity) return RMQ_ERR_UNSUPPORTED;
    for (int c = 0; c < kClasses; ++c) b->tc[c] = tc[c];
    b->t = tc[kClasses - 1];
    b->max_levels = max_levels;
    return RMQ_OK;
}

// Lays out every array's tables, allocates them and uploads the descriptors
// and the build kernels' work lists (once, at creation).
int lay_out(rmq_batch* b, cudaStream_t s) {
    std::vector<uint64_t> off[4];
    for (auto& o : off) o.assign(b->num_arrays + 1, 0);
    b->h_descs.resize(b->num_arrays);
    uint64_t bytes = 0;
    for (uint32_t a = 0; a < b->num_arrays; ++a) {
        const rmq::WinShape w = rmq::win_shape(b->sizes[a], b->form());
        b->h_descs[a] = rmq::win_desc(b->val_off[a], bytes, w);
        bytes += w.bytes;
        const rmq::WinTiles t = rmq::win_tiles(w);
        const uint64_t tiles[4] = {t.block, t.low, t.mid, t.top};
        for (int i = 0; i < 4; ++i) off[i][a + 1] = off[i][a] + tiles[i];
    }
    b->table_bytes = bytes;
    // the tables, then the descriptors and the lists: one allocation, of some
    // 50 us, and one release (create and destroy of 384 arrays: 341 us;
    // the levels with an allocation each: 506)
    uint64_t at = (bytes + 255u) & ~uint64_t(255);
    const auto take = [&](uint64_t size) {
        const uint64_t p = at;
        at += (size + 255u) & ~uint64_t(255);
        return p;
    };
    const uint64_t off_bytes = sizeof(uint64_t) * (b->num_arrays + 1), descs_at = take(sizeof(ArrayDesc) * b->num_arrays),
                   q_off_at = take(off_bytes), blk_off_at = take(off_bytes);
    uint64_t off_at[4] = {}, owner_at[4] = {};
    for (int i = 0; i < 4; ++i) {
        TileWork& w = b->work[i];
        w.total = off[i][b->num_arrays];
        if (w.total == 0) continue;
        off_at[i] = take(off_bytes);
        owner_at[i] = take(sizeof(uint32_t) * w.total);
    }
    cudaError_t e = cudaMalloc(&b->tables, at);
    if (e != cudaSuccess) return status_of(e);
    for (const TileWork& w : b->work)
        if (w.total > 0x7FFFFFFFull) return RMQ_ERR_UNSUPPORTED;  // one CTA per tile
    b->d_descs = reinterpret_cast<ArrayDesc*>(b->tables + descs_at);
    b->d_q_off = reinterpret_cast<uint64_t*>(b->tables + q_off_at);
    b->d_blk_off = reinterpret_cast<uint64_t*>(b->tables + blk_off_at);
    e = cudaMemcpyAsync(b->d_descs, b->h_descs.data(), sizeof(ArrayDesc) * b->num_arrays, cudaMemcpyHostToDevice, s);
    for (int i = 0; i < 4 && e == cudaSuccess; ++i) {
        TileWork& w = b->work[i];
        if (w.total == 0) continue;
        w.d_off = reinterpret_cast<uint64_t*>(b->tables + off_at[i]);
        w.d_owner = reinterpret_cast<uint32_t*>(b->tables + owner_at[i]);
        e = cudaMemcpyAsync(w.d_off, off[i].data(), off_bytes, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = rmq::launch_fill_owner(w.d_off, b->num_arrays, w.d_owner, s);
    }
    const cudaError_t es = cudaStreamSynchronize(s);  // the host lists die here
    return status_of(e != cudaSuccess ? e : es);
}

int plan(rmq_batch* b, uint64_t t) {
    const uint64_t tc[kClasses] = {t, t, t};
    return plan(b, tc);
}

int upload_blocks(rmq_batch* b, cudaStream_t s) {
    std::vector<uint64_t> blk(b->num_arrays + 1, 0);
    for (uint32_t a = 0; a < b->num_arrays; ++a) {
        const uint64_t qa = b->q_off[a + 1] - b->q_off[a];
        const uint64_t unit = uint64_t(b->qblock) * rmq::kBatchLaneQueries;
        blk[a + 1] = blk[a] + (qa + unit - 1) / unit;
    }
    const uint64_t units = blk[b->num_arrays];
    if (units > 0x7FFFFFFFull) return RMQ_ERR_UNSUPPORTED;  // one CTA per unit
    cudaError_t e = cudaSuccess;
    if (units > b->owner_capacity) {
        if (b->d_owner != nullptr) cudaFree(b->d_owner);
        b->d_owner = nullptr;
        b->owner_capacity = 0;
        e = cudaMalloc(&b->d_owner, sizeof(uint32_t) * units);
        if (e != cudaSuccess) return status_of(e);
        b->owner_capacity = units;
    }
    e = cudaMemcpyAsync(b->d_blk_off, blk.data(), sizeof(uint64_t) * (b->num_arrays + 1),
                        cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && units > 0) e = rmq::launch_fill_owner(b->d_blk_off, b->num_arrays, b->d_owner, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return status_of(e);
    b->total_blocks = units;
    drop_graph(b);
    return RMQ_OK;
}

cudaError_t enqueue_build(rmq_batch* b, cudaStream_t s) {
    const TileWork* w = b->work;
    const auto list = [&](int i) { return rmq::TileList{w[i].d_off, w[i].d_owner}; };
    rmq::batch_block_kernel<<<uint32_t(w[0].total), rmq::kBlockThreads, 0, s>>>(b->d_values, b->d_descs, list(0),
                                                                               b->tables);
    if (w[1].total > 0) rmq::batch_low_kernel<<<uint32_t(w[1].total), rmq::kLowThreads, 0, s>>>(b->d_descs, list(1), b->tables);
    if (w[2].total > 0) rmq::batch_mid_kernel<<<uint32_t(w[2].total), rmq::kMidThreads, 0, s>>>(b->d_descs, list(2), b->tables);
    if (w[3].total > 0) rmq::batch_top_kernel<<<uint32_t(w[3].total), rmq::kMidThreads, 0, s>>>(b->d_descs, list(3), b->tables);
    return cudaGetLastError();
}

cudaError_t enqueue_query(rmq_batch* b, cudaStream_t s) {
    rmq::BatchQueryArgs a;
    a.values = b->d_values;
    a.descs = b->d_descs;
    a.owner = b->d_owner;
    a.unit_off = b->d_blk_off;
    a.q_off = b->d_q_off;
    a.total_units = b->total_blocks;
    a.tables = b->tables;
    a.qs = reinterpret_cast<const uint2*>(b->d_lr);
    a.out_min = b->d_min;
    a.out_idx = b->d_argmin;
    a.threads = b->qblock;
    return rmq::launch_batch_query(a, s);
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) cudaSetDevice(dev);
        else prev = -1;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

}  // namespace

extern "C" {

int rmq_batch_create(const float* d_values, const uint64_t* value_offsets, const uint64_t* sizes,
                     uint32_t num_arrays, const rmq_config* cfg, rmq_stream_t stream, rmq_batch** out) {
    if (out == nullptr) return RMQ_ERR_ARG;
    *out = nullptr;
    if (d_values == nullptr || value_offsets == nullptr || sizes == nullptr || num_arrays == 0) return RMQ_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(d_values) & 31u) != 0) return RMQ_ERR_ARG;
    for (uint32_t a = 0; a < num_arrays; ++a) {
        if (sizes[a] == 0 || (value_offsets[a] & 7u) != 0) return RMQ_ERR_ARG;
        if (sizes[a] > 0xFFFFFF00ull) return RMQ_ERR_UNSUPPORTED;
    }
    const uint64_t t = (cfg != nullptr && cfg->scan_threshold != 0) ? cfg->scan_threshold : kBatchDefaultT;
    if (t < 8) return RMQ_ERR_ARG;  // VL precondition t >= rf (src/xxx.h:938)
    if (cfg != nullptr && cfg->rf_log != 0 && cfg->rf_log != 3) return RMQ_ERR_UNSUPPORTED;

    rmq_batch* b = new (std::nothrow) rmq_batch();
    if (b == nullptr) return RMQ_ERR_OOM;
    if (cudaGetDevice(&b->device) != cudaSuccess) {
        delete b;
        return RMQ_ERR_CUDA;
    }
    b->d_values = d_values;
    b->num_arrays = num_arrays;
    b->val_off.assign(value_offsets, value_offsets + num_arrays);
    b->sizes.assign(sizes, sizes + num_arrays);
    b->with_index = cfg != nullptr ? (cfg->with_index != 0) : 1;
    // the deepest layout among the user's t and the tuner's candidates
    uint64_t cap = 0;
    for (uint32_t a = 0; a < num_arrays; ++a) {
        uint64_t m = layout_entries(sizes[a], t);
        for (uint64_t ct : kTuneT) m = std::max(m, layout_entries(sizes[a], ct));
        cap += m;
    }
    b->lvl_capacity = cap;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev1);
    int st = status_of(e);
    if (st == RMQ_OK) st = plan(b, t);
    if (st == RMQ_OK) st = lay_out(b, s);
    if (st != RMQ_OK) {
        rmq_batch_destroy(b);
        return st;
    }
    *out = b;
    return RMQ_OK;
}

int rmq_batch_set_queries(rmq_batch* b, const uint32_t* d_lr, const uint64_t* query_offsets,
                          uint32_t* d_argmin, float* d_min, rmq_stream_t stream) {
    if (b == nullptr || query_offsets == nullptr) return RMQ_ERR_ARG;
    if (d_argmin == nullptr && d_min == nullptr) return RMQ_ERR_ARG;
    if (d_argmin != nullptr && !b->with_index) return RMQ_ERR_NO_INDEX;
    if (query_offsets[0] != 0) return RMQ_ERR_ARG;
    for (uint32_t a = 0; a < b->num_arrays; ++a)
        if (query_offsets[a + 1] < query_offsets[a]) return RMQ_ERR_ARG;
    const uint64_t total = query_offsets[b->num_arrays];
    if (total > 0 && (d_lr == nullptr || (reinterpret_cast<uintptr_t>(d_lr) & 7u) != 0)) return RMQ_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(d_argmin) & 3u) != 0 || (reinterpret_cast<uintptr_t>(d_min) & 3u) != 0)
        return RMQ_ERR_ARG;  // results are stored element by element
    DeviceGuard guard(b->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    b->q_off.assign(query_offsets, query_offsets + b->num_arrays + 1);
    cudaError_t e = cudaMemcpyAsync(b->d_q_off, b->q_off.data(), sizeof(uint64_t) * (b->num_arrays + 1),
                                    cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return status_of(e);
    b->d_lr = d_lr;
    b->d_argmin = d_argmin;
    b->d_min = d_min;
    const int st = upload_blocks(b, s);
    b->queries_set = st == RMQ_OK;
    return st;
}

int rmq_batch_build(rmq_batch* b, rmq_stream_t stream) {
    rmq::NvtxRange nvtx_range("rmq_batch_build");
    if (b == nullptr) return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    cudaError_t e = cudaEventRecord(b->ev0, s);
    if (e == cudaSuccess) e = enqueue_build(b, s);
    if (e == cudaSuccess) e = cudaEventRecord(b->ev1, s);
    b->build_timed = e == cudaSuccess;
    return status_of(e);
}

int rmq_batch_query(rmq_batch* b, rmq_stream_t stream) {
    rmq::NvtxRange nvtx_range("rmq_batch_query");
    if (b == nullptr || !b->queries_set) return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    return status_of(enqueue_query(b, reinterpret_cast<cudaStream_t>(stream)));
}

int rmq_batch_run(rmq_batch* b, rmq_stream_t stream) {
    rmq::NvtxRange nvtx_range("rmq_batch_run");
    if (b == nullptr || !b->queries_set) return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (b->graph == nullptr) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return status_of(e);
        cudaError_t e1 = enqueue_build(b, b->cap_stream);
        cudaError_t e2 = e1 == cudaSuccess ? enqueue_query(b, b->cap_stream) : e1;
        e = cudaStreamEndCapture(b->cap_stream, &g);
        if (e2 != cudaSuccess || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return status_of(e2 != cudaSuccess ? e2 : e);
        }
        e = cudaGraphInstantiate(&b->graph, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            b->graph = nullptr;
            return status_of(e);
        }
    }
    return status_of(cudaGraphLaunch(b->graph, s));
}

int rmq_batch_run_per_array(rmq_batch* b, rmq_stream_t stream) {
    rmq::NvtxRange nvtx_range("rmq_batch_run_per_array");
    if (b == nullptr || !b->queries_set) return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    for (uint32_t a = 0; a < b->num_arrays; ++a) {
        const ArrayDesc& d = b->h_descs[a];
        const float* vals = b->d_values + d.val_off;
        char* tables = b->tables + d.win_off;
        cudaError_t e = rmq::launch_window_build(vals, tables, b->sizes[a], b->form(), false, s);
        if (e != cudaSuccess) return status_of(e);
        const uint64_t q0 = b->q_off[a], q = b->q_off[a + 1] - q0;
        if (q == 0) continue;
        rmq::QueryArgs qa;
        std::memset(&qa, 0, sizeof(qa));
        qa.win = rmq::win_view<uint32_t>(vals, tables, b->sizes[a], b->form());
        qa.qs = reinterpret_cast<const uint2*>(b->d_lr) + q0;
        qa.q = q;
        qa.out_min = b->d_min != nullptr ? b->d_min + q0 : nullptr;
        qa.out_idx = b->d_argmin != nullptr ? b->d_argmin + q0 : nullptr;
        qa.after_build = true;
        qa.variant = RMQ_VARIANT_VL;
        qa.rf_log = 3;
        e = rmq::launch_query(qa, s);
        if (e != cudaSuccess) return status_of(e);
    }
    return RMQ_OK;
}

// Device time of one query pass with the current plan and CTA size (one
// warm-up launch, then the mean of `reps` timed launches).
int time_query(rmq_batch* b, cudaStream_t s, int reps, float* ms_out) {
    cudaError_t e = enqueue_query(b, s);  // warm-up
    if (e == cudaSuccess) e = cudaEventRecord(b->ev0, s);
    for (int rep = 0; rep < reps && e == cudaSuccess; ++rep) e = enqueue_query(b, s);
    if (e == cudaSuccess) e = cudaEventRecord(b->ev1, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(b->ev1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, b->ev0, b->ev1);
    if (e != cudaSuccess) return status_of(e);
    *ms_out = ms / float(reps);
    return RMQ_OK;
}

int rmq_batch_autotune(rmq_batch* b, rmq_stream_t stream, rmq_batch_info* info) {
    rmq::NvtxRange nvtx_range("rmq_batch_autotune");
    if (b == nullptr || !b->queries_set) return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint64_t tc[kClasses];
    for (int c = 0; c < kClasses; ++c) {
        const uint64_t* end = kTuneT + sizeof(kTuneT) / sizeof(kTuneT[0]);
        tc[c] = std::find(kTuneT, end, b->tc[c]) != end ? b->tc[c] : kBatchDefaultT;
    }
    int st = plan(b, tc);
    if (st != RMQ_OK) return st;
    cudaError_t e = enqueue_build(b, s);
    if (e != cudaSuccess) return status_of(e);
    float best = -1.f;
    uint32_t best_block = b->qblock;
    for (uint32_t qb : kTuneBlock) {
        b->qblock = qb;
        st = upload_blocks(b, s);
        if (st != RMQ_OK) return st;
        float ms = 0.f;
        st = time_query(b, s, 2, &ms);
        if (st != RMQ_OK) return st;
        if (best < 0.f || ms < best) {
            best = ms;
            best_block = qb;
        }
    }
    b->qblock = best_block;
    st = upload_blocks(b, s);
    if (st != RMQ_OK) return st;
    b->build_timed = false;
    b->query_ms = best;
    return info != nullptr ? rmq_batch_get_info(b, info) : RMQ_OK;
}

int rmq_batch_set_tuning(rmq_batch* b, uint64_t scan_threshold, uint32_t query_block, rmq_stream_t stream) {
    if (b == nullptr || scan_threshold < 8 || query_block < 32 || query_block > rmq::kMaxQueryThreads ||
        query_block % 32 != 0)
        return RMQ_ERR_ARG;
    DeviceGuard guard(b->device);
    int st = plan(b, scan_threshold);  // RMQ_ERR_UNSUPPORTED when the levels would not fit
    if (st != RMQ_OK) return st;
    b->qblock = query_block;
    drop_graph(b);
    if (b->queries_set) {
        st = upload_blocks(b, reinterpret_cast<cudaStream_t>(stream));
        if (st != RMQ_OK) return st;
    }
    b->build_timed = false;
    return RMQ_OK;
}

int rmq_batch_set_class_tuning(rmq_batch* b, const uint64_t* class_thresholds, uint32_t query_block,
                               rmq_stream_t stream) {
    if (b == nullptr || class_thresholds == nullptr || query_block < 32 || query_block > rmq::kMaxQueryThreads ||
        query_block % 32 != 0)
        return RMQ_ERR_ARG;
    uint64_t tc[kClasses];
    for (int c = 0; c < kClasses; ++c) {
        if (class_thresholds[c] < 8) return RMQ_ERR_ARG;
        tc[c] = class_thresholds[c];
    }
    DeviceGuard guard(b->device);
    int st = plan(b, tc);  // RMQ_ERR_UNSUPPORTED when the levels would not fit
    if (st != RMQ_OK) return st;
    b->qblock = query_block;
    drop_graph(b);
    if (b->queries_set) {
        st = upload_blocks(b, reinterpret_cast<cudaStream_t>(stream));
        if (st != RMQ_OK) return st;
    }
    b->build_timed = false;
    return RMQ_OK;
}

int rmq_batch_get_info(const rmq_batch* bc, rmq_batch_info* info) {
    if (bc == nullptr || info == nullptr) return RMQ_ERR_ARG;
    rmq_batch* b = const_cast<rmq_batch*>(bc);
    std::memset(info, 0, sizeof(*info));
    info->num_arrays = b->num_arrays;
    for (uint64_t n : b->sizes) info->total_values += n;
    info->level_bytes = b->table_bytes;
    info->scan_threshold = b->t;
    info->query_block = b->qblock;
    info->max_levels = b->max_levels;
    info->total_queries = b->queries_set ? b->q_off[b->num_arrays] : 0;
    if (b->build_timed) {
        DeviceGuard guard(b->device);
        if (cudaEventSynchronize(b->ev1) == cudaSuccess) cudaEventElapsedTime(&b->build_ms, b->ev0, b->ev1);
        cudaGetLastError();
    }
    info->build_ms = b->build_ms;
    info->query_ms = b->query_ms;
    for (int c = 0; c < kClasses; ++c) {
        info->class_threshold[c] = b->tc[c];
        info->class_upper[c] = kClassUpper[c];
    }
    return RMQ_OK;
}

void rmq_batch_destroy(rmq_batch* b) {
    if (b == nullptr) return;
    {
        DeviceGuard guard(b->device);
        drop_graph(b);
        if (b->cap_stream) cudaStreamDestroy(b->cap_stream);
        if (b->ev0) cudaEventDestroy(b->ev0);
        if (b->ev1) cudaEventDestroy(b->ev1);
        cudaFree(b->tables);
        cudaFree(b->d_owner);
        cudaGetLastError();
    }
    delete b;
}

}  // extern "C"
