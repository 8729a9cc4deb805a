// rmq_internal.h — launchers shared between the kernel translation units and
// the C ABI implementation.  Host-only declarations (no device code).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "rmq_common.cuh"
#include "rmq_window.cuh"

namespace rmq {

// Names this library's calls on a profiler's timeline (an NVTX range for
// the scope; without an attached tool it costs one pointer check).
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

// Host level-layout rule (reference src/xxx.h:225-243, generalised to rf = 2^rf_log).
Layout plan_layout(uint64_t n, uint64_t t, uint32_t rf_log);

// Build level k+1 from level k for every k in [0, num_levels-1).
// `val_buf`/`idx_buf` are the level buffers (layout.total entries each);
// `idx_buf` may be null (no argmin support).  With `counters` (at least
// tail_counters(lay) zeroed entries, left zeroed by every build, never used
// by two builds at once) the levels above the fused tiles are built inside
// the fused kernel (one launch in all); without, by extra launches.
cudaError_t launch_build(const Layout& lay, const float* d_values, float* val_buf,
                         uint32_t* idx_buf, cudaStream_t s, unsigned* counters = nullptr);
// Arrival counters the single-launch build needs for `lay` (0: none).
uint64_t tail_counters(const Layout& lay);

// Window tables (rmq_window.cuh) of n values into `tables` (the shape's
// bytes, 32-byte aligned).
cudaError_t launch_window_build(const float* d_values, void* tables, uint64_t n, uint32_t form, bool wide,
                                cudaStream_t s);
// Loads the code of every kernel that a build of kFormArgmin with 32-bit
// positions over up to kSmallN values and its queries can launch, on the current
// device.
cudaError_t load_small_window_kernels();

struct QueryArgs {
    Levels lv;
    const uint2* qs;
    uint64_t q;
    float* out_min;      // may be null for argmin queries
    uint32_t* out_idx;   // null for min queries
    WinView win;         // VL: the window tables (lv is CL's)
    bool after_build;    // the build was launched just before, on the same stream
    bool host_buffers;   // queries and results in host memory, over the CPU-GPU link
    bool wide;           // 64-bit positions: win64 / qs64 / out_idx64 are used instead
    WinView64 win64;
    const uint64_t* qs64;
    uint64_t* out_idx64;
    uint32_t* err;       // invalid-query counter or null
    int variant;         // rmq_variant: 1 = CL, 2 = VL, 3 / 4 / 5 = CL without shuffles / a tile per query / atomic combine
    int lanes;           // CL tile width
    uint32_t rf_log;
    const void* persist_base;   // L2 access-policy window (null = none)
    size_t persist_bytes;
    float persist_hit_ratio;
};

cudaError_t launch_query(const QueryArgs& a, cudaStream_t s);
// The window-table queries of launch_query (variants VL and VL_SHORT).
cudaError_t launch_window_query(const QueryArgs& a, cudaStream_t s);

cudaError_t launch_bruteforce(const float* vals, uint32_t n, const uint2* qs, uint32_t q,
                              float* out_min, uint32_t* out_idx, cudaStream_t s);
// Results outside device memory (page-locked host memory passed to a device
// call)?  Null: no.
bool off_device(const void* p);

// Queries per work unit: threads x kBatchLaneQueries of a batched CTA, and of
// a warp of the served kernel.
constexpr uint32_t kBatchLaneQueries = 4;
constexpr uint32_t kServeUnit = 32;

// Query launch over packed work: entry e (an array, or a request's array in
// serving mode) owns queries [q_off[e], q_off[e+1]) of qs, in units of
// threads x kBatchLaneQueries; owner[u] gives the entry of unit u (launch_fill_owner).
struct BatchQueryArgs {
    const float* values;
    const ArrayDesc* descs;
    const uint32_t* owner;
    const uint64_t* unit_off;
    const uint64_t* q_off;
    uint64_t total_units;
    const char* tables;
    const uint2* qs;
    float* out_min;
    uint32_t* out_idx;  // null: minima only
    uint32_t threads;   // CTA size, multiple of 32, <= 512
};

cudaError_t launch_batch_query(const BatchQueryArgs& a, cudaStream_t s);

// Where one served request's queries come from and its results go: device
// staging buffers, or the request's own page-locked host buffers, which the
// kernel reads and writes directly over the CPU-GPU link.  Either result
// pointer may be null.
struct ServeIO {
    const uint2* qs;
    uint32_t* out_idx;
    float* out_min;
};

// The served batch: entry e (a request) answers its q_off[e+1] - q_off[e]
// queries through io[e] and counts its invalid queries in bad[e] (zeroed by
// the caller); units of kServeUnit queries.
struct ServeQueryArgs {
    const float* values;
    const ArrayDesc* descs;
    const uint32_t* owner;
    const uint64_t* unit_off;
    const uint64_t* q_off;
    uint64_t total_units;
    const char* tables;
    const ServeIO* io;
    uint32_t* bad;
    uint32_t threads;  // CTA size, multiple of 32, <= 512
};

cudaError_t launch_serve_query(const ServeQueryArgs& a, cudaStream_t s);
cudaError_t launch_fill_owner(const uint64_t* unit_off, uint32_t num, uint32_t* owner, cudaStream_t s);

// Kernel launch with the handle's L2 access-policy window, when it has one, or,
// after a build without one, scheduled before the build's last kernel ends (for
// kernels that wait for it themselves).
template <typename K, typename... Args>
static cudaError_t launch_with_window(K kernel, uint32_t grid, uint32_t block, const QueryArgs& a,
                                      cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (a.after_build) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    } else if (a.persist_base != nullptr && a.persist_bytes > 0) {
        attr[0].id = cudaLaunchAttributeAccessPolicyWindow;
        attr[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(a.persist_base);
        attr[0].val.accessPolicyWindow.num_bytes = a.persist_bytes;
        attr[0].val.accessPolicyWindow.hitRatio = a.persist_hit_ratio;
        attr[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        attr[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    } else {
        cfg.attrs = nullptr;
        cfg.numAttrs = 0;
    }
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

#if RMQ_DEBUG_BOUNDS
// Violations counted by the checked kernels of the query / batched units
// since the last read (each read clears them).
unsigned int bounds_bad_query();
unsigned int bounds_bad_window();
unsigned int bounds_bad_batch();
#endif

// Number of kernel launches the last launch_build issued (for accounting).
int build_launch_count(const Layout& lay);

}  // namespace rmq
