// rmq_window.cu — the single-array kernels of the window tables: build
// (rmq_window_build.cuh) and queries (rmq_window.cuh).
//
// The build kernels after the first are launched with programmatic stream
// serialization, so each is scheduled before its predecessor ends and no
// launch gap separates them.
#include "rmq_internal.h"
#include "rmq_window_build.cuh"

namespace rmq {

__device__ __forceinline__ void wait_previous_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next_grid() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <bool LARGE>
__global__ void __launch_bounds__(kBlockThreads) win_block_kernel(WinOut w) {
    allow_next_grid();
    win_block_tile<LARGE>(w, blockIdx.x);
}

template <bool EIGHT>
__global__ void __launch_bounds__(kLowThreads) win_low_kernel(WinOut w) {
    __shared__ uint2 sa[kSpan + kHaloLow], sb[kSpan + kHaloLow];
    wait_previous_grid();
    allow_next_grid();
    win_low_tile<EIGHT>(w, blockIdx.x, sa, sb);
}

__global__ void __launch_bounds__(kMidThreads) win_mid_kernel(WinOut w) {
    __shared__ uint2 sa[kSpan + kHaloMid], sb[(kSpan + kHaloMid) / 2];
    wait_previous_grid();
    allow_next_grid();
    win_mid_tile(w, blockIdx.x, sa, sb);
}

__global__ void __launch_bounds__(kMidThreads) win_top_kernel(WinOut w, uint32_t k0) {
    __shared__ uint2 sa[kTopEntries], sb[kTopEntries / 2];
    wait_previous_grid();
    win_top(w, k0, sa, sb);
}

template <uint32_t HALO>
__global__ void __launch_bounds__(win_small_threads<HALO>()) win_small_kernel(WinOut w) {
    __shared__ WinSmallShared<HALO> sm;
    allow_next_grid();
    win_small_tile<HALO>(w, blockIdx.x, sm);
}

// Launch with programmatic stream serialization (the kernel waits for its
// predecessor in wait_previous_grid).
template <typename... KArgs, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(KArgs...), uint32_t grid, uint32_t block, cudaStream_t s,
                                    Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

cudaError_t launch_window_build(const float* d_values, void* tables, uint64_t n, uint32_t form, bool wide,
                                cudaStream_t s) {
    const WinShape sh = win_shape(n, form);
    WinOut w;
    char* b = static_cast<char*>(tables);
    w.a = d_values;
    w.v1 = reinterpret_cast<float*>(b);
    w.j1 = reinterpret_cast<uint8_t*>(b + sh.j1_off);
    w.t = reinterpret_cast<uint2*>(b + sh.t_off);
    w.n = n;
    w.S = sh.S;
    w.cb = sh.cb;
    w.blk = sh.blk;
    w.gb = sh.gb;
    w.c = sh.c;
    w.first = sh.first;
    w.kmax = sh.kmax;
    w.wide = wide;
    if (n <= kSmallN && sh.gb == 5u) {
        const bool brief = n <= kShortHaloN && (sh.S <= kShortHalo || sh.S > kLongHalo);
        const uint64_t halo = brief ? kShortHalo : kLongHalo;
        const uint32_t tiles = uint32_t((sh.S + halo - 1) / halo), k0 = sh.gb + (brief ? 7u : 9u);
        if (brief) win_small_kernel<kShortHalo><<<tiles, win_small_threads<kShortHalo>(), 0, s>>>(w);
        else win_small_kernel<kLongHalo><<<tiles, win_small_threads<kLongHalo>(), 0, s>>>(w);
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess || tiles == 1 || sh.kmax <= k0 ? e
                                                               : launch_dependent(win_top_kernel, 1u, kMidThreads, s, w, k0);
    }
    const WinTiles t = win_tiles(sh);
    (sh.blk > 4u ? win_block_kernel<true> : win_block_kernel<false>)<<<uint32_t(t.block), kBlockThreads, 0, s>>>(w);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && t.low > 0) e = launch_dependent(sh.gb - sh.blk == 3u ? win_low_kernel<true> : win_low_kernel<false>,
                                                        uint32_t(t.low), kLowThreads, s, w);
    if (e == cudaSuccess && t.mid > 0) e = launch_dependent(win_mid_kernel, uint32_t(t.mid), kMidThreads, s, w);
    if (e == cudaSuccess && t.top > 0) e = launch_dependent(win_top_kernel, uint32_t(t.top), kMidThreads, s, w, win_mid_log(sh));
    return e;
}

// ---------------------------------------------------------------------------
// Queries.
//
// win_query_kernel (win_block: four queries per thread in a pass, the harder
// ones listed in shared memory and answered by full warps) for launches that
// fill the GPU, win_one_kernel (one query per thread, no lists, no barriers)
// for the others.  n = 2^20, device time of one launch in us, the two kernels
// and the block-minimum descent they replace:
//
//   queries                2^18               2^20               2^22
//   uniform lengths      7.8   8.9  14.2   14.6  23.1  38.7   37.4  119  138
//   lognormal(2^13, 1)   8.7   9.0  13.0   16.3  23.9  34.1   41.1  106  120
//   lognormal(32, 0.7)  10.9   9.2   8.6   25.2  24.6  23.1   81.6   80   83
//   all three mixed     11.4  13.1  14.3   24.0  36.5  38.9   66.1        141
//
// The lengths are not known before the launch: win_one_kernel answers up to
// 2^18 queries, where it is the faster one only for short lengths but never
// slower than the descent by more than a few percent.  Results in host memory
// always come from it: its warps write whole 128-byte lines, which the
// CPU-GPU link wants (2^22 queries, page-locked: 214 us against 385; n = q =
// 2^26, results in page-locked memory: 2.78 ms against 5.26).
//
// kQueryThreads and the blocks per SM: the loads in flight live in the part
// of the SM's 256 KiB that shared memory leaves (8 KiB per block here); with
// 16 KiB per block, or 32 KiB of shared memory more in all, the headline
// workload (lognormal(2^13, 1), n = q = 2^26) takes 6 % to 100 % longer.
// Without positions ten blocks fit without spills (short queries 4 to 6 %
// faster); with them ten spill 40 bytes (the headline workload 717 -> 779 us).
constexpr uint32_t kQueryThreads = 128;
constexpr uint32_t kLaneQueries = 4;
constexpr uint32_t kBlockQueries = kQueryThreads * kLaneQueries;
constexpr uint32_t kOneThreads = 64;
constexpr uint64_t kFewQueries = uint64_t(1) << 18;

template <bool ARGMIN, bool COLD, typename I, bool LARGE = false>
__global__ void __launch_bounds__(kQueryThreads, sizeof(I) == 4 ? (ARGMIN ? 9 : 10) : 8)
win_query_kernel(WinViewT<I> w, const typename IdxTraits<I>::Pair* __restrict__ qs, uint64_t q,
                 float* __restrict__ out_min, I* __restrict__ out_idx, uint32_t* __restrict__ err) {
    __shared__ __align__(16) unsigned char smem[win_lists_bytes<I>(kBlockQueries)];
    const uint64_t at = uint64_t(blockIdx.x) * kBlockQueries;
    const uint32_t cnt = q - at < kBlockQueries ? uint32_t(q - at) : kBlockQueries;
    const WinLists<I> sm = win_lists<I>(smem, kBlockQueries);
    const uint32_t bad = win_block<ARGMIN, COLD, LARGE, kLaneQueries>(w, sm, kQueryThreads, qs + at, cnt,
                                                               out_min != nullptr ? out_min + at : nullptr,
                                                               ARGMIN ? out_idx + at : nullptr);
    if (bad != 0u && err != nullptr) atomicAdd(err, bad);
}

template <bool ARGMIN, typename I, bool LARGE = false>
__global__ void __launch_bounds__(kOneThreads)
win_one_kernel(WinViewT<I> w, const typename IdxTraits<I>::Pair* __restrict__ qs, uint64_t q,
               float* __restrict__ out_min, I* __restrict__ out_idx, uint32_t* __restrict__ err) {
    // After a build (QueryArgs::after_build) its last kernel may still run.  The
    // loads are not volatile, and all depend on a query's: its address comes
    // from the wait, so none can move before it.
    asm volatile("griddepcontrol.wait;" : "+l"(qs) : : "memory");
    using C = typename IdxTraits<I>::Count;
    const C i = C(blockIdx.x) * kOneThreads + threadIdx.x;
    if (uint64_t(blockIdx.x) * kOneThreads + threadIdx.x >= q) return;
    const typename IdxTraits<I>::Pair Q = ld_query(qs + i);
    WinBest<I> c{f_nan(), IdxTraits<I>::none, false};
    I l = IdxTraits<I>::none;
    if (Q.x <= Q.y && Q.y < w.n) {
        l = Q.x;
        c = win_one<LARGE>(w, l, I(Q.y));
    } else if (err != nullptr) {
        atomicAdd(err, 1u);
    }
    if (out_min != nullptr) st_stream(out_min + i, c.v);
    if (ARGMIN) st_stream(out_idx + i, win_place(w, c, l));
}

// Asked only before launches that take several microseconds.
bool off_device(const void* p) {
    if (p == nullptr) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeHost || at.type == cudaMemoryTypeUnregistered;
}

template <bool ARGMIN, typename I>
static cudaError_t launch_window_typed(const QueryArgs& a, const WinViewT<I>& w,
                                       const typename IdxTraits<I>::Pair* qs, I* out_idx, cudaStream_t s) {
    const bool large = w.blk > 4u;
    if (a.q <= kFewQueries || a.host_buffers || off_device(a.out_min) || off_device(out_idx))
        return launch_with_window(large ? win_one_kernel<ARGMIN, I, true> : win_one_kernel<ARGMIN, I>,
                                  uint32_t((a.q + kOneThreads - 1u) / kOneThreads), kOneThreads, a, s, w, qs, a.q,
                                  a.out_min, out_idx, a.err);
    QueryArgs plain = a;  // the block kernel does not wait for a build
    plain.after_build = false;
    return launch_with_window(large             ? win_query_kernel<ARGMIN, true, I, true>
                              : w.n > kWarmN    ? win_query_kernel<ARGMIN, true, I>
                                                : win_query_kernel<ARGMIN, false, I>,
                              uint32_t((a.q + kBlockQueries - 1u) / kBlockQueries), kQueryThreads, plain, s, w, qs, a.q,
                              a.out_min, out_idx, a.err);
}

cudaError_t launch_window_query(const QueryArgs& a, cudaStream_t s) {
    if (a.wide) {
        const ulonglong2* qs = reinterpret_cast<const ulonglong2*>(a.qs64);
        return a.out_idx64 != nullptr ? launch_window_typed<true, uint64_t>(a, a.win64, qs, a.out_idx64, s)
                                      : launch_window_typed<false, uint64_t>(a, a.win64, qs, nullptr, s);
    }
    return a.out_idx != nullptr ? launch_window_typed<true, uint32_t>(a, a.win, a.qs, a.out_idx, s)
                                : launch_window_typed<false, uint32_t>(a, a.win, a.qs, nullptr, s);
}

// The runtime loads a kernel's code with its first launch unless something
// asks for its attributes before.
cudaError_t load_small_window_kernels() {
    const void* const kernels[] = {reinterpret_cast<const void*>(&win_small_kernel<kShortHalo>),
                                   reinterpret_cast<const void*>(&win_small_kernel<kLongHalo>),
                                   reinterpret_cast<const void*>(&win_top_kernel),
                                   reinterpret_cast<const void*>(&win_one_kernel<true, uint32_t>),
                                   reinterpret_cast<const void*>(&win_query_kernel<true, false, uint32_t>)};
    for (const void* k : kernels) {
        cudaFuncAttributes at;
        const cudaError_t e = cudaFuncGetAttributes(&at, k);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

#if RMQ_DEBUG_BOUNDS
RMQ_BOUNDS_COUNTER_READER(bounds_bad_window)
#endif

}  // namespace rmq
