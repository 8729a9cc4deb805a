// rmq_window.cuh — the window tables and the query over them.
//
// What bounds a query is the number of random sectors it reads: an SM looks up
// one 128-byte line per cycle (289 to 302 G lines/s over the chip by box, measured
// with random 4- to 16-byte loads of 16 MiB) and DRAM serves about 46 G random
// lines/s, so a level-by-level descent that reads ten sectors per query, two
// of them at level 0 in DRAM, ends near 26 G queries/s however it is
// scheduled.  The tables cut both counts: a long query reads two 8-byte
// entries, usually nothing else, and level 0 only when a block at one of its
// ends may hold the answer.
//
// Tables over an array of n values:
//   V1, J1     per block of 2^blk entries: the minimum (float) and the offset
//              of its first occurrence (byte);
//   T_k        for window sizes 2^k, k = first .. kmax: one entry per stride
//              2^s(k), the minimum of [i 2^s, i 2^s + 2^k) (cut off at n) and
//              its first occurrence: the position, or, in tables of 64-bit
//              handles, the offset from the window's start.  A window starts
//              at every 2^c-th part of its size, so the sizes shrink
//              geometrically.
//
// A query of at least half the first window takes the two windows that cover
// it with the least overhang (at most one stride at each end).  The first
// occurrence of the minimum of that cover is the answer whenever it lies
// inside the query.  On values in no particular order that fails for one query
// in 23 (c = 4) or 12 (c = 3); then the query is answered exactly, from
// windows and blocks that lie inside it, with the two blocks at its ends read
// at level 0 only when their minimum would win (win_exact).  A shorter query
// is answered from its blocks: the ones inside it and its ends (win_short), or
// by the cover of the blocks that touch it where level 0 is in DRAM.
//
// Measured, min + argmin, against the block-minimum descent (one thread per
// query, rf = 8) that it replaces, us per launch: lognormal(2^13, 1) lengths,
// n = q = 2^26: 2567 -> 696; the mixture of three length laws with 1 % of the
// values at the minimum, n = q = 2^26: 3377 -> 1614, n = 2^28, q = 2^27:
// 9962 -> 4792; uniform lengths, minima, n = 5e7, q = 3e7: 1226 -> 236;
// lognormal(32, 0.7), positions, n = 2^26, q = 2^25: 1370 -> 696; 64-bit
// positions, lognormal(2^13, 1), n = 2^26, q = 2^25: 1503 -> 564.
#pragma once

#include "rmq_common.cuh"

namespace rmq {

// Sizes of the tables: log2 of the block, of the smallest stride, of the
// strides per window (from window 2^(gb + c) on; smaller ones keep the
// smallest stride), and of the first window.
struct WinForm {
    uint32_t blk, gb, c, first;
};

// The forms, with their bytes per value.  A handle takes the finest one that
// needs no more than the levels that its scan threshold t and reduction factor
// rf plan (win_form_for): a caller chooses its memory by those.  With argmin (8
// bytes per level entry, 12 with 64-bit positions) levels take 1.143 bytes per
// value at rf = 8, 0.533 at 16 and 0.258 at 32; without, half of the 8-byte
// figures; a little less for a large t, nothing for t >= n, where the last form
// is taken all the same.  The coarser forms lose on short and middle lengths.
// n = 2^26, q = 2^24, min + argmin, us, at rf 8 / 16 / 32, and what descending
// such levels took:
//   lognormal(32, 0.7)    365 / 351 / 486     707 / 752 / 850
//   length 500            171 / 469 / 385     677 / 715 / 844
//   lognormal(2^13, 1)    184 / 224 / 248     655 / 854 / 1092
//   uniform lengths       135 / 150 / 150     758 / 1150 / 1376
// Only minima of lengths up to about 60 in arrays that stay in L2 were faster
// there (n = 2^23, rf = 16, length 24: 267 us, here 297).
//
// Windows at every 16th of their size (kFormArgmin) fail half as often as at
// every 8th, which counts for more than short queries do: with blocks of eight
// entries and c = 3 for argmin too, 384 arrays of 2^10 .. 2^20 values built and
// queried together take 2149 us instead of 1960, and n = 2^20, q = 2^22, us,
// length 24: 65 instead of 75, lognormal(2^13, 1): 48 instead of 41.
// Up to kSmallN entries the levels do not count: argmin tables take 4.3 MiB at
// most, and without argmin blocks of eight (4.5 MiB at most, 2.3 MB more than
// levels at rf = 8) pay, since short queries are bound by instructions there
// (length 24: 52 us, with blocks of 16: 67).
constexpr WinForm kForms[] = {
    {4, 5, 4, 8},   // 1.0625
    {3, 5, 3, 8},   // 1.125
    {4, 6, 3, 9},   // 0.5625
    {4, 7, 3, 10},  // 0.4375
    {5, 8, 3, 11},  // 0.2188
    {6, 9, 3, 12},  // 0.1094
};
constexpr uint32_t kFormArgmin = 0, kFormSmallMin = 1, kFormMin = 2, kFormLast = 5;
constexpr uint64_t kSmallN = uint64_t(1) << 22;
constexpr uint32_t kMaxWinLog = 32;  // largest window (offsets are 32-bit)

// log2 of the stride of windows of 2^k entries.
template <typename V>
__host__ __device__ __forceinline__ uint32_t win_stride_log(const V& w, uint32_t k) {
    return k < w.gb + w.c ? w.gb : k - w.c;
}

__host__ __device__ __forceinline__ uint32_t popc_u64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return uint32_t(__popcll(x));
#else
    return uint32_t(__builtin_popcountll(x));
#endif
}
__host__ __device__ __forceinline__ uint32_t popc_of(uint32_t x) {
#ifdef __CUDA_ARCH__
    return uint32_t(__popc(x));
#else
    return uint32_t(__builtin_popcount(x));
#endif
}
__host__ __device__ __forceinline__ uint32_t popc_of(uint64_t x) { return popc_u64(x); }

// Sizes and places of the tables of an array of n values: V1 at byte 0, J1 at
// j1_off, the T entries (8 bytes each) at t_off.  With kb = gb + c, the tables
// below T_kb (stride 2^gb, at most one) come first, and T_(kb + j) (stride
// 2^(gb + j), (S >> j) + 1 entries, S = ceil(n / 2^gb)) starts at entry
// base + sum over i < j of ((S >> i) + 1), which is
// cb + j - 2 (S >> j) + popc(S >> j) with cb = base + 2 S - popc(S).
struct WinShape {
    uint64_t n, nb, S, cb, t_entries, j1_off, t_off, bytes;
    uint32_t blk, gb, c, first, kmax;
};

inline WinShape win_shape(uint64_t n, uint32_t form) {
    const WinForm f = kForms[form];
    WinShape w;
    w.n = n;
    w.blk = f.blk;
    w.gb = f.gb;
    w.c = f.c;
    w.first = f.first;
    w.nb = (n + (uint64_t(1) << f.blk) - 1) >> f.blk;
    w.S = (n + (uint64_t(1) << f.gb) - 1) >> f.gb;
    uint32_t k = 0;
    while (k < kMaxWinLog && (uint64_t(1) << k) < n) ++k;
    w.kmax = k < f.first ? f.first : k;
    const uint32_t kb = f.gb + f.c;
    const uint64_t base = f.first < kb ? w.S + 1u : 0u;
    w.cb = base + 2u * w.S - popc_u64(w.S);
    w.t_entries = 0;
    if (n >= (uint64_t(1) << f.first)) {
        w.t_entries = base;
        for (uint32_t j = 0; kb + j <= w.kmax; ++j) w.t_entries += (w.S >> j) + 1u;
    }
    w.j1_off = (w.nb * sizeof(float) + 31u) & ~uint64_t(31);
    w.t_off = (w.j1_off + w.nb + 31u) & ~uint64_t(31);
    w.bytes = (w.t_off + w.t_entries * 8u + 31u) & ~uint64_t(31);
    return w;
}

// The form of an array's tables: `levels`, the bytes that its planned levels take.
inline uint32_t win_form_for(uint64_t n, bool with_index, uint64_t levels) {
    if (n <= kSmallN) return with_index ? kFormArgmin : kFormSmallMin;
    uint32_t f = with_index ? kFormArgmin : kFormMin;
    while (f < kFormLast && win_shape(n, f).bytes > levels) f = f < kFormMin ? kFormMin : f + 1u;
    return f;
}

// The tables as the kernels see them (I: position type).
template <typename I>
struct WinViewT {
    const float* a;
    const float* v1;
    const uint8_t* j1;
    const uint2* t;
    I n, S, cb;
    uint32_t blk, gb, c, first, kmax;
};
using WinView = WinViewT<uint32_t>;
using WinView64 = WinViewT<uint64_t>;

template <typename I>
inline WinViewT<I> win_view(const float* a, const void* base, uint64_t n, uint32_t form) {
    const WinShape w = win_shape(n, form);
    WinViewT<I> v;
    const char* b = static_cast<const char*>(base);
    v.a = a;
    v.v1 = reinterpret_cast<const float*>(b);
    v.j1 = reinterpret_cast<const uint8_t*>(b + w.j1_off);
    v.t = reinterpret_cast<const uint2*>(b + w.t_off);
    v.n = I(n);
    v.S = I(w.S);
    v.cb = I(w.cb);
    v.blk = w.blk;
    v.gb = w.gb;
    v.c = w.c;
    v.first = w.first;
    v.kmax = w.kmax;
    return v;
}

// The tables as the build kernels write them.
struct WinOut {
    const float* a;
    float* v1;
    uint8_t* j1;
    uint2* t;
    uint64_t n, S, cb;
    uint32_t blk, gb, c, first, kmax;
    bool wide;  // T holds offsets from the window's start instead of positions
};

// Descriptor of one array inside packed buffers (batched and served modes).
struct ArrayDesc {
    uint64_t val_off;   // first value of the array, in floats from the values base
    uint64_t win_off;   // its tables, in bytes from the tables base
    uint32_t n, S, cb;  // as in WinShape
    uint32_t j1_off, t_off;
    uint32_t blk, gb, c, first, kmax;
};

inline ArrayDesc win_desc(uint64_t val_off, uint64_t win_off, const WinShape& w) {
    ArrayDesc d;
    d.val_off = val_off;
    d.win_off = win_off;
    d.n = uint32_t(w.n);
    d.S = uint32_t(w.S);
    d.cb = uint32_t(w.cb);
    d.j1_off = uint32_t(w.j1_off);
    d.t_off = uint32_t(w.t_off);
    d.blk = w.blk;
    d.gb = w.gb;
    d.c = w.c;
    d.first = w.first;
    d.kmax = w.kmax;
    return d;
}

__device__ __forceinline__ WinOut win_out(const ArrayDesc& d, const float* values, char* tables) {
    char* b = tables + d.win_off;
    return WinOut{values + d.val_off, reinterpret_cast<float*>(b), reinterpret_cast<uint8_t*>(b + d.j1_off),
                  reinterpret_cast<uint2*>(b + d.t_off), d.n, d.S, d.cb, d.blk, d.gb, d.c, d.first, d.kmax,
                  false};
}

__device__ __forceinline__ void win_load_view(const ArrayDesc& d, const float* values, const char* tables,
                                              WinView& v) {
    const char* b = tables + d.win_off;
    v.a = values + d.val_off;
    v.v1 = reinterpret_cast<const float*>(b);
    v.j1 = reinterpret_cast<const uint8_t*>(b + d.j1_off);
    v.t = reinterpret_cast<const uint2*>(b + d.t_off);
    v.n = d.n;
    v.S = d.S;
    v.cb = d.cb;
    v.blk = d.blk;
    v.gb = d.gb;
    v.c = d.c;
    v.first = d.first;
    v.kmax = d.kmax;
}

__host__ __device__ __forceinline__ uint32_t win_log2(uint32_t x) {
#ifdef __CUDA_ARCH__
    return 31u - uint32_t(__clz(int(x)));
#else
    return 31u - uint32_t(__builtin_clz(x));
#endif
}
__host__ __device__ __forceinline__ uint32_t win_log2(uint64_t x) {
#ifdef __CUDA_ARCH__
    return 63u - uint32_t(__clzll((long long)x));
#else
    return 63u - uint32_t(__builtin_clzll(x));
#endif
}

// First entry of T_k.
template <typename I, typename V>
__host__ __device__ __forceinline__ I win_table_at(const V& w, uint32_t k) {
    const uint32_t kb = w.gb + w.c;
    if (k < kb) return I(0);
    const I sj = I(w.S) >> (k - kb);
    return I(w.cb) + I(k - kb) - I(2) * sj + I(popc_of(sj));
}

// ---------------------------------------------------------------------------
// Loads.  Tables: evict-last in L2 (shared by all queries).  Level 0:
// evict-first (a block that had to be read once is seldom read again soon).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint2 ld_win(const uint2* p) {
    uint2 v;
    asm("{\n\t.reg .b64 pol;\n\t"
        "createpolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
        "ld.global.nc.L2::cache_hint.v2.u32 {%0,%1}, [%2], pol;\n\t}"
        : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t ld_off(const uint8_t* p) {
    uint32_t v;
    asm("{\n\t.reg .b64 pol;\n\t"
        "createpolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
        "ld.global.nc.L2::cache_hint.u8 %0, [%1], pol;\n\t}"
        : "=r"(v) : "l"(p));
    return v;
}

// A candidate: value (its first occurrence's own bits) and position, or, with
// `blk`, the number of the V1 block whose first minimum it is.  Empty:
// (+inf, none).  Candidates are offered in ascending position order and taken
// when strictly less, so the first minimum stays; a range of +inf alone ends
// empty, and its answer is its first entry (win_place).
template <typename I>
struct WinBest {
    float v;
    I p;
    bool blk;
};

template <typename I>
__device__ __forceinline__ void win_take(WinBest<I>& cur, float v, I p) {
    if (v < cur.v) {
        cur.v = v;
        cur.p = p;
        cur.blk = false;
    }
}

template <typename I>
__device__ __forceinline__ WinBest<I> win_none() {
    return WinBest<I>{f_inf(), IdxTraits<I>::none, false};
}

// Bits lo .. hi - 1 of a byte (hi <= 8).
__device__ __forceinline__ uint32_t win_bits(uint32_t lo, uint32_t hi) { return ((1u << hi) - 1u) & ~((1u << lo) - 1u); }

__device__ __forceinline__ float win_pick(const float (&v)[8], uint32_t j) {
    const bool b0 = (j & 1u) != 0u, b1 = (j & 2u) != 0u;
    const float x0 = b0 ? v[1] : v[0], x1 = b0 ? v[3] : v[2], x2 = b0 ? v[5] : v[4], x3 = b0 ? v[7] : v[6];
    const float y0 = b1 ? x1 : x0, y1 = b1 ? x3 : x2;
    return (j & 4u) != 0u ? y1 : y0;
}

// v[j] where bit j of `mask` is set, else +inf; the minimum of those.
__device__ __forceinline__ float win_mask8(float (&v)[8], uint32_t mask) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = ((mask >> j) & 1u) != 0u ? v[j] : f_inf();
    return fmin3(fmin3(v[0], v[1], v[2]), fmin3(v[3], v[4], v[5]), fminf(v[6], v[7]));
}

// The minimum of v[j] over the bits of `mask`, where its place is not wanted
// (a predicated min per entry: 3 % faster than win_mask8 there).
__device__ __forceinline__ float win_min8(const float (&v)[8], uint32_t mask) {
    float m = f_inf();
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if ((mask & (1u << j)) != 0u) m = fminf(m, v[j]);
    return m;
}

// First entry of u equal to x, their minimum (not NaN), and in x its own bits.
__device__ __forceinline__ uint32_t win_locate8(const float (&u)[8], float& x) {
    uint32_t jb = 7u;
#pragma unroll
    for (int j = 6; j >= 0; --j)
        if (u[j] == x) jb = uint32_t(j);
    if (x == 0.0f) x = win_pick(u, jb);  // the first zero's own sign
    return jb;
}

// Position of an entry of T for the window starting at `start`.
__device__ __forceinline__ uint32_t win_pos(uint2 e, uint32_t) { return e.y; }
__device__ __forceinline__ uint64_t win_pos(uint2 e, uint64_t start) { return start + e.y; }

// Entry of T_k for the window starting at `start` (a multiple of its stride).
template <typename I>
__device__ __forceinline__ uint2 win_entry(const WinViewT<I>& w, uint32_t k, I start) {
    const uint32_t s = win_stride_log(w, k);
    const I i = start >> s;
#if RMQ_DEBUG_BOUNDS
    if (!bounds_ok(k >= w.first && k <= w.kmax && start < w.n && (start & ((I(1) << s) - 1u)) == 0 &&
                   i <= (k < w.gb + w.c ? w.S : (w.S >> (k - w.gb - w.c)))))
        return make_uint2(0x7f800000u, 0u);
#endif
    return ld_win(w.t + win_table_at<I>(w, k) + i);
}

// V1 of blocks b .. b + 7 (b a multiple of 8; V1 is padded to a sector).
template <typename I>
__device__ __forceinline__ void ld_blocks8(const WinViewT<I>& w, I b, float (&v)[8]) {
#if RMQ_DEBUG_BOUNDS
    if (!bounds_ok((b & 7u) == 0 && (b << w.blk) < w.n)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = f_inf();
        return;
    }
#endif
    asm("ld.global.nc.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(w.v1 + b), "l"(policy_evict_last()));
}

template <typename I>
__device__ __forceinline__ uint32_t ld_block_off(const WinViewT<I>& w, I b) {
#if RMQ_DEBUG_BOUNDS
    if (!bounds_ok((b << w.blk) < w.n)) return 0u;
#endif
    return ld_off(w.j1 + b);
}

// Sector of level 0 from s (a multiple of 8, s < n).
template <typename I>
__device__ __forceinline__ void ld_values8(const WinViewT<I>& w, I s, float (&v)[8]) {
#if RMQ_DEBUG_BOUNDS
    if (!bounds_ok((s & 7u) == 0 && s < w.n)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = f_inf();
        return;
    }
#endif
    if (s + 8u <= w.n) {
        asm("ld.global.nc.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
            : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
            : "l"(w.a + s), "l"(policy_evict_first()));
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (s + I(j) < w.n) ? w.a[s + j] : f_inf();
    }
}

// The same loads where `p` holds, zeros elsewhere (the caller masks them out);
// a sector of level 0 has to lie inside the array.  Without the zeros the
// registers of a load that may not happen count as live from the start of the
// kernel, and it spills 176 bytes.
template <typename I>
__device__ __forceinline__ void ld_blocks8_if(const WinViewT<I>& w, bool p, I b, float (&v)[8]) {
#if RMQ_DEBUG_BOUNDS
    p = p && bounds_ok((b & 7u) == 0 && (b << w.blk) < w.n);
#endif
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.0f;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %10, 0;\n\t"
        "@p ld.global.nc.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;\n\t}"
        : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7])
        : "l"(w.v1 + b), "l"(policy_evict_last()), "r"(uint32_t(p)));
}

template <typename I>
__device__ __forceinline__ void ld_values8_if(const WinViewT<I>& w, bool p, I s, float (&v)[8]) {
#if RMQ_DEBUG_BOUNDS
    p = p && bounds_ok((s & 7u) == 0 && s + 8u <= w.n);
#endif
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.0f;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %10, 0;\n\t"
        "@p ld.global.nc.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;\n\t}"
        : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7])
        : "l"(w.a + s), "l"(policy_evict_first()), "r"(uint32_t(p)));
}

// First minimum of level-0 entries [lo, hi) (lo < hi), which touch at most N
// sectors: every sector's load is issued before the first is used.
template <int N, typename I>
__device__ __forceinline__ WinBest<I> win_raw(const WinViewT<I>& w, I lo, I hi) {
    WinBest<I> c{f_inf(), lo, false};
    const I s0 = lo & ~I(7);
    float v[N][8];
#pragma unroll
    for (uint32_t h = 0; h < N; ++h)
        if (h == 0 || s0 + 8u * h < hi) ld_values8(w, I(s0 + 8u * h), v[h]);
    const uint32_t bits = ((2u << uint32_t(hi - 1u - s0)) - 1u) & ~((1u << uint32_t(lo - s0)) - 1u);
    c.v = win_mask8(v[0], bits);
    uint32_t at = 0;
#pragma unroll
    for (uint32_t h = 1; h < N; ++h) {
        if (s0 + 8u * h < hi) {
            const float y = win_mask8(v[h], bits >> (8u * h));
            if (y < c.v) {
                c.v = y;
                at = 8u * h;
#pragma unroll
                for (int j = 0; j < 8; ++j) v[0][j] = v[h][j];
            }
        }
    }
    // +inf throughout: entries outside the range compare equal, the first inside is lo
    if (c.v < f_inf()) c.p = s0 + at + win_locate8(v[0], c.v);
    return c;
}

// The same over any number of sectors, two at a time (four at once spill).
template <typename I>
__device__ __forceinline__ WinBest<I> win_raw_long(const WinViewT<I>& w, I lo, I hi) {
    WinBest<I> c{f_inf(), lo, false};
#pragma unroll 1
    for (I at = lo; at < hi;) {
        const I cut = (at & ~I(15)) + 16u, end = hi < cut ? hi : cut;
        const WinBest<I> d = win_raw<2>(w, at, end);
        if (d.v < c.v) c = d;
        at = end;
    }
    return c;
}

// The blocks b + j, j in the bits of `mask`, of a loaded sector, offered to cur.
template <typename I>
__device__ __forceinline__ void win_take_blocks(float (&v)[8], uint32_t mask, I b, WinBest<I>& cur) {
    float x = win_mask8(v, mask);
    if (x < cur.v) {
        cur.p = b + win_locate8(v, x);
        cur.v = x;
        cur.blk = true;
    }
}

// First minimum of the V1 blocks [b0, b1), offered to cur: two sectors at a
// time, their minima first and then the place in the sector that holds it.
template <typename I>
__device__ __forceinline__ void win_blocks(const WinViewT<I>& w, I b0, I b1, WinBest<I>& cur) {
#pragma unroll 1
    for (I b = b0 & ~I(7); b < b1; b += 16u) {
        float u[8], v[8];
        const bool more = b + 8u < b1;
        ld_blocks8(w, b, u);
        if (more) ld_blocks8(w, I(b + 8u), v);
        const uint32_t lo = b < b0 ? uint32_t(b0 - b) : 0u, hi = b1 - b < 16u ? uint32_t(b1 - b) : 16u;
        const uint32_t bits = ((1u << hi) - 1u) & ~((1u << lo) - 1u);
        float x = win_mask8(u, bits);
        uint32_t at = 0;
        if (more) {
            const float y = win_mask8(v, bits >> 8);
            if (y < x) {
                x = y;
                at = 8u;
#pragma unroll
                for (int j = 0; j < 8; ++j) u[j] = v[j];
            }
        }
        if (x < cur.v) {
            cur.p = b + at + win_locate8(u, x);
            cur.v = x;
            cur.blk = true;
        }
    }
}

// The partial blocks at the two ends of [l, R): the left one offered before
// cur's position (it wins ties), the right one after.  vl, vr: the whole
// blocks' minima; +inf leaves the right end out.  A block's stored first
// minimum serves when it lies inside the query; otherwise its part of the
// query is read at level 0.  LARGE: blocks of more than 16 entries.
template <bool LARGE, typename I>
__device__ __forceinline__ void win_ends(const WinViewT<I>& w, I l, I R, float vl, float vr, WinBest<I>& cur) {
#pragma unroll 1
    for (uint32_t side = 0; side < 2; ++side) {
        const float vb = side ? vr : vl;
        if (side ? !(vb < cur.v) : !(vb <= cur.v)) continue;
        const I b = (side ? R - 1u : l) >> w.blk;
        const I s = b << w.blk, p = s + ld_block_off(w, b);
        const I e = s + (I(1) << w.blk), lo = s < l ? l : s, hi = e < R ? e : R;
        WinBest<I> c{vb, p, false};
        if (p < lo || p >= hi) c = LARGE ? win_raw_long(w, lo, hi) : win_raw<2>(w, lo, hi);
        if (side ? c.v < cur.v : c.v <= cur.v) cur = c;
    }
}

// A query [l, R) shorter than the first window, answered by the first minimum
// of the blocks that touch it: true when that lies inside.
template <typename I>
__device__ __forceinline__ bool win_short_cover(const WinViewT<I>& w, I l, I R, WinBest<I>& cur) {
    cur = win_none<I>();
    win_blocks(w, l >> w.blk, ((R - 1u) >> w.blk) + 1u, cur);
    if (cur.p == IdxTraits<I>::none) return false;  // +inf throughout
    cur.p = (cur.p << w.blk) + ld_block_off(w, cur.p);
    cur.blk = false;
    return cur.p >= l && cur.p < R;
}

// Arrays whose values stay in L2 beside their tables; a sector of a larger one
// comes from DRAM.
constexpr uint64_t kWarmN = uint64_t(1) << 24;

// A query [l, R) shorter than the first window, in an array that stays in L2
// (win_block reads those from DRAM by win_short_cover, whose few level-0
// sectors are what counts there: lognormal(32, 0.7), n = 2^26, q = 2^25:
// 698 us against 805).  The whole blocks inside it from V1, then the part of
// the query in each of the two blocks at its ends from level 0, only where
// that block's minimum is below (left: not above) theirs: 2.3 to 2.9 sectors
// instead of 3.1 to 4.8 with both ends and no V1 minima to compare.  What
// bounds it is the ALU pipe (70-75 % busy), so the lanes of a warp stay in
// step (loads under a predicate, no branches around them) and the place of
// the minimum is looked up once, at the end.  Length 24, n = 2^20, q = 2^22,
// us: min + argmin 89 -> 75, minima 66 -> 52; lognormal(32, 0.7) 87 -> 82 and
// 80 -> 68 (by blocks that touch the query, the failures listed and redone).
// The query must be longer than a block, so that its ends lie in two blocks (with
// both in one, the right end's part would begin before l): callers answer up to
// 16 entries by win_raw.  The last sector of level 0 must not be cut off
// (R <= n rounded down to 8).
// SECTORS: of a block.  POS: the position is wanted.
template <bool POS, uint32_t SECTORS, typename I>
__device__ __forceinline__ WinBest<I> win_short(const WinViewT<I>& w, I l, I R) {
    constexpr uint32_t blk = SECTORS == 1u ? 3u : 4u;
    const I bl = l >> blk, br = (R - 1u) >> blk, b = bl & ~I(7);
    const uint32_t i = uint32_t(bl - b), last = uint32_t(br - b);
    WinBest<I> c{f_inf(), b, true};
    float K[8], U[8];  // POS: the sector that holds c.v, its other entries masked out
    ld_blocks8(w, b, K);
    ld_blocks8_if(w, last > 7u, I(b + 8u), U);
    const float vl = win_pick(K, i), v0 = win_pick(K, last & 7u), v1 = win_pick(U, last & 7u);
    float vr = last < 8u ? v0 : v1;
    const uint32_t hi = last < 16u ? last : 16u;
    const uint32_t bits = ((1u << hi) - 1u) & ~((2u << i) - 1u);
    const auto least = [](float (&v)[8], uint32_t mask) { return POS ? win_mask8(v, mask) : win_min8(v, mask); };
    // x, the least of U, offered to c; `at`: U's first entry, of V1 or of level 0
    const auto take = [&](float x, I at, bool block, bool ties) {
        if (ties ? x <= c.v : x < c.v) {
            c.v = x;
            c.p = at;
            c.blk = block;
            if (POS) {
#pragma unroll
                for (int j = 0; j < 8; ++j) K[j] = U[j];
            }
        }
    };
    c.v = least(K, bits);
    take(least(U, bits >> 8), I(b + 8u), true, false);
#pragma unroll 1
    for (uint32_t k = 16; k <= last; k += 8u) {
        ld_blocks8(w, I(b + k), U);
        vr = win_pick(U, last & 7u);
        take(least(U, last - k < 8u ? (1u << (last - k)) - 1u : 255u), I(b + k), true, false);
    }
    const I e = (bl + 1u) << blk;
    I lo = l, end = R < e ? R : e;
    bool need = vl <= c.v;
#pragma unroll 1
    for (uint32_t side = 0; side < 2; ++side) {
        const I s = lo & ~I(7);
        const uint32_t part = need ? ((2u << uint32_t(end - 1u - s)) - 1u) & ~((1u << uint32_t(lo - s)) - 1u) : 0u;
        if (SECTORS > 1u) {
            float A[8];
            ld_values8_if(w, need, s, A);
            ld_values8_if(w, (part >> 8) != 0u, I(s + 8u), U);
            float x = least(A, part);
            const float y = least(U, part >> 8);
            I at = s + 8u;
            if (!(y < x)) {
                at = s;
                if (POS) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) U[j] = A[j];
                }
            } else {
                x = y;
            }
            // as take(), which ptxas makes 6 % slower here
            if (side ? x < c.v : x <= c.v) {
                c.v = x;
                c.p = at;
                c.blk = false;
                if (POS) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) K[j] = U[j];
                }
            }
        } else {
            ld_values8_if(w, need, s, U);
            take(least(U, part), s, false, side == 0u);
        }
        lo = br << blk;
        end = R;
        need = vr < c.v;
    }
    if (POS) {
        if (c.v < f_inf()) {
            c.p += win_locate8(K, c.v);
        } else {
            c.p = l;
            c.blk = false;
        }
    } else if (__float_as_uint(c.v) == 0x80000000u) {
        // min.f32 takes -0 before +0: the sign is that of the query's first zero
        I p = l;
        while (w.a[p] != 0.0f) ++p;
        c.v = w.a[p];
    }
    return c;
}

// A short query [l, R) in one round trip: its ends at level 0 and its whole
// blocks, all read at once.  SECTORS: of a block.
template <uint32_t SECTORS, typename I>
__device__ __forceinline__ WinBest<I> win_short_once(const WinViewT<I>& w, I l, I R) {
    const I bl = l >> w.blk, br = (R - 1u) >> w.blk;
    const I a0 = l & ~I(7), ae = (bl + 1u) << w.blk, ar = R < ae ? R : ae;  // left end: [l, ar)
    const I r0 = br << w.blk, b0 = (bl + 1u) & ~I(7);
    const bool right = br != bl, a1 = SECTORS > 1u && a0 + 8u < ar,
               r1 = SECTORS > 1u && right && r0 + 8u < R, mid = br > bl + 1u;
    float A[8], A1[8], V[8], B[8], B1[8];
    ld_values8(w, a0, A);
    if (a1) ld_values8(w, I(a0 + 8u), A1);
    if (right) ld_values8(w, r0, B);
    if (r1) ld_values8(w, I(r0 + 8u), B1);
    if (mid) ld_blocks8(w, b0, V);
    const uint32_t abits = ((2u << uint32_t(ar - 1u - a0)) - 1u) & ~((1u << uint32_t(l - a0)) - 1u);
    const uint32_t rbits = (2u << uint32_t(R - 1u - r0)) - 1u;
    WinBest<I> c{f_inf(), l, false};
    const auto take = [&](float (&u)[8], uint32_t bits, I s, bool blk) {
        float x = win_mask8(u, bits);
        if (x < c.v) {
            c.p = s + win_locate8(u, x);
            c.v = x;
            c.blk = blk;
        }
    };
    take(A, abits, a0, false);
    if (a1) take(A1, abits >> 8, I(a0 + 8u), false);
    if (mid) {
        take(V, win_bits(uint32_t(bl + 1u - b0), br - b0 < 8u ? uint32_t(br - b0) : 8u), b0, true);
#pragma unroll 1
        for (I b = b0 + 8u; b < br; b += 8u) {
            ld_blocks8(w, b, V);
            take(V, win_bits(0u, br - b < 8u ? uint32_t(br - b) : 8u), b, true);
        }
    }
    if (right) take(B, rbits, r0, false);
    if (r1) take(B1, rbits >> 8, I(r0 + 8u), false);
    return c;
}

// The part [x, y) of a query [l, R) that lies on whole strides of 2^gb: true
// when it holds eight of them, so that windows inside the query serve it.  With
// 32-bit positions the distance decides, since x plus eight strides would wrap
// near 2^32; x itself does for l above 2^32 - 2^9 with the strides of 2^9 that only tables with LARGE
// blocks have (n goes up to 2^32 - 2^8).
template <bool LARGE, typename I>
__host__ __device__ __forceinline__ bool win_inner(I l, I R, uint32_t gb, I& x, I& y) {
    const I gm = (I(1) << gb) - 1u;
    x = (l + gm) & ~gm;
    y = R & ~gm;
    if (sizeof(I) == 8) return y >= x + (I(8) << gb);
    return (!LARGE || x >= l) && y >= x && y - x >= (I(8) << gb);
}

// The exact answer of [l, R) from entries inside it, for a query whose cover
// had its first minimum outside: all but the partial blocks at the two ends,
// which are left to win_ends with their blocks' minima vl and vr (vr +inf: not
// needed).  A range of a few strides is taken block by block.  Otherwise,
// between x = l rounded up and y = R rounded down to the smallest stride, the
// range is taken from windows: at each end one window per 2^c-fold of
// alignment, then the two windows that cover the rest; the few whole blocks
// between l and x, and y and R, come from the end blocks' sectors of V1.
// `bound` is a lower bound of the answer (the cover's minimum; NaN: none): an
// entry equal to it that is found first from the left ends the search
// (repeated minima: the usual case after a cover whose first occurrence lay
// left of l; in the first sector of V1 already for three in five where one
// value in 100 is the minimum: the mixture of lengths with n = 2^28, q = 2^27
// 4858 -> 4801 us).
template <bool LARGE, typename I>
__device__ __forceinline__ void win_exact(const WinViewT<I>& w, I l, I R, float bound, WinBest<I>& cur, float& vl,
                                          float& vr) {
    const uint32_t gb = w.gb, step = w.c;
    const I bl = l >> w.blk, br = (R - 1u) >> w.blk, last = br & ~I(7);
    I x, y;
    const bool windows = win_inner<LARGE>(l, R, gb, x, y);
    const I by = y >> w.blk;
    I b = bl & ~I(7);
    {
        const I end = windows ? x >> w.blk : br;
        float v[8];
        ld_blocks8(w, b, v);
        vl = win_pick(v, uint32_t(bl - b));
        if (b == last && br != bl) vr = win_pick(v, uint32_t(br - b));
        win_take_blocks(v, win_bits(uint32_t(bl - b) + 1u, end <= b ? 0u : (end - b < 8u ? uint32_t(end - b) : 8u)), b, cur);
        if (b == last || cur.v == bound) return;
    }
    b += 8u;
    if (windows) {
        uint32_t s = gb;
        WinBest<I> right = win_none<I>();
        I d = y - x;
        constexpr uint32_t kTop = sizeof(I) == 4 ? 30u : kMaxWinLog;  // two windows of 2^31 exceed 32 bits
#pragma unroll 1
        while (s + step <= kTop && d >= (I(2) << (s + step))) {
            const uint32_t k = s + step;
            const I W = I(1) << k;
            const uint2 el = win_entry(w, k, x), er = win_entry(w, k, I(y - W));
            win_take(cur, __uint_as_float(el.x), win_pos(el, x));
            if (cur.v == bound) return;
            const float rv = __uint_as_float(er.x);
            if (rv <= right.v) {
                right.v = rv;
                right.p = win_pos(er, I(y - W));
            }
            x = (x + W - 1u) & ~(W - 1u);
            y &= ~(W - 1u);
            s = k;
            d = y - x;
        }
        uint32_t k = win_log2(d);
        if (sizeof(I) == 8 && k > kMaxWinLog) k = kMaxWinLog;
        const I W = I(1) << k;
        // The whole blocks right of y lie in the last sector (y is not below its
        // start, a multiple of the stride); its load and the two windows' go
        // out together, as do a pair's above: a block of queries waits for the
        // few that come here (headline workload 727 -> 703 us on one box,
        // sorted values 6 % faster).
        float u[8];
        ld_blocks8(w, last, u);
        const uint2 e1 = win_entry(w, k, x), e2 = win_entry(w, k, I(y - W));
        win_take(cur, __uint_as_float(e1.x), win_pos(e1, x));
        if (sizeof(I) == 8) {
            for (I z = x; y - z >= 2u * W;) {
                z += W;
                const uint2 e = win_entry(w, k, z);
                win_take(cur, __uint_as_float(e.x), win_pos(e, z));
            }
        }
        win_take(cur, __uint_as_float(e2.x), win_pos(e2, I(y - W)));
        win_take(cur, right.v, right.p);
        vr = win_pick(u, uint32_t(br - last));
        win_take_blocks(u, win_bits(uint32_t(by - last), uint32_t(br - last)), last, cur);
        return;
    }
#pragma unroll 1
    for (;; b += 8u) {
        float v[8];
        ld_blocks8(w, b, v);
        if (b == last) vr = win_pick(v, uint32_t(br - b));
        win_take_blocks(v, win_bits(0u, b == last ? uint32_t(br - b) : 8u), b, cur);
        if (b == last) return;
    }
}

// ---------------------------------------------------------------------------
// A block answers a run of queries, LQ per thread in a pass.  Every lane looks
// up the covering windows of LQ queries at once (eight loads in flight at 4);
// the queries that need more are listed in shared memory by kind and then
// answered by the whole block, 32 to a warp, so that the few long queries
// whose cover failed and the short queries of a mixture run with full warps
// instead of one or two lanes.  Without the lists 9.4 of 32 lanes are active
// and the headline workload is bound by instruction issue at 51 G queries/s;
// with them it runs at 93.
// ---------------------------------------------------------------------------

// Shared memory of a block that answers up to `cap` queries (cap <= 65536).
template <typename I>
struct WinLists {
    typename IdxTraits<I>::Pair* q;
    float* bound;      // failed covers: their minimum (NaN: none), by place in `rest`
    uint16_t* first;   // short queries from the front, the shortest from the back
    uint16_t* rest;    // queries that need win_exact
    uint32_t* count;   // entries: short, shortest, rest
    uint32_t cap;
};
template <typename I>
__host__ __device__ constexpr uint32_t win_lists_bytes(uint32_t cap) {
    return cap * (uint32_t(sizeof(typename IdxTraits<I>::Pair)) + 8u) + 16u;
}
template <typename I>
__device__ __forceinline__ WinLists<I> win_lists(unsigned char* smem, uint32_t cap) {
    using Pair = typename IdxTraits<I>::Pair;
    WinLists<I> s;
    s.q = reinterpret_cast<Pair*>(smem);
    s.bound = reinterpret_cast<float*>(s.q + cap);
    s.first = reinterpret_cast<uint16_t*>(s.bound + cap);
    s.rest = s.first + cap;
    s.count = reinterpret_cast<uint32_t*>(s.rest + cap);
    s.cap = cap;
    return s;
}

// Queries of up to this many entries (at most 16: three sectors) are read at
// level 0: one round trip, and the cover by blocks fails for more than half of
// them (n = 2^20, q = 2^22, length 8 / 16: 49 / 62 us against 103 / 98).
// Beyond 2^27 entries only up to eight: there the address translation of
// random level-0 sectors bounds the chip at 55 G sectors/s (n = 2^28, length
// 16: 231 us at level 0, 158 by blocks).  LARGE: up to 32 entries, since a
// cover of blocks of 32 or 64 fails for most of them (n = 2^23, q = 2^24,
// blocks of 32, length 24: 354 us against 480; length 40: 455 against 439).
template <bool LARGE, typename I>
__device__ __forceinline__ I win_raw_limit(I n) { return n > (I(1) << 27) ? I(8) : I(LARGE ? 32 : 16); }

// The two windows of T_k that cover [l, r] (len entries, at least half the
// first window): starts s1 <= s2, equal when one window covers it.  k is the
// smallest size of which two windows cover any query of this length wherever
// it lies: two windows of 2^k hold len + 2 strides - 2 entries when
// len < 7/4 2^k (a stride is at most 1/8 of the window).
template <typename I>
__host__ __device__ __forceinline__ bool win_cover(const WinViewT<I>& w, I l, I r, I len, uint32_t& k, I& s1, I& s2) {
    k = win_log2(len);
    if ((len >> (k - 3u)) >= 14u) ++k;
    if (k < w.first) k = w.first;
    if (sizeof(I) == 8 && k > kMaxWinLog) k = kMaxWinLog;
    const uint32_t s = win_stride_log(w, k);
    const I a = l >> s, e = (r >> s) + 1u, wu = I(1) << (k - s);
    s1 = a << s;
    s2 = (e - (e - a < wu ? e - a : wu)) << s;
    return sizeof(I) == 4 || e - a <= 2u * wu;  // 64-bit: longer than two of the largest windows
}

// Position of an answer.
template <typename I>
__device__ __forceinline__ I win_place(const WinViewT<I>& w, const WinBest<I>& c, I l) {
    if (c.blk) return (c.p << w.blk) + ld_block_off(w, c.p);
    return c.p == IdxTraits<I>::none ? l : c.p;
}

// Queries qs[0 .. cnt) (cnt <= sm.cap, a multiple of threads x LQ; every thread
// of the block of `threads` calls), results to the same places of out_min /
// out_idx (null: not wanted).  COLD: level 0 is in DRAM (n > kWarmN).  ARGMIN:
// of tables with positions, whose blocks are not of eight entries.  LARGE: blocks
// of more than 16 entries (COLD only).  Returns this thread's number of invalid
// queries (l > r or r >= n), which get NaN and all ones.
template <bool ARGMIN, bool COLD, bool LARGE, uint32_t LQ, typename I>
__device__ __forceinline__ uint32_t win_block(const WinViewT<I>& w, const WinLists<I>& sm, uint32_t threads,
                                              const typename IdxTraits<I>::Pair* __restrict__ qs, uint32_t cnt,
                                              float* __restrict__ out_min, I* __restrict__ out_idx) {
    using Pair = typename IdxTraits<I>::Pair;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = w.first;
    const bool tables = w.n >= (I(1) << first);
    const I raw_limit = COLD ? win_raw_limit<LARGE, I>(w.n) : I(16), whole = w.n & ~I(7);
    uint32_t bad = 0;
    const auto store = [&](const WinBest<I>& c, I l, uint32_t slot) {
        if (out_min != nullptr) st_stream(out_min + slot, c.v);
        if (ARGMIN) st_stream(out_idx + slot, win_place(w, c, l));
    };
    if (threadIdx.x < 4u) sm.count[threadIdx.x] = 0u;
    __syncthreads();
#pragma unroll 1
    for (uint32_t pass = 0; pass < cnt; pass += threads * LQ) {
        Pair Q[LQ];
        uint2 e1[LQ], e2[LQ];
        I s1[sizeof(I) == 8 ? LQ : 1], s2[sizeof(I) == 8 ? LQ : 1];
#pragma unroll
        for (uint32_t j = 0; j < LQ; ++j) {
            const uint32_t slot = pass + threadIdx.x + threads * j;
            Q[j].x = 1u;
            Q[j].y = 0u;
            if (slot < cnt) Q[j] = ld_query(qs + slot);
        }
#pragma unroll
        for (uint32_t j = 0; j < LQ; ++j) {
            const I l = Q[j].x, r = Q[j].y, len = r - l + 1u;
            if (l <= r && r < w.n && (len >> (first - 1u)) != 0u && tables) {
                uint32_t k;
                I a, b;
                const bool covered = win_cover(w, l, r, len, k, a, b);
                e1[j] = win_entry(w, k, a);
                e2[j] = win_entry(w, k, b);
                if constexpr (sizeof(I) == 8) {
                    s1[j] = covered ? a : IdxTraits<I>::none;
                    s2[j] = b;
                }
            }
        }
        uint32_t kinds = 0;  // per query: 0 answered, 1 short, 2 shortest, 3 rest
        float bound[LQ];
#pragma unroll
        for (uint32_t j = 0; j < LQ; ++j) {
            const uint32_t slot = pass + threadIdx.x + threads * j;
            const I l = Q[j].x, r = Q[j].y, len = r - l + 1u;
            uint32_t kind = 0;
            if (!(l <= r && r < w.n)) {
                if (slot < cnt) {
                    ++bad;
                    store(WinBest<I>{f_nan(), IdxTraits<I>::none, false}, IdxTraits<I>::none, slot);
                }
            } else if (len <= raw_limit) {
                kind = 2u;
            } else if ((len >> (first - 1u)) == 0u || !tables) {
                kind = 1u;
                if (!COLD && r >= whole) {
                    kind = 3u;
                    bound[j] = f_nan();
                }
            } else {
                WinBest<I> c{__uint_as_float(e1[j].x), I(e1[j].y), false};
                I p2 = I(e2[j].y);
                bool covered = true;
                if constexpr (sizeof(I) == 8) {
                    c.p += s1[j];
                    p2 += s2[j];
                    covered = s1[j] != IdxTraits<I>::none;
                }
                win_take(c, __uint_as_float(e2[j].x), p2);
                if (covered && c.p >= l && c.p <= r) {
                    store(c, l, slot);
                } else {
                    kind = (len >> first) != 0u || (!COLD && r >= whole) ? 3u : 1u;
                    bound[j] = covered ? c.v : f_nan();
                }
            }
            if (kind != 0u) sm.q[slot] = Q[j];
            kinds |= kind << (8u * j);
        }
        // Places in the lists: this lane's counts of the three kinds (one byte
        // each), summed over the warp's lanes below, from the warp's base.
        if (__any_sync(0xffffffffu, kinds != 0u)) {
            uint32_t own = 0;
#pragma unroll
            for (uint32_t j = 0; j < LQ; ++j) {
                const uint32_t kind = (kinds >> (8u * j)) & 3u;
                own += kind != 0u ? 1u << (8u * (kind - 1u)) : 0u;
            }
            uint32_t sum = own;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += x;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, sum, 31);
            uint32_t base = 0;
            if (lane < 3u) base = atomicAdd(&sm.count[lane], (total >> (8u * lane)) & 255u);
            const uint32_t before = sum - own;
            uint32_t at1 = __shfl_sync(0xffffffffu, base, 0) + (before & 255u);
            uint32_t at2 = __shfl_sync(0xffffffffu, base, 1) + ((before >> 8) & 255u);
            uint32_t at3 = __shfl_sync(0xffffffffu, base, 2) + ((before >> 16) & 255u);
#pragma unroll
            for (uint32_t j = 0; j < LQ; ++j) {
                const uint32_t slot = pass + threadIdx.x + threads * j;
                const uint32_t kind = (kinds >> (8u * j)) & 3u;
                if (kind == 1u) sm.first[at1++] = uint16_t(slot);
                if (kind == 2u) sm.first[sm.cap - 1u - at2++] = uint16_t(slot);
                if (kind == 3u) {
                    sm.rest[at3] = uint16_t(slot);
                    sm.bound[at3++] = bound[j];
                }
            }
        }
    }
    __syncthreads();
    const uint32_t nshort = sm.count[0], nraw = sm.count[1];
#pragma unroll 1
    for (uint32_t t0 = threadIdx.x - lane; t0 < nshort; t0 += threads) {
        bool fail = false;
        uint32_t slot = 0;
        if (t0 + lane < nshort) {
            slot = sm.first[t0 + lane];
            const Pair q = sm.q[slot];
            const I l = q.x, R = q.y + 1u;
            WinBest<I> c;
            if (COLD)
                fail = !win_short_cover(w, l, R, c);
            else if (ARGMIN || w.blk != 3u)
                c = win_short<ARGMIN, 2>(w, l, R);
            else
                c = win_short<ARGMIN, 1>(w, l, R);
            if (!fail) store(c, l, slot);
        }
        if (COLD) {
            const uint32_t mf = __ballot_sync(0xffffffffu, fail);
            if (mf != 0u) {
                uint32_t base = 0;
                if (lane == 0u) base = atomicAdd(&sm.count[2], uint32_t(__popc(mf)));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (fail) {
                    const uint32_t at = base + __popc(mf & ((1u << lane) - 1u));
                    sm.rest[at] = uint16_t(slot);
                    sm.bound[at] = f_nan();
                }
            }
        }
    }
#pragma unroll 1
    for (uint32_t t = threadIdx.x; t < nraw; t += threads) {
        const uint32_t slot = sm.first[sm.cap - 1u - t];
        const Pair q = sm.q[slot];
        const I l = q.x, R = q.y + 1u;
        store(LARGE ? win_raw_long(w, l, R) : win_raw<3>(w, l, R), l, slot);
    }
    if (COLD) __syncthreads();
    const uint32_t nrest = sm.count[2];
#pragma unroll 1
    for (uint32_t t = threadIdx.x; t < nrest; t += threads) {
        const uint32_t slot = sm.rest[t];
        const Pair q = sm.q[slot];
        const I l = q.x, R = q.y + 1u;
        WinBest<I> c = win_none<I>();
        float vl = f_inf(), vr = f_inf();
        win_exact<LARGE>(w, l, R, sm.bound[t], c, vl, vr);
        win_ends<LARGE>(w, l, R, vl, vr, c);
        store(c, l, slot);
    }
    return bad;
}

// One query [l, r] by one thread.  LARGE: blocks of more than 16 entries, whose
// short queries go by win_exact as well.
template <bool LARGE, typename I>
__device__ __forceinline__ WinBest<I> win_one(const WinViewT<I>& w, I l, I r) {
    const I R = r + 1u, len = R - l;
    float bound = f_nan();
    if ((len >> (w.first - 1u)) != 0u && w.n >= (I(1) << w.first)) {
        uint32_t k;
        I a, b;
        const bool covered = win_cover(w, l, r, len, k, a, b);
        const uint2 e1 = win_entry(w, k, a), e2 = win_entry(w, k, b);
        WinBest<I> c{__uint_as_float(e1.x), win_pos(e1, a), false};
        win_take(c, __uint_as_float(e2.x), win_pos(e2, b));
        if (covered && c.p >= l && c.p <= r) return c;
        if (covered) bound = c.v;
    }
    if (!LARGE && (len >> w.first) == 0u) return w.blk == 3u ? win_short_once<1>(w, l, R) : win_short_once<2>(w, l, R);
    WinBest<I> c = win_none<I>();
    float vl = f_inf(), vr = f_inf();
    win_exact<LARGE>(w, l, R, bound, c, vl, vr);
    win_ends<LARGE>(w, l, R, vl, vr, c);
    return c;
}

}  // namespace rmq
