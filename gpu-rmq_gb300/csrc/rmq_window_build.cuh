// rmq_window_build.cuh — device functions of the window-table build, shared by
// the single-array kernels (rmq_window.cu) and the batched ones (rmq_batch.cu).
//
// One streaming pass over level 0 writes the minimum and its offset for every
// block (0.31 n bytes with blocks of 16 entries); everything above is computed
// from those, which are still in L2.  A tile pass holds 2048 strides and a halo
// of 512 in shared memory and makes every table whose windows fit the halo; a
// second tile pass does the same for the next six sizes; one CTA makes the few
// entries above.  Small arrays take smaller tiles, straight from level 0, and
// that last CTA.  Each table is one doubling of the one below:
// T_(k+1)[i] = first minimum of T_k[2i] and T_k[2i + windows per stride].
#pragma once

#include "rmq_window.cuh"

namespace rmq {

constexpr uint32_t kBlockTile = 8192;      // level-0 entries per CTA of the block pass
constexpr uint32_t kBlockThreads = 256;
constexpr uint32_t kLowThreads = 512;
constexpr uint32_t kMidThreads = 1024;
constexpr uint32_t kSpan = 2048;           // own strides per tile of the window kernels
constexpr uint32_t kHaloLow = 512;         // halo of the first window kernel, in strides of 2^gb
constexpr uint32_t kHaloMid = 1024;        // halo of the second, in its input's strides
constexpr uint32_t kTopEntries = 4096;     // entries the last kernel holds in shared memory
constexpr uint32_t kMidSteps = 6;          // sizes the second window kernel adds

// Largest window the first kernel makes from a tile and its halo (512 strides
// of 2^gb), and the second (its halo: 2^kMidSteps windows of that size).
template <typename V>
__host__ __device__ __forceinline__ uint32_t win_low_log(const V& w) { return w.gb + 9u; }
template <typename V>
__host__ __device__ __forceinline__ uint32_t win_mid_log(const V& w) { return w.gb + 9u + kMidSteps; }

// Blocks of a warp's 1024 values from `base`, handed to put(block, minimum,
// offset).  A load covers 32 consecutive sectors (1 KiB); each lane takes its
// sector's first minimum, and the two lanes of a block exchange one sector each
// of two loads, so that every lane ends with one whole block and a warp stores
// 32 consecutive blocks.  LARGE: blocks of 32 or 64 entries, four or eight lanes
// each.
template <bool LARGE, typename Put>
__device__ __forceinline__ void win_block_part(const WinOut& w, uint64_t base, const Put& put) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t sec0 = (base >> 3) + lane;
    const uint64_t pol = policy_evict_first();
    float v[4][8];
    if (base + 1024u <= w.n) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) ld_sector_policy(w.a + 8u * (sec0 + 32u * i), v[i], pol);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const uint64_t s = 8u * (sec0 + 32u * i);
            if (s + 8u <= w.n) {
                ld_sector_policy(w.a + s, v[i], pol);
            } else {
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) v[i][j] = s + j < w.n ? w.a[s + j] : f_inf();
            }
        }
    }
    float m[4];
    uint32_t off[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
        const float x = fmin3(fmin3(v[i][0], v[i][1], v[i][2]), fmin3(v[i][3], v[i][4], v[i][5]),
                              fminf(v[i][6], v[i][7]));
        uint32_t j = 0;
        float mv = v[i][0];  // the first equal entry's own bits (a zero keeps its sign)
#pragma unroll
        for (int jj = 7; jj >= 0; --jj) {
            if (v[i][jj] == x) {
                j = uint32_t(jj);
                mv = v[i][jj];
            }
        }
        m[i] = mv;
        off[i] = j;
    }
    if (LARGE) {
        const uint32_t sectors = 1u << (w.blk - 3u);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            off[i] += 8u * (lane & (sectors - 1u));
            for (uint32_t o = 1; o < sectors; o <<= 1) {
                const float ov = __shfl_down_sync(0xffffffffu, m[i], o);
                const uint32_t oo = __shfl_down_sync(0xffffffffu, off[i], o);
                if (ov < m[i]) {  // the first lane of each 2 o: equal, its entry stays
                    m[i] = ov;
                    off[i] = oo;
                }
            }
            const uint64_t sec = sec0 + 32u * i;
            if ((lane & (sectors - 1u)) == 0u && (sec << 3) < w.n) put(sec >> (w.blk - 3u), m[i], off[i]);
        }
        return;
    }
    if (w.blk == 3u) {  // a sector is a block
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            const uint64_t blk = sec0 + 32u * i;
            if ((blk << 3) < w.n) put(blk, m[i], off[i]);
        }
        return;
    }
    const bool odd = (lane & 1u) != 0u;
#pragma unroll
    for (uint32_t p = 0; p < 4; p += 2) {
        const float mine = odd ? m[p + 1] : m[p];
        const uint32_t mo = odd ? off[p + 1] : off[p];
        const float other = __shfl_xor_sync(0xffffffffu, odd ? m[p] : m[p + 1], 1);
        const uint32_t oo = __shfl_xor_sync(0xffffffffu, odd ? off[p] : off[p + 1], 1);
        const float lov = odd ? other : mine, hiv = odd ? mine : other;
        const uint32_t loo = odd ? oo : mo, hio = odd ? mo : oo;
        const bool hi = hiv < lov;  // equal: the first sector's entry stays
        const uint64_t blk = (sec0 + 32u * (odd ? p + 1u : p)) >> 1;
        if ((blk << 4) < w.n) put(blk, hi ? hiv : lov, hi ? 8u + hio : loo);
    }
}

// Blocks of one tile, by kBlockThreads threads.
template <bool LARGE>
__device__ __forceinline__ void win_block_tile(const WinOut& w, uint64_t tile) {
    win_block_part<LARGE>(w, tile * kBlockTile + (threadIdx.x >> 5) * 1024u, [&](uint64_t blk, float m, uint32_t off) {
        w.v1[blk] = m;
        w.j1[blk] = uint8_t(off);
    });
}

// First minimum of two entries; hi_off: what the upper one's offset gains (0
// for positions).
__device__ __forceinline__ uint2 win_first(uint2 lo, uint2 hi, uint32_t hi_off) {
    return __uint_as_float(hi.x) < __uint_as_float(lo.x) ? make_uint2(hi.x, hi.y + hi_off) : lo;
}

// Doubles T_k held in `src` (`cnt` entries from entry `at` of T_k) up to
// T_(last), writing each table's own entries (the tile's kSpan strides of the
// first source) to the table and keeping them in shared memory in turn.
// Entries whose window starts at or past n do not exist and are never read.
__device__ __forceinline__ void win_double_up(const WinOut& w, uint32_t k, uint32_t last, uint64_t at, uint32_t cnt,
                                              uint32_t own, uint2* src, uint2* dst) {
    const uint32_t wpu = 1u << w.c;
    for (; k < last; ++k) {
        const uint32_t s = win_stride_log(w, k + 1u);
        const uint32_t half = 1u << k, off = w.wide ? half : 0u;  // k < 32
        cnt >>= 1;
        own >>= 1;
        at >>= 1;
        uint2* out = w.t + win_table_at<uint64_t>(w, k + 1u) + at;
        for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
            const uint64_t start = (at + i) << s;
            if (start >= w.n) break;
            uint2 e = src[2u * i];
            const uint32_t h = 2u * i + wpu;
            if (h < 2u * cnt && start + half < w.n) e = win_first(e, src[h], off);
            dst[i] = e;
            if (i < own) out[i] = e;
        }
        __syncthreads();
        uint2* x = src;
        src = dst;
        dst = x;
    }
}

// First minimum of the blocks of stride g (g < S), as an entry of T.  EIGHT: a
// stride is eight blocks, else two or four.
template <bool EIGHT>
__device__ __forceinline__ uint2 win_group(const WinOut& w, uint64_t g) {
    constexpr uint32_t kMost = EIGHT ? 8u : 4u;
    const uint32_t bpg = EIGHT ? 8u : 1u << (w.gb - w.blk);
    const uint64_t nb = (w.n + (uint64_t(1) << w.blk) - 1) >> w.blk, b = g * bpg;
    float v[kMost];
    uint64_t off;
    // V1 and J1 are padded to 32 bytes, so a whole stride of either can be read
    if (EIGHT) {
        const float4 x = *reinterpret_cast<const float4*>(w.v1 + b), y = *reinterpret_cast<const float4*>(w.v1 + b + 4);
        v[0] = x.x;
        v[1] = x.y;
        v[2] = x.z;
        v[3] = x.w;
        v[kMost - 4] = y.x;
        v[kMost - 3] = y.y;
        v[kMost - 2] = y.z;
        v[kMost - 1] = y.w;
        off = *reinterpret_cast<const uint64_t*>(w.j1 + b);
    } else if (bpg == 2u) {
        const float2 x = *reinterpret_cast<const float2*>(w.v1 + b);
        v[0] = x.x;
        v[1] = x.y;
        v[2] = v[3] = f_inf();
        off = *reinterpret_cast<const uint16_t*>(w.j1 + b);
    } else {
        const float4 x = *reinterpret_cast<const float4*>(w.v1 + b);
        v[0] = x.x;
        v[1] = x.y;
        v[2] = x.z;
        v[3] = x.w;
        off = *reinterpret_cast<const uint32_t*>(w.j1 + b);
    }
    uint2 e = make_uint2(__float_as_uint(v[0]), uint32_t(off) & 255u);
#pragma unroll
    for (uint32_t c = 1; c < kMost; ++c)
        if (c < bpg && b + c < nb)
            e = win_first(e, make_uint2(__float_as_uint(v[c]), uint32_t(off >> (8u * c)) & 255u), c << w.blk);
    if (!w.wide) e.y += uint32_t(b << w.blk);
    return e;
}

// The tables up to T_(gb + log2 HALO) (all of them when the array has one tile)
// of a tile's SPAN strides from g0, by THREADS threads; group(i, g): the entry
// of stride g, the tile's i-th.  A tile is a chain of some ten steps with a
// barrier each, so its time is their latency: every thread keeps its entries in
// registers, all loads of a step in flight (one tile of kSpan strides: 16 ->
// 8.5 us against one entry after another with 256 threads).
template <uint32_t SPAN, uint32_t HALO, uint32_t THREADS, typename Group>
__device__ __forceinline__ void win_tile_tables(const WinOut& w, uint64_t g0, uint32_t top, uint2* sa, uint2* sb,
                                                const Group& group) {
    constexpr uint32_t kPer = (SPAN + HALO) / THREADS;
    uint2 e[kPer];
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint64_t g = g0 + threadIdx.x + THREADS * u;
        if (g < w.S) e[u] = group(threadIdx.x + THREADS * u, g);
    }
    // Windows of 2, 4, 8 strides (2^first entries), the last one the first
    // table; where the next one has the same stride, a doubling of 8.
    uint2 *src = sa, *dst = sb;
    const uint32_t kb = w.gb + w.c;
    for (uint32_t d = 1;; d <<= 1) {
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) src[threadIdx.x + THREADS * u] = e[u];
        __syncthreads();
        if (d > (w.first < kb ? 8u : 4u)) break;
        uint2* out = nullptr;
        if (d == 4u) out = w.t + win_table_at<uint64_t>(w, w.first) + g0;
        if (d == 8u && w.kmax >= kb) out = w.t + win_table_at<uint64_t>(w, kb) + g0;
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) {
            const uint32_t i = threadIdx.x + THREADS * u;
            if (g0 + i + d < w.S && i + d < SPAN + HALO) e[u] = win_first(e[u], src[i + d], w.wide ? d << w.gb : 0u);
            if (out != nullptr && i < SPAN && g0 + i < w.S) out[i] = e[u];
        }
        uint2* x = src;
        src = dst;
        dst = x;
    }
    const uint32_t last = w.S <= SPAN ? w.kmax : (w.kmax < top ? w.kmax : top);
    win_double_up(w, kb, last, g0, SPAN + HALO, SPAN, src, dst);
}

// The tables up to T_(gb+9) of one tile, from V1 and J1.
template <bool EIGHT>
__device__ __forceinline__ void win_low_tile(const WinOut& w, uint64_t tile, uint2* sa, uint2* sb) {
    win_tile_tables<kSpan, kHaloLow, kLowThreads>(w, tile * kSpan, win_low_log(w), sa, sb,
                                                  [&](uint32_t, uint64_t g) { return win_group<EIGHT>(w, g); });
}

// Small arrays (kFormArgmin and kFormSmallMin, up to kSmallN entries) are built
// by one kernel from level 0 and, above one tile, one CTA for the sizes above:
// what such a build costs is its launches and the chain of steps in each, not
// bytes.  A tile is HALO strides of 32 values of its own and as many behind
// them, whose blocks it computes again: 128 keep the chain short, but leave
// n / 2^8 entries to the last CTA, which holds 4096, so above 2^20 values (and
// for the one tile of 2^12 to 2^14) it is 512.  Device time of rmq_build for
// 1000, 2^14, 2^18, 2^20 and 2^22 values, us: 10.5, 11.9, 14.6, 16.2 and 20.6; with
// the kernels for large arrays 13.8, 14.9, 19.4, 20.7 and 23.1; the block-minimum
// levels took 11.1, 11.1, 13.4, 14.1 and 17.8.
constexpr uint64_t kShortHaloN = uint64_t(1) << 20;
constexpr uint32_t kShortHalo = 128, kLongHalo = 512;
template <uint32_t HALO>
__host__ __device__ constexpr uint32_t win_small_threads() { return HALO == kShortHalo ? 256u : 512u; }

template <uint32_t HALO>
struct WinSmallShared {
    float v1[8 * HALO];  // up to four blocks per stride
    uint8_t j1[8 * HALO];
    uint2 a[2 * HALO], b[2 * HALO];
};

template <uint32_t HALO>
__device__ __forceinline__ void win_small_tile(const WinOut& w, uint64_t tile, WinSmallShared<HALO>& sm) {
    constexpr uint32_t kThreads = win_small_threads<HALO>(), kWarps = kThreads / 32u;
    const uint64_t g0 = tile * HALO;
    const uint32_t bpg = 1u << (w.gb - w.blk);  // blocks per stride: 2 or 4
    const uint64_t b0 = g0 * bpg, nb = (w.n + (uint64_t(1) << w.blk) - 1) >> w.blk;
#pragma unroll 1
    for (uint32_t part = threadIdx.x >> 5; part < HALO / 16u; part += kWarps) {  // 32 strides a part
        const uint64_t base = (g0 << w.gb) + part * 1024u;
        if (base >= w.n) break;
        win_block_part<false>(w, base, [&](uint64_t blk, float m, uint32_t off) {
            const uint32_t i = uint32_t(blk - b0);
            sm.v1[i] = m;
            sm.j1[i] = uint8_t(off);
            if (i < HALO * bpg) {
                w.v1[blk] = m;
                w.j1[blk] = uint8_t(off);
            }
        });
    }
    if (w.n < (uint64_t(1) << w.first)) return;
    __syncthreads();
    win_tile_tables<HALO, HALO, kThreads>(w, g0, w.gb + (HALO == kShortHalo ? 7u : 9u), sm.a, sm.b, [&](uint32_t i, uint64_t g) {
        const uint32_t b = i * bpg;
        uint2 e = make_uint2(__float_as_uint(sm.v1[b]), sm.j1[b]);
        for (uint32_t c = 1; c < bpg && g * bpg + c < nb; ++c)
            e = win_first(e, make_uint2(__float_as_uint(sm.v1[b + c]), sm.j1[b + c]), c << w.blk);
        if (!w.wide) e.y += uint32_t(g << w.gb);
        return e;
    });
}


// The next kMidSteps tables above T_(gb+9) of one tile of its entries.
__device__ __forceinline__ void win_mid_tile(const WinOut& w, uint64_t tile, uint2* sa, uint2* sb) {
    const uint32_t k = win_low_log(w), s = win_stride_log(w, k);
    const uint64_t e0 = tile * kSpan;
    const uint32_t cnt = kSpan + kHaloMid;
    const uint64_t entries = (w.n + (uint64_t(1) << s) - 1) >> s;
    const uint2* src = w.t + win_table_at<uint64_t>(w, k) + e0;
    constexpr uint32_t kPer = (kSpan + kHaloMid) / kMidThreads;
    uint2 e[kPer];
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t i = threadIdx.x + kMidThreads * u;
        if (e0 + i < entries) e[u] = __ldcg(src + i);
    }
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) sa[threadIdx.x + kMidThreads * u] = e[u];
    __syncthreads();
    const uint32_t last = entries <= kSpan ? w.kmax : (w.kmax < win_mid_log(w) ? w.kmax : win_mid_log(w));
    win_double_up(w, k, last, e0, cnt, kSpan, sa, sb);
}

// CTAs of each build kernel for one array (0: not needed).
struct WinTiles {
    uint64_t block, low, mid, top;
};
inline WinTiles win_tiles(const WinShape& w) {
    WinTiles t{(w.n + kBlockTile - 1) / kBlockTile, 0, 0, 0};
    if (w.t_entries == 0) return t;
    t.low = (w.S + kSpan - 1) / kSpan;
    if (t.low == 1 || w.kmax <= win_low_log(w)) return t;
    const uint32_t s = win_stride_log(w, win_low_log(w));
    t.mid = (((w.n + (uint64_t(1) << s) - 1) >> s) + kSpan - 1) / kSpan;
    t.top = t.mid > 1 && w.kmax > win_mid_log(w) ? 1 : 0;
    return t;
}

// The tables above T_k0, by one CTA of kMidThreads: from shared memory where its
// entries fit there (k0 = win_mid_log: up to 2^28 values), else each table from
// the one below in global memory.
__device__ __forceinline__ void win_top(const WinOut& w, uint32_t k0, uint2* sa, uint2* sb) {
    const uint32_t s0 = win_stride_log(w, k0);
    const uint64_t have = (w.n + (uint64_t(1) << s0) - 1) >> s0;
    const uint2* from = w.t + win_table_at<uint64_t>(w, k0);
    if (have <= kTopEntries) {
#pragma unroll
        for (uint32_t u = 0; u < kTopEntries / kMidThreads; ++u) {
            const uint32_t i = threadIdx.x + kMidThreads * u;
            if (i < have) sa[i] = __ldcg(from + i);
        }
        __syncthreads();
        win_double_up(w, k0, w.kmax, 0, kTopEntries, kTopEntries, sa, sb);
        return;
    }
    const uint32_t wpu = 1u << w.c;
    for (uint32_t k = k0; k < w.kmax; ++k) {
        const uint32_t s = win_stride_log(w, k + 1u);
        const uint64_t entries = (w.n + (uint64_t(1) << s) - 1) >> s;
        const uint2* src = w.t + win_table_at<uint64_t>(w, k);
        uint2* dst = w.t + win_table_at<uint64_t>(w, k + 1u);
        const uint64_t half = uint64_t(1) << k;
        for (uint64_t i = threadIdx.x; i < entries; i += blockDim.x) {
            uint2 e = __ldcg(src + 2u * i);
            if ((i << s) + half < w.n) e = win_first(e, __ldcg(src + 2u * i + wpu), w.wide ? uint32_t(half) : 0u);
            dst[i] = e;
        }
        __syncthreads();
    }
}

}  // namespace rmq
