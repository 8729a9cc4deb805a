// rmq_cl.cuh — level loads and reductions of the CL query kernels
// (rmq_query.cu).  CL reads the levels past L1: its tiles re-read the same
// sectors from L2 lane by lane, and an L1 branch cost it 2 %.
#pragma once

#include "rmq_common.cuh"

namespace rmq {

// L2 eviction priorities (tuning knobs; 0 selects the default shown).
#ifndef RMQ_L0_HINT
#define RMQ_L0_HINT 0  // level-0 sectors: 0 = evict_first, 1 = evict_normal
#endif
#ifndef RMQ_UP_HINT
#define RMQ_UP_HINT 0  // coarse-level sectors: 0 = evict_last, 1 = evict_normal
#endif
#ifndef RMQ_IDX_HINT
#define RMQ_IDX_HINT 0  // argmin index lookups: 0 = evict_last, 1 = evict_normal
#endif

struct L2Policies {
    uint64_t fine;    // level 0: read once per query
    uint64_t coarse;  // levels >= 1: shared by all queries
};

__device__ __forceinline__ uint64_t policy_evict_normal() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ L2Policies make_policies() {
    return L2Policies{RMQ_L0_HINT == 0 ? policy_evict_first() : policy_evict_normal(),
                      RMQ_UP_HINT == 0 ? policy_evict_last() : policy_evict_normal()};
}

__device__ __forceinline__ uint32_t ld_index(const uint32_t* p) {
#if RMQ_IDX_HINT == 0
    uint32_t v;
    asm("{\n\t.reg .b64 pol;\n\t"
        "createpolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
        "ld.global.nc.L2::cache_hint.u32 %0, [%1], pol;\n\t}"
        : "=r"(v) : "l"(p));
    return v;
#else
    return __ldg(p);
#endif
}

// Loads the sector starting at s of level k.  Level 0 is the caller's array,
// which is not padded: a sector that crosses its end is read element-wise.
__device__ __forceinline__ void load_level_sector(const Levels& lv, uint32_t k, uint32_t s,
                                                  const L2Policies& pol, float (&v)[8]) {
#if RMQ_DEBUG_BOUNDS
    // Level 0 is read up to its last entry; a coarse level up to its 32-entry padding.
    if (!bounds_ok(k < lv.num_levels && (s & 7u) == 0 &&
                   (k == 0 ? s < lv.size[0] : s + 8u <= ((lv.size[k] + 31u) & ~31u)))) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = f_inf();
        return;
    }
#endif
    const float* base = lv.val[k];
    if (k > 0) {
        ld_sector_policy(base + s, v, pol.coarse);
    } else if (s + 8u <= lv.size[0]) {
        ld_sector_policy(base + s, v, pol.fine);
    } else {
        const uint32_t size = lv.size[0];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (s + uint32_t(j) < size) ? base[s + j] : f_inf();
    }
}

// Minimum of v[j] for jlo <= j < jhi (+inf if empty).
__device__ __forceinline__ float sector_min(const float (&v)[8], uint32_t jlo, uint32_t jhi) {
    float w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = (uint32_t(j) >= jlo && uint32_t(j) < jhi) ? v[j] : f_inf();
    const float a = fmin3(w[0], w[1], w[2]);
    const float b = fmin3(w[3], w[4], w[5]);
    return fmin3(a, b, fminf(w[6], w[7]));
}

// Unsigned key ordered like the float's value (NaN outside the contract):
// negative values map below positive ones with their order reversed, and
// -0.0 maps to the key of +0.0, as the two compare equal.
__device__ __forceinline__ uint32_t min_key(float x) {
    const uint32_t u = x == 0.0f ? 0u : __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

}  // namespace rmq
