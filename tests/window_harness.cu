// Host side of the window-table query's index arithmetic (rmq_window.cuh),
// 32-bit positions against 64-bit ones.  Prints the number of pairs checked
// and of those that differ; argv[1]: the tables' form.
#include <cstdio>
#include <cstdlib>

#include "rmq_window.cuh"

using namespace rmq;

static uint64_t checked = 0, wrong = 0;

static void report(const char* what, uint64_t l, uint64_t R) {
    if (++wrong <= 5) std::printf("%s l %llu R %llu\n", what, (unsigned long long)l, (unsigned long long)R);
}

static void check(const WinView& w32, const WinView64& w64, uint64_t l, uint64_t R) {
    ++checked;
    uint32_t x32, y32;
    uint64_t x64, y64;
    const bool large = w32.blk > 4;
    const bool a = large ? win_inner<true>(uint32_t(l), uint32_t(R), w32.gb, x32, y32)
                         : win_inner<false>(uint32_t(l), uint32_t(R), w32.gb, x32, y32);
    const bool b = win_inner<true>(l, R, w64.gb, x64, y64);
    if (a != b || (a && (x32 != x64 || y32 != y64 || y64 < x64 || y64 - x64 < uint64_t(8) << w64.gb)))
        report("inner", l, R);
    const uint64_t len = R - l;
    if ((len >> (w32.first - 1u)) == 0) return;
    uint32_t k32, k64, s1, s2;
    uint64_t t1, t2;
    const bool c = win_cover(w32, uint32_t(l), uint32_t(R - 1), uint32_t(len), k32, s1, s2);
    const bool d = win_cover(w64, l, R - 1, len, k64, t1, t2);
    const uint64_t W = uint64_t(1) << k64;
    const bool covers = t1 <= l && t2 <= t1 + W && R <= t2 + W && t2 < R && k64 <= w64.kmax;
    if (c != d || k32 != k64 || s1 != t1 || s2 != t2 || !d || !covers) report("cover", l, R);
}

int main(int argc, char** argv) {
    const uint32_t form = argc > 1 ? uint32_t(std::atoi(argv[1])) : 0u;
    const uint64_t n = 0xFFFFFF00ull;  // the largest array with 32-bit positions
    const WinView w32 = win_view<uint32_t>(nullptr, nullptr, n, form);
    const WinView64 w64 = win_view<uint64_t>(nullptr, nullptr, n, form);
    for (uint64_t l = n - 4096; l < n; ++l)
        for (uint64_t R = l + 1; R <= n; ++R) check(w32, w64, l, R);
    uint64_t h = 1;  // lengths up to n, starts anywhere
    for (int i = 0; i < 2000000; ++i) {
        h = h * 6364136223846793005ull + 1442695040888963407ull;
        const uint64_t len = 1 + (h >> 32) % (i % 3 ? n : uint64_t(1) << (1 + i % 32));
        h = h * 6364136223846793005ull + 1442695040888963407ull;
        if (len > n) continue;
        const uint64_t l = i % 5 ? (h >> 31) % (n - len + 1) : n - len - (h >> 40) % (n - len < 600 ? n - len + 1 : 600);
        check(w32, w64, l, l + len);
    }
    std::printf("checked %llu wrong %llu\n", (unsigned long long)checked, (unsigned long long)wrong);
    return 0;
}
