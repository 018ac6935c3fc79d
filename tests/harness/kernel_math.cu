// Host-side checks of the arithmetic that the kernels share with the host (no
// CUDA call is made; nothing needs a GPU).  Prints "ok" or the first failure.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "gxy_device.cuh"

using namespace gxy;

static int fail(const char* what, unsigned long long a, unsigned long long b) {
    printf("%s: %llu, expected %llu\n", what, a, b);
    return 1;
}

int main() {
    // The hits of a group as k_enumerate sums them: every lane its entries, the
    // halves across the warp, then the reservation against the buffer.
    const struct {
        uint32_t lanes, entries, size;
    } cases[] = {{32, 1, 1},           {32, 16, 14},          {32, 1, 140000000u},  {32, 1, (1u << 27) - 1},
                 {32, 1, 1u << 27},    {32, 16, 0xffffffffu}, {1, 1, 0xffffffffu},  {2, 1, 0x80000000u},
                 {32, 14, 0x0001ffffu}, {32, 14, 0xffff0000u}};
    for (const auto& c : cases) {
        uint64_t want = 0;
        HitSum warp;
        for (uint32_t l = 0; l < c.lanes; l++) {
            HitSum lane;
            for (uint32_t e = 0; e < c.entries; e++) {
                lane.add(c.size - (e & 1u));   // (sizes that differ)
                want += c.size - (e & 1u);
            }
            warp.lo += lane.lo;
            warp.hi += lane.hi;
        }
        if (warp.total() != want) return fail("hits of a group", warp.total(), want);
        for (uint64_t cap : {4096ull, 268435456ull, 4294967295ull})
            for (uint64_t base : {0ull, 1ull, 4095ull, 4096ull, 268435455ull, 300000000ull, 5000000000ull}) {
                const bool inside = (unsigned __int128)base + want <= cap;
                if (hits_fit(base, want, cap) != inside) return fail("reservation", want, cap);
            }
    }
    if (hits_fit(~0ull - 1, 5, 4096)) return fail("reservation past 2^64", 1, 0);
    // The windows of every span of 16 positions, against the multiples of the step.
    for (uint64_t step : {1ull, 2ull, 3ull, 7ull, 15ull, 16ull, 17ull, 100ull, 65536ull, 0x80000000ull, 0xfffffff0ull,
                          0xfffffff8ull, 0xfffffff9ull, 0xffffffffull}) {
        for (uint64_t windows : {1ull, 2ull, 3ull, 50ull}) {
            const uint64_t last = (windows - 1) * step;
            if (last > 0xffffffffull) continue;
            std::vector<uint64_t> got;
            for (uint64_t w = 0; w < windows; w++)   // the spans that hold one, and their neighbours
                for (int64_t x = (int64_t)(w * step / 16) - 1; x <= (int64_t)(w * step / 16) + 1; x++) {
                    if (x < 0 || (uint64_t)x > last / 16 || (got.size() && got.back() / 16 >= (uint64_t)x)) continue;
                    const SpanWindows at((uint64_t)x * 16, last, (uint32_t)step, 16);
                    if (at.first < 16)
                        for (uint32_t j = at.first; j < at.stop; j += at.stride) got.push_back((uint64_t)x * 16 + j);
                }
            if (got.size() != windows) return fail("windows of a span", got.size(), windows);
            for (uint64_t w = 0; w < windows; w++)
                if (got[w] != w * step) return fail("window", got[w], w * step);
        }
    }
    printf("ok\n");
    return 0;
}
