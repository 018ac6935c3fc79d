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
    printf("ok\n");
    return 0;
}
