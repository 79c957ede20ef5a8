// Test-only: mod_by (gw_philox.cuh) against the % operator, fastmod_magic_by
// against fastmod_magic for reciprocals off by up to four units in the last
// place, and the buckets that mark a run of positions against the bucket of every
// draw that falls in it (gw_step.cuh, warp_first_accept_runs).
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "gw_philox.cuh"

static uint64_t s = 0x9E3779B97F4A7C15ull, checked = 0;
static uint64_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }

static bool check(uint32_t d)
{
    const uint32_t m = gw::mod_magic(d);
    const uint32_t edge[] = {0u, 1u, 2u, d - 1, d, d + 1, 2 * d - 1, 2 * d, 0x7FFFFFFFu, 0x80000000u, 0xFFFFFFFEu,
                             0xFFFFFFFFu, 0xFFFFFFFFu / d * d, 0xFFFFFFFFu / d * d - 1};
    for (uint32_t a : edge) if (gw::mod_by(a, d, m) != a % d) return false;
    for (int k = 0; k < 100; ++k) {
        const uint32_t a = (uint32_t)next();
        if (gw::mod_by(a, d, m) != a % d) return false;
    }
    const uint64_t M = gw::fastmod_magic(d);
    for (int ulp = -4; ulp <= 4; ++ulp) {
        float inv = 1.0f / (float)d;
        uint32_t bits;
        memcpy(&bits, &inv, 4);
        bits += (uint32_t)ulp;
        memcpy(&inv, &bits, 4);
        if (gw::fastmod_magic_by(d, m, inv) != M) return false;
    }
    // a run [lo, hi) of positions; draws that give its first, last and some other position
    constexpr uint32_t B = 12;
    for (int k = 0; k < 8; ++k) {
        const uint32_t lo = k == 0 ? 0 : (uint32_t)(next() % d), hi = k & 1 ? d : lo + 1 + (uint32_t)(next() % (d - lo));
        const uint32_t b0 = gw::fraction_first(lo, M) >> (32 - B), b1 = gw::fraction_last(hi, M) >> (32 - B);
        for (int j = 0; j < 24; ++j) {
            const uint32_t pos = j < 8 ? lo : j < 16 ? hi - 1 : lo + (uint32_t)(next() % (hi - lo));
            const uint32_t rounds = (0xFFFFFFFFu - pos) / d;  // draws pos + i d, i <= rounds
            const uint32_t i = j % 8 == 0 ? 0 : j % 8 == 1 ? rounds : (uint32_t)(next() % ((uint64_t)rounds + 1));
            const uint32_t x = pos + i * d;
            const uint32_t b = (uint32_t)((M * x) >> (64 - B));
            if (x % d != pos || b < b0 || b > b1) return false;
            ++checked;
        }
    }
    checked += 123;
    return true;
}

int main()
{
    for (uint32_t d = 1; d <= 70000; ++d) if (!check(d)) { printf("FAIL %u\n", d); return 1; }
    for (uint32_t k = 4; k < 32; ++k)
        for (int o = -3; o <= 3; ++o) if (!check((1u << k) + (uint32_t)o)) { printf("FAIL 2^%u%+d\n", k, o); return 1; }
    for (uint32_t d : {0xFFFFFFFFu, 0xFFFFFFFEu, 0xFFFF0000u, 0xFFFF0001u, 0x80000001u, 0x55555555u, 0xAAAAAAABu, 641u, 6700417u})
        if (!check(d)) { printf("FAIL %u\n", d); return 1; }
    for (int k = 0; k < 300000; ++k) {
        const uint32_t d = (uint32_t)(next() >> (32 + next() % 32));
        if (d && !check(d)) { printf("FAIL %u\n", d); return 1; }
    }
    printf("ok %llu\n", (unsigned long long)checked);
    return 0;
}
