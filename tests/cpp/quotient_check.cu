// The quotient on the integer units (csrc/fp64_int.cuh) against the host's division: every
// bit, for mantissas of all kinds and whatever the first reciprocal's error (2^-22) is.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "fp64_int.cuh"

static double from_bits(uint64_t b)
{
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}
static uint64_t to_bits(double d)
{
    uint64_t b;
    std::memcpy(&b, &d, 8);
    return b;
}

int main()
{
    std::mt19937_64 rng(7);
    const uint64_t M = (1ull << 52) - 1;
    auto mantissa = [&](int kind) -> uint64_t {
        const uint64_t r = rng();
        switch (kind) {
        case 0: return r & M;
        case 1: return r & 0xFFFF;                       // just above a power of two
        case 2: return M - (r & 0xFFFF);                 // just below one
        case 3: return (r & M) & ~((1ull << (r >> 58)) - 1) & M;  // few bits
        default: return ((1ull << (r & 63) % 52) - 1) & M;
        }
    };
    long long n = 0;
    for (int i = 0; i < 8000000; ++i) {
        uint64_t a = ((uint64_t)(1023 + rng() % 900) << 52) | mantissa(i % 5);
        uint64_t b = ((uint64_t)(1023 + rng() % 64) << 52) | mantissa((i / 5) % 5);
        if (i % 3 == 0) {  // quotients next to the middle of two doubles
            const double q = from_bits((uint64_t)1023 << 52 | mantissa(0)), d = from_bits(b);
            a = to_bits(q * d);  // a near q d: then by a unit up or down
            a += (uint64_t)(int64_t)((int)(rng() % 3) - 1);
            if (a >> 52 < 1023) continue;
        }
        const uint64_t mb = (b & M) | (M + 1);
        const double r = 9223372036854775808.0 / (double)(mb >> 21);
        const double off = 1.0 + ((double)(int64_t)(rng() % 2001) - 1000.0) / 1000.0 / 4194304.0;
        double r0 = r * off;
        if (r0 > 4294967295.0) r0 = 4294967295.0;
        const uint64_t got = gu::quotient_bits(a, b, (unsigned)r0), want = to_bits(from_bits(a) / from_bits(b));
        if (got != want) {
            std::printf("%.17g / %.17g: %016llx, not %016llx\n", from_bits(a), from_bits(b), (unsigned long long)got,
                        (unsigned long long)want);
            return 1;
        }
        ++n;
    }
    std::printf("%lld quotients\n", n);
    return n > 7000000 ? 0 : 1;
}
