// dadd_bits (csrc/dadd_int.cuh) against the host's FP64 adder: seeded pairs of
// any signs around equal exponents (cancellation, ties, carries), zeros,
// subnormals and the ends of the exponent range.  Prints the pairs checked
// and how many were handed back.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../masterthesis_gb300/csrc/dadd_int.cuh"

static uint64_t state;
static uint64_t rnd() {  // splitmix64
    uint64_t z = (state += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

int main(int argc, char** argv) {
    state = strtoull(argv[1], nullptr, 10);
    const long long pairs = atoll(argv[2]);
    long long back = 0;
    for (long long i = 0; i < pairs; ++i) {
        uint64_t a = rnd(), b = rnd();
        const unsigned kind = (unsigned)(i % 8);
        if (kind < 6) {  // near exponents: d from -11 to 11
            const int ea = kind == 5 ? (int)(rnd() % 2048) : 300 + (int)(rnd() % 1400);
            int eb = ea + (int)(rnd() % 23) - 11;
            eb = eb < 0 ? 0 : eb > 2047 ? 2047 : eb;
            a = (a & 0x800fffffffffffffull) | (uint64_t)ea << 52;
            b = (b & 0x800fffffffffffffull) | (uint64_t)eb << 52;
            if (kind == 1) b = (a ^ (1ull << 63)) + (rnd() % 9) - 4;      // almost cancels
            if (kind == 2) a &= ~0xffffffull, b &= ~0xffffffull;          // ties
            if (kind == 3) a |= 0xfffffffffffffull, b |= rnd() & 0xfffffffffffffull;
            if (kind == 5 && i % 16 == 5) b = a ^ (1ull << 63);            // cancels, infinities and NaNs too
        } else if (kind == 6) {
            if (rnd() & 1) a &= 1ull << 63;
            if (rnd() & 1) b &= 1ull << 63;
        } else {
            b &= 0x800fffffffffffffull;  // subnormal
        }
        bool ok;
        const uint64_t r = scafes::dadd_bits(a, b, ok);
        double x, y, w, got;
        memcpy(&x, &a, 8), memcpy(&y, &b, 8), memcpy(&got, &r, 8);
        w = x + y;
        const unsigned ea = (a >> 52) & 0x7ff, eb = (b >> 52) & 0x7ff, big = ea > eb ? ea : eb, small = ea > eb ? eb : ea;
        const bool want_ok = (big - small <= 9 || small == 0) && ((big >= 64 && big <= 2045) || w == 0.0);
        if (ok != want_ok || (ok && !(got == w))) {
            std::printf("%016llx + %016llx = %016llx (%g, want %g), ok %d\n", (unsigned long long)a,
                        (unsigned long long)b, (unsigned long long)r, got, w, ok);
            return 1;
        }
        back += !ok;
    }
    std::printf("%lld %lld\n", pairs, back);
    return 0;
}
