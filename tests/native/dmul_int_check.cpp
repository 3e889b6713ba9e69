// dmul_bits (csrc/dadd_int.cuh) against the host's FP64 multiplier: seeded
// pairs over the exponent range, short significands (ties), products near one
// and two, subnormals, zeros, infinities.  Prints the pairs and how many were
// handed back.
#include <cmath>
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
        const int kind = (int)(i % 6);
        if (kind < 4) {  // ordinary magnitudes
            a = (a & 0x800fffffffffffffull) | (uint64_t)(1000 + rnd() % 60) << 52;
            b = (b & 0x800fffffffffffffull) | (uint64_t)(1000 + rnd() % 60) << 52;
        }
        if (kind == 1) a &= ~((1ull << (20 + rnd() % 32)) - 1), b &= ~((1ull << (20 + rnd() % 32)) - 1);
        if (kind == 2) a |= 0xffffffffffff0ull, b |= rnd() & 0xfffffffffff00ull;
        if (kind == 3) {  // half-way products: odd * odd of 54 bits
            a = (a & ~0xfffffffffffffull) | (rnd() & 0x7ffffffull) << 25;
            b = (b & ~0xfffffffffffffull) | (rnd() & 0x7ffffffull) << 25;
        }
        if (kind == 5) a = (a & ~(0x7ffull << 52)) | (uint64_t)(rnd() % 4 ? rnd() % 2048 : 0) << 52;
        double c, u, got;
        memcpy(&c, &a, 8), memcpy(&u, &b, 8);
        bool ok;
        const uint64_t r = scafes::dmul_bits(scafes::make_int_factor(c), b, ok);
        memcpy(&got, &r, 8);
        const double want = c * u;
        if (ok && memcmp(&got, &want, 8) != 0) {
            std::printf("%016llx * %016llx: %a, want %a\n", (unsigned long long)a, (unsigned long long)b, got, want);
            return 1;
        }
        if (!ok && kind < 4) return 2;  // ordinary magnitudes stay on the integer path
        if (ok && !std::isnormal(want)) return 3;
        back += !ok;
    }
    std::printf("%lld %lld\n", pairs, back);
    return 0;
}
