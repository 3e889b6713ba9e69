// dadd_bits (csrc/dadd_int.cuh) against the host's FP64 adder bit for bit, the
// sign of a zero sum included: zeros of both signs, operands that cancel, and
// near exponents.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <utility>

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
    for (long long i = 0; i < pairs; ++i) {
        uint64_t a = rnd(), b = rnd();
        const int kind = (int)(i % 4);
        if (kind < 2) {
            const int e = 1 + (int)(rnd() % 2045);
            int f = e + (int)(rnd() % 19) - 9;
            f = f < 1 ? 1 : f > 2045 ? 2045 : f;
            a = (a & 0x800fffffffffffffull) | (uint64_t)e << 52;
            b = (b & 0x800fffffffffffffull) | (uint64_t)f << 52;
            if (kind == 1) b = a ^ (1ull << 63);  // cancels
        } else if (kind == 2) {  // zeros of both signs
            a &= 1ull << 63, b &= 1ull << 63;
        } else {
            a &= 1ull << 63;
            if (rnd() & 1) std::swap(a, b);
        }
        bool ok;
        const uint64_t got = scafes::dadd_bits(a, b, ok);
        double x, y, w;
        memcpy(&x, &a, 8), memcpy(&y, &b, 8);
        w = x + y;
        uint64_t want;
        memcpy(&want, &w, 8);
        if (kind < 3 && kind != 0 && !ok && (a >> 52 & 0x7ff) < 2046) return 2;  // zero sums stay on this path
        if (ok && got != want) {
            std::printf("%016llx + %016llx = %016llx, want %016llx\n", (unsigned long long)a, (unsigned long long)b,
                        (unsigned long long)got, (unsigned long long)want);
            return 1;
        }
    }
    return 0;
}
