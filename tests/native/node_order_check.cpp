// Walks the node numbers of a grid (csrc/node_order.cuh) against plain
// loops: every inner and border node once, in Fortran order.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "../../masterthesis_gb300/csrc/node_order.cuh"

int main(int argc, char** argv) {
    for (int a = 1; a + 3 < argc; a += 4) {
        const int nx = atoi(argv[a]), ny = atoi(argv[a + 1]), nz = atoi(argv[a + 2]), nl = atoi(argv[a + 3]);
        const scafes::NodeOrder o = scafes::make_node_order(nx, ny, nz, nl);
        uint32_t i = 0, b = 0;
        for (int z = 0; z < nz; ++z)
            for (int y = 0; y < ny; ++y)
                for (int x = 0; x < nx; ++x) {
                    const bool border = x < nl || x >= nx - nl || y < nl || y >= ny - nl || z < nl || z >= nz - nl;
                    int p, q, r;
                    if (border) scafes::border_node(o, b++, p, q, r);
                    else scafes::inner_node(o, i++, p, q, r);
                    if (p != x || q != y || r != z) {
                        std::printf("%d x %d x %d, %d layers: (%d, %d, %d) read as (%d, %d, %d)\n", nx, ny, nz, nl, x,
                                    y, z, p, q, r);
                        return 1;
                    }
                }
        if (i != o.n_inner || b != o.n_border) return 2;
    }
    // The division at the top of its range.
    for (uint32_t d : {1u, 2u, 3u, 7u, 641u, 65535u, 1048575u, 1u << 20, 2147483647u})
        for (uint32_t n = 0x7fffffffu; n > 0x7fffffffu - 5000; --n)
            if (scafes::fastdiv(n, scafes::make_fastdiv(d)) != n / d) return 3;
    std::puts("ok");
    return 0;
}
