/* One Lame-Navier leapfrog step in the written-out operation order, for
 * bit-for-bit checks of the kernel that shares the mixed derivatives'
 * differences and adds on the integer pipe: per component c
 *   acc = 2 u_c - u_c^{n-1};
 *   acc = fma(a[c][p], (u_c(+p) + u_c(-p)) - 2 u_c, acc)         p = x, y, z
 *   acc = fma(b[c][q], (u_q(+c+q) - u_q(+c-q)) - (u_q(-c+q) - u_q(-c-q)), acc)  q != c
 * (products by 2 are exact, so contraction does not matter).  Fields x fastest;
 * component c of u, up, out at offset c * nx * ny * nz; border nodes of out 0. */
#include <math.h>

void lame_step_f64(const double* u, const double* up, double* out, int nx, int ny, int nz, const double* a,
                   const double* b) {
    const long long st[3] = {1, nx, (long long)nx * ny}, comp = st[2] * nz;
    for (int z = 0; z < nz; ++z)
        for (int y = 0; y < ny; ++y)
            for (int x = 0; x < nx; ++x) {
                const long long m = x + y * st[1] + z * st[2];
                const int border = x == 0 || y == 0 || z == 0 || x == nx - 1 || y == ny - 1 || z == nz - 1;
                for (int c = 0; c < 3; ++c) {
                    if (border) {
                        out[m + c * comp] = 0.0;
                        continue;
                    }
                    const double* uc = u + c * comp;
                    double acc = 2.0 * uc[m] - up[m + c * comp];
                    for (int p = 0; p < 3; ++p)
                        acc = fma(a[3 * c + p], (uc[m + st[p]] + uc[m - st[p]]) - 2.0 * uc[m], acc);
                    for (int q = 0; q < 3; ++q) {
                        if (q == c) continue;
                        const double* uq = u + q * comp;
                        const long long i = st[c], j = st[q];
                        acc = fma(b[3 * c + q], (uq[m + i + j] - uq[m + i - j]) - (uq[m - i + j] - uq[m - i - j]), acc);
                    }
                    out[m + c * comp] = acc;
                }
            }
}
