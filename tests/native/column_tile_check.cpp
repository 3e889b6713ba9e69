// make_column_tile (csrc/node_order.cuh): the tiles cover the inner columns,
// keep the limits that callers size their shared memory by, and come from a
// bounded search.
#include <chrono>
#include <cstdio>
#include <initializer_list>

#include "../../masterthesis_gb300/csrc/node_order.cuh"

static bool check(int ix, int iy, int rows) {
    const scafes::ColumnTile t = scafes::make_column_tile(ix, iy, rows);
    if (ix == 0 || iy == 0) return t.nx * t.ny == 0;  // no inner node
    const int w = (int)t.w.d, ty = (iy + rows - 1) / rows;
    const bool limits = w >= 1 && w <= 64 && t.h >= 1 && t.h <= 16 && w * t.h <= scafes::MARCH_THREADS;
    const bool cover = (long long)t.nx * w >= ix && (long long)(t.nx - 1) * w < ix && (long long)t.ny * t.h >= ty &&
                       (long long)(t.ny - 1) * t.h < ty;
    const bool wide = w >= 9 || w == ix;
    if (!(limits && cover && wide)) std::printf("%d x %d, %d rows: w %d h %d, %d x %d tiles\n", ix, iy, rows, w, t.h, t.nx, t.ny);
    return limits && cover && wide;
}

int main() {
    for (int rows = 1; rows <= 2; ++rows)
        for (int ix = 0; ix <= 700; ++ix)
            for (int iy : {0, 1, 2, 3, 15, 16, 17, 31, 63, 64, 98, 255, 510, 4096, 1048574})
                if (!check(ix, iy, rows)) return 1;
    for (int ix : {1022, 1023, 1024, 1025, 2047, 4095, 32765, 65534, 99999, 524286, 1048573, 1048574})
        for (int iy : {1, 2, 40, 98})
            if (!check(ix, iy, 1) || !check(ix, iy, 2)) return 1;
    // A launch per step calls it.
    const auto t0 = std::chrono::steady_clock::now();
    int sum = 0;
    for (int i = 0; i < 1000; ++i) sum += scafes::make_column_tile(1048574 - i, 1, 1).h;
    const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count() / 1000;
    std::printf("%.2f us a call (%d)\n", us, sum);
    return us > 5.0 ? 2 : 0;
}
