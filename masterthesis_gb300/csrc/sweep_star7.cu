// Plain 7-point sweep: one launch advances the whole grid by one time step.
//
// Replaces the per-node loop of ScaFES's evalTypeTwoAt
// (src/ScaFES_Problem.hpp:5399-5476) for the heat-type callbacks
// (tests/system/HeatEqnFDM/HeatEqnFDM.hpp:205-218,
//  tests/system/PennesBioheatEqnFDM/PennesBioheatEqnFDM.hpp:153-168) and
// their Dirichlet border (.../Dirichlet/Dirichlet.hpp:125-131), and the copy
// old->new that precedes it (:5078-5082): every node is written each step.
// Each CTA runs one tile (star7_tile.cuh) over a chunk of z-planes; the
// kernels are instantiated per element type in sweep_star7_{f64,f32x2,f32}.cu.
// This file holds the host helpers and the dispatch on the element type.
#include "star7_tb.cuh"
#include "star7_tile.cuh"

namespace scafes {

Star7Coeffs make_star7_coeffs(double c0, const double cp[3], double cf) {
    Star7Coeffs c;
    c.c0 = c0; c.cx = cp[0]; c.cy = cp[1]; c.cz = cp[2]; c.cf = cf;
    auto split3 = [](double v, float& h, float& l, float& ll) {
        h = (float)v;
        double r = v - (double)h;
        l = (float)r;
        ll = (float)(r - (double)l);
    };
    split3(c0, c.c0h, c.c0l, c.c0ll);
    split3(cp[0], c.cxh, c.cxl, c.cxll);
    split3(cp[1], c.cyh, c.cyl, c.cyll);
    split3(cp[2], c.czh, c.czl, c.czll);
    split3(cf, c.cfh, c.cfl, c.cfll);
    return c;
}

int star7_box_width(int precision) {
    return BX + 2 * (16 / (int)element_size(precision));
}

int star7_box_height(int tile) {
    return kTiles[tile].by + 2;
}

int star7_default_tile(const Layout& L, int precision) {
    // FP64: one row per thread (the integer-pipe sums want resident warps,
    // not registers; the autotuner's choice at every size measured).  Else
    // four rows per thread once the grid has enough tiles to fill the GPU.
    if (precision == SCAFES_PREC_F64) return 0;
    const long long cols = (long long)L.nx * L.ny;
    return cols >= 256LL * 256LL ? 2 : 0;
}

cudaError_t launch_star7_f64(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_f32(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_f32x2(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_tb_f64(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_tb_f32(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_tb_f32x2(const Star7Launch& a, cudaStream_t stream);
cudaError_t prepare_star7_tb_f64();
cudaError_t prepare_star7_tb_f32();
cudaError_t prepare_star7_tb_f32x2();

bool star7_tb_eligible(const Star7Launch& a) {
    return a.border == SCAFES_BORDER_DIRICHLET && a.L.nl == 1 && a.fb == nullptr && !a.vc;
}

void star7_tb_box(int precision, int* width, int* rows) {
    const int esz = (int)element_size(precision);
    *width = tb_bw(esz);
    *rows = TB_BH;
}

cudaError_t launch_star7_tb(const Star7Launch& a, cudaStream_t stream) {
    switch (a.precision) {
        case SCAFES_PREC_F64: return launch_star7_tb_f64(a, stream);
        case SCAFES_PREC_F32: return launch_star7_tb_f32(a, stream);
        case SCAFES_PREC_F32X2: return launch_star7_tb_f32x2(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_star7_tb_prepare(int precision) {
    switch (precision) {
        case SCAFES_PREC_F64: return prepare_star7_tb_f64();
        case SCAFES_PREC_F32: return prepare_star7_tb_f32();
        case SCAFES_PREC_F32X2: return prepare_star7_tb_f32x2();
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_star7_loop_f64(const Star7Loop& q, cudaStream_t stream);
cudaError_t launch_star7_loop_f32(const Star7Loop& q, cudaStream_t stream);
cudaError_t launch_star7_loop_f32x2(const Star7Loop& q, cudaStream_t stream);

// Largest grid whose steps run faster as a one-launch loop than as tile
// sweeps (both measured on cubes, us per step, loop / sweeps):
//   rule-table border: at every size; the sweeps evaluate the rules in one or
//     two lanes of every warp at a face (f64 64^3 7.5 / 26, 448^3 1210 / 1908;
//     f32 448^3 584 / 1462; pairs 448^3 781 / 1941);
//   FP64, bound by the FP64 pipe in both forms: 96^3 12 / 18, 201 x 181 x 163
//     61 / 78, 256^3 171 / 176, 320^3 320 / 315; with node coefficients 96^3
//     12 / 31, 256^3 227 / 234, 320^3 424 / 411;
//   FP32 and pairs: while the iterates and the source (and the coefficients)
//     stay in the 126 MB L2, since the loop reads neighbours through L1 only:
//     f32 201 x 181 x 163 20 / 23, 224^3 (90 MB) 35 / 34.5, with a source
//     (135 MB) 52 / 39; pairs 201 x 181 x 163 (106 MB) 32 / 35, 224^3 (180
//     MB) 75 / 55.  Node coefficients and rules: f32 224^3 69 / 85, 256^3
//     106 / 96.
long long star7_loop_max_nodes(const Star7Launch& a) {
    const long long all = (1LL << 31) - 1;  // node numbers are 32-bit
    if (a.border == SCAFES_BORDER_TABLE) return all;
    if (a.precision == SCAFES_PREC_F64) return 256LL * 256 * 256;
    if (a.vc) return 224LL * 224 * 224;
    const int fields = 2 + (a.fa ? 1 : 0) + (a.fb ? 1 : 0);
    return 100000000LL / (fields * (long long)element_size(a.precision));
}

cudaError_t launch_star7_loop(const Star7Loop& q, cudaStream_t stream) {
    switch (q.step.precision) {
        case SCAFES_PREC_F64: return launch_star7_loop_f64(q, stream);
        case SCAFES_PREC_F32: return launch_star7_loop_f32(q, stream);
        case SCAFES_PREC_F32X2: return launch_star7_loop_f32x2(q, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_star7(const Star7Launch& a, cudaStream_t stream) {
    switch (a.precision) {
        case SCAFES_PREC_F64: return launch_star7_f64(a, stream);
        case SCAFES_PREC_F32: return launch_star7_f32(a, stream);
        case SCAFES_PREC_F32X2: return launch_star7_f32x2(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace scafes
