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
    c.m0 = make_int_factor(c0);
    c.mx = make_int_factor(cp[0]);
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

// Measured in us per step (cubes unless given):
//   FP64: the march (star7_march.cuh) at every size;
//   rule tables: the march, whose border rules run in full warps (256^3 with a
//     rule table: f64 226 against 500 with the best tile, f32 85 / 369, pairs
//     144 / 586);
//   pairs with a source affine in time: the march, in whose registers its
//     second field costs no staging (64^3 4.5 against 5.2 with the best tile,
//     130^3 14.5 / 22.3, 201 x 181 x 163 44 / 52, 300 x 280 x 260 146 / 157);
//   pairs with a static source: the {16,2} tile (130^3 17.9, {32,4} 20.0; 201
//     x 181 x 163 37.9 / 39.2; 250 x 240 x 230 68.1 / 73.1) up to 256 x 256
//     columns, then {32,4} (300 x 280 x 260: 105.4 against 107.4; {16,4} 105.3,
//     with a mirror border 109.5 against 106.7);
//   pairs without a source: the {16,4} tile (256^3: 64.7, {32,4} 81.2);
//   FP32: the {16,4} tile (400^3 89 - 94, {32,4} 94 - 95, {8,1} 154; with
//     node coefficients 256^3 88, {32,4} 95, the march 96; 448^3 345, 354, 439),
//     with a source affine in time {16,2} below 2 M nodes (200 x 200 x 20 5.7 /
//     7.9, 120^3 9.2 / 9.4, 130^3 11.2 / 10.4);
//   FP32 and pairs below 700 000 nodes: the {8,1} tile, which has the most
//     CTAs (130 x 130 x 5 3.4, {16,4} 4.7; 80^3 4.4 / 5.2; 97^3 6.4 / 5.4; 100 x
//     100 x 300 15.0 / 10.4; several steps of these grids run as a one-launch
//     loop);
//   several border layers (Dirichlet): one tile is built for them.  FP32 takes
//     it from 1.2 M nodes on (march / tile: 112^3 7.9 / 7.5, 130^3 10.2 / 9.5,
//     160^3 13.5 / 11.6, 250 x 240 x 230 38.5 / 31.2), pairs from 8 M nodes
//     on (201 x 181 x 163 28.9 / 33.1, with a source 36.9 / 39.0; 224^3 50.7 /
//     49.1 and 62.1 / 57.8, 300 x 280 x 260 95.5 / 93.0 and 116 / 110); with a
//     source affine in time the march stays (FP32 201 x 181 x 163 25.7 / 28.3,
//     300 x 280 x 260 80.8 / 85.0).
int star7_default_tile(const Star7Launch& a) {
    const long long cols = (long long)a.L.nx * a.L.ny, nodes = cols * a.L.nz;
    const bool pairs = a.precision == SCAFES_PREC_F32X2;
    const bool march = nodes < (1LL << 31);  // the march numbers nodes in 32 bits
    if (march && (a.precision == SCAFES_PREC_F64 || a.border == SCAFES_BORDER_TABLE || (pairs && a.fb)))
        return STAR7_MARCH;
    if (a.L.nl != 1)
        return march && (a.fb || nodes < (pairs ? 8000000 : 1200000)) ? STAR7_MARCH : STAR7_MULTI_LAYER_TILE;
    if (a.precision == SCAFES_PREC_F64 || nodes < 700000) return 0;
    if (pairs && a.fa) return cols < 256LL * 256LL ? 1 : 2;
    return !pairs && a.fb && nodes < 2000000 ? 1 : 3;
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

// Largest grid whose steps run faster as a one-launch loop than as sweeps, in
// nodes (both measured, us per step, loop / default sweep; the loop reads its
// neighbours through L1 only and falls behind where the sweep's pipes or HBM
// are busy, while the grid barrier is the smaller share):
//   FP64: 96^3 10.3 / 11.1, 112^3 16.0 / 15.3, 128^3 21.5 / 20.6, 136^3 24.7 /
//     24.0, 144^3 29.2 / 27.0, 201 x 181 x 163 54 / 53, with a source 71 / 63, but
//     fields that change sign, whose sums fall back to FP64 in both, 128^3 27.8 /
//     31.2, 144^3 37.6 / 42.0; node coefficients 128^3 23.7 /
//     26.8, 160 x 150 x 140 43.7 / 42.7; node rules and rule tables 201 x 181 x
//     163 63 / 69 and 70 / 74 (256^3 270 / 226);
//   FP32: 112^3 6.6 / 6.5, 128^3 8.7 / 6.8, 160^3 14.7 / 9.8, 250 x 240 x 230
//     53.8 / 26.2; node coefficients 104^3 5.7 / 6.2, 112^3 6.6 / 6.5; several
//     border layers 128^3 8.4 / 8.0, 136^3 9.9 / 10.0, 144^3 11.3 / 10.4; with a
//     source affine in time 145^3 11.4 / 11.7, 160 x 150 x 140 12.5 / 11.2;
//   pairs: 145^3 16.0 / 17.9, 160^3 20.7 / 19.1; with a source 160^3 22.9 / 24.2,
//     180^3 no faster; with one affine in time 97^3 7.1 / 7.9, 112^3 10.5 / 10.4,
//     130^3 15.5 / 13.8;
//   rule tables in FP32 and pairs: 80^3 5.7 / 6.0 and 8.6 / 10.0, 96^3 7.5 / 6.4
//     and 12.2 / 10.6;
//   node rules in FP32 (160^3 16.7 / 30.9, 201 x 181 x 163 36 / 42): while the
//     fields stay in the 126 MB L2.
long long star7_loop_max_nodes(const Star7Launch& a) {
    const bool table = a.border == SCAFES_BORDER_TABLE, rules = a.border == SCAFES_BORDER_NODES;
    switch (a.precision) {
        case SCAFES_PREC_F64: return table || rules ? 8000000 : a.vc ? 3000000 : 2600000;
        case SCAFES_PREC_F32X2: return table ? 600000 : a.fb ? 1500000 : a.fa ? 4200000 : 3200000;
        default:
            if (table) return 600000;
            if (rules) return 120000000 / ((a.fa ? 5 : 4) * 4);
            return a.fb ? 3000000 : a.L.nl != 1 ? 2600000 : 1500000;
    }
}

cudaError_t launch_star7_loop(const Star7Loop& q, cudaStream_t stream) {
    switch (q.step.precision) {
        case SCAFES_PREC_F64: return launch_star7_loop_f64(q, stream);
        case SCAFES_PREC_F32: return launch_star7_loop_f32(q, stream);
        case SCAFES_PREC_F32X2: return launch_star7_loop_f32x2(q, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_star7_march_f64(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_march_f32(const Star7Launch& a, cudaStream_t stream);
cudaError_t launch_star7_march_f32x2(const Star7Launch& a, cudaStream_t stream);

cudaError_t launch_star7(const Star7Launch& a, cudaStream_t stream) {
    if (a.tile == STAR7_MARCH) {
        switch (a.precision) {
            case SCAFES_PREC_F64: return launch_star7_march_f64(a, stream);
            case SCAFES_PREC_F32: return launch_star7_march_f32(a, stream);
            case SCAFES_PREC_F32X2: return launch_star7_march_f32x2(a, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (a.precision) {
        case SCAFES_PREC_F64: return launch_star7_f64(a, stream);
        case SCAFES_PREC_F32: return launch_star7_f32(a, stream);
        case SCAFES_PREC_F32X2: return launch_star7_f32x2(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace scafes
