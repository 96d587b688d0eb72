// sf_interp.cuh -- the reference's grid interpolations on the device (core/TriLerp.h, core/TriCuInterp.h,
// core/Grid.h:33-35, core/GridData.h:31), for translation units compiled with -fmad=false: each expression is
// evaluated in the reference's order, so the results are bit-identical to its C++ on the same inputs.
#pragma once
#include <cmath>

#include "sf_f64_int.cuh"
#include "sf_internal.cuh"

namespace sf {

struct Origin {
    double o[3];  // staggered-grid corner (StaggeredGrid::GetOrigin)
};

// Where the FP64 pipe is the bound, the weights' products and the products with the field go to the integer pipe
// (sf_f64_int.cuh, about 13 clocks a warp and SM against 19, side by side) and the FP64 pipe keeps the sums.

// The lower cell and the weights of coordinate p on one axis of a grid with origin co -- Grid::CalcLower<1> /
// CalcLowerFrac.
struct AxisPoint {
    int lo;
    double w[2];  // lower, upper
};
__device__ __forceinline__ AxisPoint axis_point(double p, double co, double h, double invh) {
    AxisPoint g;
    const double t = p - co;
    double fl;
    g.lo = f64_floor(t * invh, fl);
    const double fr = (t - fl * h) * invh;
    g.w[0] = 1. - fr;
    g.w[1] = fr;
    return g;
}

// A point on the staggered grids: per axis on the grid of the faces normal to it ([0], origin at the corner) and on the
// grids of the other faces and of the cells ([1], half a cell further).  Six sets serve the three face grids.
struct GridPoint {
    AxisPoint on[2][3];
    // every fraction is zero or in [2^-200, 2), so 1 - fraction is zero or at least 2^-53 in size: the integer products
    // of three weights are exact to their range
    bool plain;
    __device__ __forceinline__ void check() {
        plain = false;
#pragma unroll
        for (int s = 0; s < 2; s++)
#pragma unroll
            for (int a = 0; a < 3; a++) plain = plain || !f64_in_range(on[s][a].w[1], -200, 1);
    }
};
__device__ __forceinline__ GridPoint grid_point(const double o[3], double h, double invh, const double p[3]) {
    GridPoint g;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        g.on[0][a] = axis_point(p[a], o[a], h, invh);  // core/StaggeredGrid.h:16-20
        g.on[1][a] = axis_point(p[a], o[a] + h / 2, h, invh);
    }
    g.check();
    return g;
}

// TriLerp::Interpolate of a face grid of sx * sy * sz faces (fewer than 2^31) at a point: the eight clamped faces in the
// reference's order, x fastest.  In plain FP64, for weights or values outside the integer form's range; its own function,
// because beside the other form its instructions would be issued with their lanes off.
__device__ __noinline__ double trilinear_plain(const double *v, int sx, int sy, int sz, AxisPoint x, AxisPoint y,
                                               AxisPoint z) {
    const int cx[2] = {min(max(x.lo, 0), sx - 1), min(max(x.lo + 1, 0), sx - 1)};
    const int cy[2] = {min(max(y.lo, 0), sy - 1), min(max(y.lo + 1, 0), sy - 1)};
    const int cz[2] = {min(max(z.lo, 0), sz - 1), min(max(z.lo + 1, 0), sz - 1)};
    double f[8];
#pragma unroll
    for (int q = 0; q < 8; q++) f[q] = v[cz[q >> 2] + sz * (cy[(q >> 1) & 1] + sy * cx[q & 1])];
    double val = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) val += f[q] * (x.w[q & 1] * y.w[(q >> 1) & 1] * z.w[q >> 2]);
    return val;
}

// The same; `plain`: the weights are outside the integer form's range (GridPoint::plain).  A call rather than inlined: a
// kernel that takes many samples then stays in the instruction cache (with every sample inlined, warps of the advection
// kernels waited for instructions as often as they issued one).
__device__ __noinline__ double trilinear(const double *v, int sx, int sy, int sz, AxisPoint x, AxisPoint y, AxisPoint z,
                                         bool plain) {
    const int cx[2] = {min(max(x.lo, 0), sx - 1), min(max(x.lo + 1, 0), sx - 1)};
    const int cy[2] = {min(max(y.lo, 0), sy - 1), min(max(y.lo + 1, 0), sy - 1)};
    const int cz[2] = {min(max(z.lo, 0), sz - 1), min(max(z.lo + 1, 0), sz - 1)};
    double f[8];
    uint32_t any = 0, most = 0;  // magnitude bits of the values; the largest exponent above 2^-300
#pragma unroll
    for (int q = 0; q < 8; q++) {
        f[q] = v[cz[q >> 2] + sz * (cy[(q >> 1) & 1] + sy * cx[q & 1])];
        uint32_t h, l;
        f64_words(f[q], h, l);
        any |= (h << 1) | l;
        most = max(most, f64_above(f[q], -300));
    }
    // eight zeros (the air beyond the extrapolated layers, a normal's other components) times finite weights sum to +0
    if (any == 0 && !plain) return 0.;
    if (plain || most >= (600u << 20)) return trilinear_plain(v, sx, sy, sz, x, y, z);
    double val = 0.;
#pragma unroll
    for (int dz = 0; dz < 2; dz++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double wt = f64_mul(f64_mul(x.w[q & 1], y.w[q >> 1]), z.w[dz]);
            const double term = f64_mul<false>(f[4 * dz + q], wt);
            val = 4 * dz + q == 0 ? term : val + term;
        }
    return f64_is_zero(val) ? 0. : val;  // the reference sums from +0, which leaves no -0
}

// Face grid b's field v at a point.
__device__ __forceinline__ double trilinear_face(const Dims &d, int b, const GridPoint &g, const double *v) {
    return trilinear(v, d.nx + (b == 0), d.ny + (b == 1), d.nz + (b == 2), g.on[b == 0 ? 0 : 1][0],
                     g.on[b == 1 ? 0 : 1][1], g.on[b == 2 ? 0 : 1][2], g.plain);
}

// CalcLower<3> and the cubic Lagrange weights of one axis (core/TriCuInterp.h:12-37): lower = floor((p - o)/h - 1).
struct CubicPoint {
    int lo;
    double w[4];
};
__device__ __forceinline__ CubicPoint cubic_point(double p, double co, double h, double invh) {
    CubicPoint g;
    const double t = p - co;
    double fl;
    g.lo = f64_floor(t * invh - 1.0, fl);
    const double fr = (t - fl * h) * invh;
    const double a1 = fr - 1, a2 = fr - 2, a3 = fr - 3;
    if (f64_in_range(fr, -200, 3)) {  // and so the differences are zero or at least 2^-53 in size
        const double f1 = f64_mul(fr, a1);
        g.w[0] = f64_half<true>(f64_third(f64_mul(f64_mul(a1, a2), a3)));  // x / 6 is x / 3 halved, exactly
        g.w[1] = f64_half(f64_mul(f64_mul(fr, a2), a3));
        g.w[2] = f64_half<true>(f64_mul(f1, a3));
        g.w[3] = f64_half(f64_third(f64_mul(f1, a2)));
    } else {
        g.w[0] = a1 * a2 * a3 / -6;
        g.w[1] = fr * a2 * a3 / 2;
        g.w[2] = fr * a1 * a3 / -2;
        g.w[3] = fr * a1 * a2 / 6;
    }
    return g;
}

// TriCuInterp::Interpolate of the cell grid: 64 points in (k, j, i) order, clamped At().  In plain FP64, for weights outside
// the integer form's range.
__device__ __noinline__ double tricubic_plain(int nx, int ny, int nz, const double *f, CubicPoint x, CubicPoint y,
                                              CubicPoint z) {
    int cx[4], cy[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        cx[q] = min(max(x.lo + q, 0), nx - 1) * (ny * nz);
        cy[q] = min(max(y.lo + q, 0), ny - 1) * nz;
    }
    double val = 0;
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        const double *plane = f + min(max(z.lo + k, 0), nz - 1);
        const double wz = k == 0 ? z.w[0] : (k == 1 ? z.w[1] : (k == 2 ? z.w[2] : z.w[3]));
        double v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = plane[cx[q & 3] + cy[q >> 2]];
#pragma unroll
        for (int q = 0; q < 16; q++) val += v[q] * (x.w[q & 3] * y.w[q >> 2] * wz);
    }
    return val;
}

// A sum's next four terms, a row of the stencil: values of any size times products xy[i] wz, in plain FP64.  Its own
// function for the reason of trilinear_plain.
__device__ __noinline__ double tricubic_row(double val, double v0, double v1, double v2, double v3, const double *xy,
                                            double wz) {
    val += v0 * (xy[0] * wz);
    val += v1 * (xy[256] * wz);
    val += v2 * (xy[512] * wz);
    val += v3 * (xy[768] * wz);
    return val;
}

// The same.  An axis on which the point sits on a cell (weights exactly 0, 1, 0, 0: no motion along it) keeps its second
// point alone: the others would add a signed zero to a sum that starts at +0, as long as their values are finite.
// Otherwise the weights are normal and so is every product, as long as the values are in [2^-100, 2^300); a row that holds
// another value (a zero, as on a layer of cells that the surface passes through exactly) is summed in FP64.
// The sixteen products of the x and y weights wait in shared memory (`xy`, this thread's column of 256), so that the
// loops over k and j stay loops: unrolled over j they took 2600 us at 192^3, the warps waiting for instructions.
__device__ __forceinline__ double tricubic(const Dims &d, const double *__restrict__ f, const CubicPoint g[3],
                                           double (*xy)[256]) {
    const int tid = threadIdx.y * 32 + threadIdx.x;
    int cx[4];
    bool one[3];
    uint32_t most = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        one[a] = f64_is_zero(g[a].w[0]) && f64_is_one(g[a].w[1]) && f64_is_zero(g[a].w[2]) && f64_is_zero(g[a].w[3]);
#pragma unroll
        for (int q = 0; q < 4; q++) most = one[a] ? most : max(most, f64_above(g[a].w[q], -300));
    }
    bool hard = most >= (330u << 20);
    double val = 0;
    if (!hard) {
#pragma unroll
        for (int q = 0; q < 4; q++) cx[q] = min(max(g[0].lo + q, 0), d.nx - 1) * (d.ny * d.nz);  // fewer than 2^31 cells
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) xy[4 * j + i][tid] = f64_mul(g[0].w[i], g[1].w[j]);
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            const double wk = k == 0 ? g[2].w[0] : (k == 1 ? g[2].w[1] : (k == 2 ? g[2].w[2] : g[2].w[3]));
            const int ck = min(max(g[2].lo + k, 0), d.nz - 1);
#pragma unroll 1
            for (int j = 0; j < 4; j++) {
                const int row = ck + min(max(g[1].lo + j, 0), d.ny - 1) * d.nz;
                double v[4];
                uint32_t far = 0, size = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    v[i] = f[row + cx[i]];
                    far = max(far, f64_above(v[i], -100));
                    size = max(size, f64_above(v[i], -1023));  // the exponent field itself
                }
                if (size < kF64Exp && ((one[2] && k != 1) || (one[1] && j != 1))) continue;  // finite times zero
                if (far >= (400u << 20)) {
                    val = tricubic_row(val, v[0], v[1], v[2], v[3], &xy[4 * j][tid], wk);
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (one[0] && i != 1) continue;
                    const double w2 = xy[4 * j + i][tid];
                    const double wt = one[2] ? w2 : f64_mul<false, false>(w2, wk);
                    // three products in four on the integer pipe balance the two
                    val += i < 3 ? f64_mul<false, false>(v[i], wt) : v[i] * wt;
                }
            }
        }
    }
    return hard ? tricubic_plain(d.nx, d.ny, d.nz, f, g[0], g[1], g[2]) : val;
}

}  // namespace sf
