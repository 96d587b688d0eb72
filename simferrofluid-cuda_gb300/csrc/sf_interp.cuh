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

// TriLerp::Interpolate of face grid b (size res + e_b, origin = corner + h/2 on the other axes) at p:
// Grid::CalcLower<1> / CalcLowerFrac and clamped At().
__device__ __forceinline__ double trilerp_face(const Dims &d, const double *__restrict__ v, int b, const double o[3],
                                               double h, double invh, const double p[3]) {
    const int s[3] = {d.nx + (b == 0), d.ny + (b == 1), d.nz + (b == 2)};
    int lo[3];
    double w[2][3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double co = a == b ? o[a] : o[a] + h / 2;  // face grid origin (core/StaggeredGrid.h:16-20)
        lo[a] = (int)floor((p[a] - co) * invh - 0.0);
        const double fr = (p[a] - co - (double)lo[a] * h) * invh;
        w[0][a] = 1. - fr;
        w[1][a] = fr;
    }
    double val = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int dx = q & 1, dy = (q >> 1) & 1, dz = (q >> 2) & 1;
        int ci[3] = {lo[0] + dx, lo[1] + dy, lo[2] + dz};
#pragma unroll
        for (int a = 0; a < 3; a++) ci[a] = ci[a] < 0 ? 0 : (ci[a] > s[a] - 1 ? s[a] - 1 : ci[a]);
        const double wt = w[dx][0] * w[dy][1] * w[dz][2];
        val += v[(long long)ci[2] + (long long)s[2] * ((long long)ci[1] + (long long)s[1] * ci[0])] * wt;
    }
    return val;
}

// The cells and weights of a point on the staggered grids: per axis on the grid of the faces normal to it ([0], origin
// at the corner) and on the grids of the other faces and of the cells ([1], half a cell further) -- Grid::CalcLower<1> /
// CalcLowerFrac.  Six sets serve the three face grids.
struct GridPoint {
    int lo[2][3];
    double w[2][2][3];  // [grid][lower, upper][axis]
};
__device__ __forceinline__ GridPoint grid_point(const double o[3], double h, double invh, const double p[3]) {
    GridPoint g;
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double co = s == 0 ? o[a] : o[a] + h / 2;  // core/StaggeredGrid.h:16-20
            const double t = p[a] - co;
            double fl;
            g.lo[s][a] = f64_floor(t * invh, fl);
            const double fr = (t - fl * h) * invh;
            g.w[s][0][a] = 1. - fr;
            g.w[s][1][a] = fr;
        }
    return g;
}

// TriLerp::Interpolate of face grid b at a point: the eight clamped faces and their weights, shared by every field on
// that grid.
struct Trilinear {
    int at[8];
    double w[8];
    __device__ __forceinline__ double of(const double *__restrict__ v) const {
        double f[8];
        uint32_t any = 0;  // magnitude bits of the eight values
#pragma unroll
        for (int q = 0; q < 8; q++) {
            f[q] = v[at[q]];
            uint32_t h, l;
            f64_words(f[q], h, l);
            any |= (h << 1) | l;
        }
        // eight zeros (the air beyond the extrapolated layers, a normal's other components) sum to +0 as long as the
        // weights are finite, which all are when the first, (1 - x)(1 - y)(1 - z), is
        uint32_t wh, wl;
        f64_words(w[0], wh, wl);
        if (any == 0 && (wh & kF64Exp) != kF64Exp) return 0.;
        // 0 + v w rounds as v w does, and takes -0 to +0 as the sum from zero does
        double val = __fma_rn(f[0], w[0], 0.);
#pragma unroll
        for (int q = 1; q < 8; q++) val += f[q] * w[q];
        return val;
    }
};
__device__ __forceinline__ Trilinear trilinear(const Dims &d, int b, const GridPoint &g) {
    const int s[3] = {d.nx + (b == 0), d.ny + (b == 1), d.nz + (b == 2)};
    int c[2][3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int lo = g.lo[a == b ? 0 : 1][a];
        c[0][a] = min(max(lo, 0), s[a] - 1);
        c[1][a] = min(max(lo + 1, 0), s[a] - 1);
    }
    Trilinear t;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int dx = q & 1, dy = (q >> 1) & 1, dz = (q >> 2) & 1;
        t.at[q] = c[dz][2] + s[2] * (c[dy][1] + s[1] * c[dx][0]);  // a face grid has fewer than 2^31 faces
        t.w[q] = g.w[b == 0 ? 0 : 1][dx][0] * g.w[b == 1 ? 0 : 1][dy][1] * g.w[b == 2 ? 0 : 1][dz][2];
    }
    return t;
}

// TriCuInterp::Interpolate of the cell grid at p (core/TriCuInterp.h:12-37): CalcLower<3> = floor((p - o)/h - 1),
// cubic Lagrange weights per axis, 64 points in (k, j, i) order, clamped At().
__device__ __forceinline__ double tricubic_cell(const Dims &d, const double *__restrict__ f, const double o[3],
                                                double h, double invh, const double p[3]) {
    const int sz[3] = {d.nx, d.ny, d.nz};
    int lo[3];
    double w[4][3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double co = o[a] + h / 2;  // cell grid origin
        lo[a] = (int)floor((p[a] - co) * invh - 1.0);
        const double fr = (p[a] - co - (double)lo[a] * h) * invh;
        w[0][a] = (fr - 1) * (fr - 2) * (fr - 3) / -6;
        w[1][a] = fr * (fr - 2) * (fr - 3) / 2;
        w[2][a] = fr * (fr - 1) * (fr - 3) / -2;
        w[3][a] = fr * (fr - 1) * (fr - 2) / 6;
    }
    double val = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int ci[3] = {lo[0] + i, lo[1] + j, lo[2] + k};
#pragma unroll
                for (int a = 0; a < 3; a++) ci[a] = ci[a] < 0 ? 0 : (ci[a] > sz[a] - 1 ? sz[a] - 1 : ci[a]);
                val += f[cid(d, ci[0], ci[1], ci[2])] * (w[i][0] * w[j][1] * w[k][2]);
            }
    return val;
}

}  // namespace sf
