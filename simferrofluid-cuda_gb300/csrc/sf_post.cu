// sf_post.cu -- the velocity pipeline after the pressure projection (core/Simulation.cpp:236-241): extrapolation
// of the projected velocity into the air (Extrapolation::Solve) and the collider's boundary condition
// (Collider::Enforce), on device-resident face arrays.
//
// Compiled with -fmad=false: each expression rounds as the reference's C++ does, so the results are bit-identical
// to the CPU restatement on the same inputs.
#include <cmath>

#include "sf_f64_int.cuh"
#include "sf_interp.cuh"
#include "sf_ops.h"

namespace sf {

namespace {

inline dim3 blk2() { return dim3(32, 8, 1); }
inline dim3 face_grid(const Dims &d, int a) {
    return dim3((d.nz + (a == 2) + 31) / 32, (d.ny + (a == 1) + 7) / 8, d.nx + (a == 0));
}

struct FDims {
    int fx, fy, fz;
};
__device__ __forceinline__ FDims fdims(const Dims &d, int a) { return FDims{d.nx + (a == 0), d.ny + (a == 1), d.nz + (a == 2)}; }
__device__ __forceinline__ long long fidx(const FDims &f, int i, int j, int k) {
    return (long long)k + (long long)f.fz * ((long long)j + (long long)f.fy * i);
}

// Extrapolation validity (core/Simulation.cpp:237-240): fraction < 1 and an adjacent cell (face - e_a, face)
// is liquid; a cell outside the grid is not liquid.
__global__ void __launch_bounds__(256) k_extrap_init(Dims d, int a, const double *__restrict__ phi,
                                                     const double *__restrict__ frac, uint8_t *__restrict__ valid) {
    const FDims f = fdims(d, a);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const long long fi = fidx(f, i, j, k);
    uint8_t v = 0;
    if (frac[fi] < 1) {
        int c0[3] = {i, j, k};
        c0[a] -= 1;
        const bool in0 = c0[0] >= 0 && c0[1] >= 0 && c0[2] >= 0;
        const bool in1 = i < d.nx && j < d.ny && k < d.nz;
        const bool l0 = in0 && phi[cid(d, c0[0], c0[1], c0[2])] <= 0;
        const bool l1 = in1 && phi[cid(d, i, j, k)] <= 0;
        v = (l0 || l1) ? 1 : 0;
    }
    valid[fi] = v;
}

// One sweep of Extrapolation::Solve (core/Extrapolation.cpp:7-28) on face grid a: invalid faces take the mean of
// their valid 6-neighbours (order -x,+x,-y,+y,-z,+z) and become valid, or clear_val without any.  Valid faces are
// never written in a sweep, so the in-place update reads only values of the previous sweep.
__global__ void __launch_bounds__(256) k_extrap_step(Dims d, int a, double *__restrict__ u,
                                                     const uint8_t *__restrict__ valid, uint8_t *__restrict__ valid1,
                                                     double clear_val) {
    const FDims f = fdims(d, a);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const long long fi = fidx(f, i, j, k);
    if (valid[fi]) {
        valid1[fi] = 1;
        return;
    }
    int cnt = 0;
    double sum = 0;
    const int n3[3] = {f.fx, f.fy, f.fz};
#pragma unroll
    for (int o = 0; o < 6; o++) {
        const int ax = o >> 1, s = (o & 1) ? 1 : -1;
        int q[3] = {i, j, k};
        q[ax] += s;
        if (q[ax] < 0 || q[ax] >= n3[ax]) continue;
        const long long nb = fidx(f, q[0], q[1], q[2]);
        if (valid[nb]) {
            sum += u[nb];
            cnt++;
        }
    }
    if (cnt > 0) {
        u[fi] = sum / cnt;
        valid1[fi] = 1;
    } else {
        u[fi] = clear_val;
        valid1[fi] = 0;
    }
}

// Collider::Enforce (core/Collider.cpp:75-86) on the faces of axis a with fraction == 1: the interpolated old
// velocity minus its normal component relative to the solid velocity (us.p[0] == nullptr: zero).
__global__ void __launch_bounds__(256) k_enforce(Dims d, int a, Origin og, double h, double invh, Faces old,
                                                 Faces us, Faces normal, const double *__restrict__ frac,
                                                 double *__restrict__ u) {
    const FDims f = fdims(d, a);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const long long fi = fidx(f, i, j, k);
    if (frac[fi] != 1.) return;
    const int c3[3] = {i, j, k};
    double p[3];
#pragma unroll
    for (int b = 0; b < 3; b++) p[b] = (b == a ? og.o[b] : og.o[b] + h / 2) + (double)c3[b] * h;  // PositionOf
    double vel[3], vel0[3], n[3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        vel[b] = trilerp_face(d, old.p[b], b, og.o, h, invh, p);
        vel0[b] = us.p[0] ? trilerp_face(d, us.p[b], b, og.o, h, invh, p) : 0.0;
        n[b] = trilerp_face(d, normal.p[b], b, og.o, h, invh, p);
    }
    const double nn = sqrt((n[0] * n[0] + n[1] * n[1]) + n[2] * n[2]);  // Vector3d::normalized
    if (nn > 0)
#pragma unroll
        for (int b = 0; b < 3; b++) n[b] = n[b] / nn;
    const double dv0 = vel[0] - vel0[0], dv1 = vel[1] - vel0[1], dv2 = vel[2] - vel0[2];
    const double dn = (dv0 * n[0] + dv1 * n[1]) + dv2 * n[2];
    u[fi] = vel[a] - dn * n[a];
}

// MagneticField::CalculateVertexPressures (core/MagneticField.cpp:37-48) for vertex v: H trilinear at its position,
// p = mu0/2 chi (|H|^2 + chi^2/(4chi+4) (H.n)^2), mu0 = 4e-7 pi (core/MagneticField.cpp:7-8).
__global__ void k_vertex_pressures(Dims d, Origin og, double h, double invh, Faces H, double chi,
                                   const double *__restrict__ pos, const double *__restrict__ nrm, long long nv,
                                   double *__restrict__ out) {
    const double pi = 3.141592653589793238462643383279502884;
    const double mu0 = 4e-7 * pi;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nv; v += (long long)gridDim.x * blockDim.x) {
        const double p[3] = {pos[3 * v], pos[3 * v + 1], pos[3 * v + 2]};
        const double n[3] = {nrm[3 * v], nrm[3 * v + 1], nrm[3 * v + 2]};
        double hv[3];
#pragma unroll
        for (int b = 0; b < 3; b++) hv[b] = trilerp_face(d, H.p[b], b, og.o, h, invh, p);
        double coeff = (hv[0] * hv[0] + hv[1] * hv[1]) + hv[2] * hv[2];
        const double hn = (hv[0] * n[0] + hv[1] * n[1]) + hv[2] * n[2];
        coeff += chi * chi / (4 * chi + 4) * hn * hn;
        out[v] = mu0 * 0.5 * chi * coeff;
    }
}

struct EdgeMarks {
    const int32_t *p[3];
};

// The pressure-jump callback of core/Simulation.cpp:216-235 on the faces of axis a: the vertex of edge
// (a, face - e_a) (Contour::VertexIndexOf; edge grid of axis a = cell grid minus e_a, -1 = no vertex) gives
// J = kappa sigma / rho / h dt - p_m / rho / h dt (terms present when their arrays are), 0 without a vertex.
__global__ void __launch_bounds__(256) k_pressure_jump(Dims d, int a, EdgeMarks em, const double *__restrict__ kappa,
                                                       const double *__restrict__ pm, double sigma, double rho,
                                                       double invh, double dt, double *__restrict__ jump) {
    const FDims f = fdims(d, a);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const int ex = d.nx - (a == 0), ey = d.ny - (a == 1), ez = d.nz - (a == 2);
    int e[3] = {i, j, k};
    e[a] -= 1;
    int idx = -1;
    if (e[0] >= 0 && e[1] >= 0 && e[2] >= 0 && e[0] < ex && e[1] < ey && e[2] < ez)
        idx = em.p[a][(long long)e[2] + (long long)ez * ((long long)e[1] + (long long)ey * e[0])];
    double pressure = 0;
    if (kappa && idx >= 0) pressure += kappa[idx] * sigma / rho * invh * dt;
    if (pm && idx >= 0) pressure -= pm[idx] / rho * invh * dt;
    jump[fidx(f, i, j, k)] = pressure;
}

// ------------------------------------------------------------------------------------------------ level set
// Advection::Trace<2> (core/Advection.h:15-18): TVD Runge-Kutta trace of second order from p over dt.
__device__ __forceinline__ void trace_rk2(const Dims &d, const Faces &u, const double o[3], double h, double invh,
                                          const double p[3], double dt, double out[3]) {
    double v0[3], v1[3], q[3];
#pragma unroll
    for (int b = 0; b < 3; b++) v0[b] = trilerp_face(d, u.p[b], b, o, h, invh, p);
#pragma unroll
    for (int b = 0; b < 3; b++) q[b] = p[b] + v0[b] * dt;
#pragma unroll
    for (int b = 0; b < 3; b++) v1[b] = trilerp_face(d, u.p[b], b, o, h, invh, q);
#pragma unroll
    for (int b = 0; b < 3; b++) out[b] = p[b] + (v0[b] + v1[b]) * dt / 2;
}

// Advection::Solve<2>(levelSet, velocity, dt) (core/Advection.h:40-49): phi at each cell centre's RK2 departure
// point (trace over -dt), by tricubic interpolation of the old phi.
__global__ void __launch_bounds__(256) k_advect_levelset(Dims d, Origin og, double h, double invh, Faces u,
                                                         double dt, const double *__restrict__ phi,
                                                         double *__restrict__ out) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const double p[3] = {og.o[0] + h / 2 + (double)i * h, og.o[1] + h / 2 + (double)j * h,
                         og.o[2] + h / 2 + (double)k * h};
    double q[3];
    trace_rk2(d, u, og.o, h, invh, p, -dt, q);
    out[cid(d, i, j, k)] = tricubic_cell(d, phi, og.o, h, invh, q);
}

// Advection::Solve<2>(velocity, velocity, dt) (core/Advection.h:51-59) for the faces of axis a: trilinear
// interpolation of the old face grid a at each face's RK2 departure point.
__global__ void __launch_bounds__(256) k_advect_velocity(Dims d, int a, Origin og, double h, double invh, Faces u,
                                                         const double *__restrict__ ua, double dt,
                                                         double *__restrict__ out) {
    const FDims f = fdims(d, a);
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= f.fz || j >= f.fy) return;
    const int c3[3] = {i, j, k};
    double p[3], q[3];
#pragma unroll
    for (int b = 0; b < 3; b++) p[b] = (b == a ? og.o[b] : og.o[b] + h / 2) + (double)c3[b] * h;
    trace_rk2(d, u, og.o, h, invh, p, -dt, q);
    out[fidx(f, i, j, k)] = trilerp_face(d, ua, a, og.o, h, invh, q);
}

// v < 0 on the bits (false for NaN and -0)
__device__ __forceinline__ bool below0(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    const uint64_t b = ((uint64_t)h << 32) | l;
    return b > 0x8000000000000000ULL && b <= 0xfff0000000000000ULL;
}

__device__ __forceinline__ double dmax0(double a, double b) { return (a < b) ? b : a; }  // std::max(a, b)

// GetDrv (core/Reinitialization.cpp:4-27): the WENO5 one-sided derivative from five differences, the upwind side's
// outermost first, in plain FP64: the form for differences outside the fast form's range.
__device__ __noinline__ double weno_plain(double d0, double d1, double d2, double d3, double d4, double invdx) {
    const double dev[5] = {d0, d1, d2, d3, d4};
    double eps = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) eps = dmax0(eps, dev[j] * dev[j]);
    eps = eps * 1e-6 + 1e-99;
    const double phix1 = dev[0] / 3 - dev[1] * 7 / 6 + dev[2] * 11 / 6;
    const double phix2 = -dev[1] / 6 + dev[2] * 5 / 6 + dev[3] / 3;
    const double phix3 = dev[2] / 3 + dev[3] * 5 / 6 - dev[4] / 6;
    double t = dev[0] - 2 * dev[1] + dev[2];
    double s1 = t * t * 13 / 12;
    t = dev[0] - 4 * dev[1] + 3 * dev[2];
    s1 = s1 + t * t / 4;
    t = dev[1] - 2 * dev[2] + dev[3];
    double s2 = t * t * 13 / 12;
    t = dev[1] - dev[3];
    s2 = s2 + t * t / 4;
    t = dev[2] - 2 * dev[3] + dev[4];
    double s3 = t * t * 13 / 12;
    t = 3 * dev[2] - 4 * dev[3] + dev[4];
    s3 = s3 + t * t / 4;
    t = s1 + eps;
    const double alpha1 = .1 / (t * t);
    t = s2 + eps;
    const double alpha2 = .6 / (t * t);
    t = s3 + eps;
    const double alpha3 = .3 / (t * t);
    const double sum = alpha1 + alpha2 + alpha3;
    return (alpha1 * phix1 + alpha2 * phix2 + alpha3 * phix3) / sum * invdx;
}

// The same derivative with the same roundings for differences that are zero or in [2^-100, 2^60) and not all zero.
// What changes is how each rounded value is obtained:
//   * x / 3 and quotients on the integer pipe; x / 6, x / 12 and x / 4 are x / 3 or x scaled by a power of two, which
//     is exact, so the scaling moves into the following sum as a fused multiply-add (one rounding either way);
//   * 2 d and 4 d are exact, so d0 - 2 d1 is one fused multiply-add;
//   * the largest square is the square of the largest magnitude (rounding is monotone), found by integer compares;
//     its millionth is at least 2^-221, so adding 1e-99 leaves it unchanged.
//   * products go to the integer pipe too, so that the FP64 pipe is left with the sums.
// Measured per warp and SM: an FP64 instruction takes 19 clocks, the compiler's division 137, its x / 3 140 and its
// square root 143; on the integer pipe, beside it, a product takes 12-14, a division 27, a third 9, a root 24.
__device__ __forceinline__ double weno_fast(const double dev[5], double invdx) {
    // the magnitudes as integers (an absolute value of doubles would take the FP64 pipe)
    uint64_t big = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) {
        uint32_t h, l;
        f64_words(dev[j], h, l);
        const uint64_t v = ((uint64_t)(h & 0x7fffffffu) << 32) | l;
        big = v > big ? v : big;
    }
    const double top = f64_from_words((uint32_t)(big >> 32), (uint32_t)big);
    const double eps = f64_mul<true>(f64_sqr<true>(top), 1e-6);
    const double third1 = f64_third(dev[1]), third2 = f64_third(dev[2]), third3 = f64_third(dev[3]);
    const double phix1 = __fma_rn(.5, f64_times_third<11>(dev[2]),
                                  __fma_rn(-.5, f64_times_third<7>(dev[1]), f64_third(dev[0])));
    const double phix2 = __fma_rn(.5, f64_times_third<5>(dev[2]) - third1, third3);
    const double phix3 = __fma_rn(-.5, f64_third(dev[4]), __fma_rn(.5, f64_times_third<5>(dev[3]), third2));
    const double three2 = 3 * dev[2];
    // s1, s2, s3: four times the reference's values
    const double s1 = f64_times_third<13>(f64_sqr(__fma_rn(-2., dev[1], dev[0]) + dev[2])) +
                      f64_sqr(__fma_rn(-4., dev[1], dev[0]) + three2);
    const double s2 = f64_times_third<13>(f64_sqr(__fma_rn(-2., dev[2], dev[1]) + dev[3])) +
                      f64_sqr(dev[1] - dev[3]);
    const double s3 = f64_times_third<13>(f64_sqr(__fma_rn(-2., dev[3], dev[2]) + dev[4])) +
                      f64_sqr(__fma_rn(-4., dev[3], three2) + dev[4]);
    const double alpha1 = f64_div(.1, f64_sqr<true>(__fma_rn(.25, s1, eps)));
    const double alpha2 = f64_div(.6, f64_sqr<true>(__fma_rn(.25, s2, eps)));
    const double alpha3 = f64_div(.3, f64_sqr<true>(__fma_rn(.25, s3, eps)));
    const double sum = alpha1 + alpha2 + alpha3;
    return f64_mul(f64_div(f64_mul(alpha1, phix1) + f64_mul(alpha2, phix2) + f64_mul(alpha3, phix3), sum), invdx);
}

// An FP32 value within 2^-23 of v (truncated), v zero or in [2^-100, 2^60).
__device__ __forceinline__ float f32_near(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    const uint32_t m = (h & 0x7fffffffu) - (896u << 20);  // exponent rebased
    return (h << 1) == 0u ? 0.f : __uint_as_float(((m << 3) | (l >> 29)) | (h & 0x80000000u));
}

// Sign of the WENO derivative of differences d0..d4 (FP32, truncated) when FP32 arithmetic can tell: +1 / -1, else 0.
//   * Its three candidate derivatives clearly share a sign (each exceeds 2^-19 of the sum of its terms' magnitudes;
//     truncations and roundings stay below 2^-21 of it): then so does their convex combination.
//   * Otherwise the weights are formed in FP32 from the differences scaled to a largest magnitude in [1, 2).  The
//     scaled differences are off by at most 2^-22, a smoothness measure's terms by 2^-18, and since the measure has
//     1e-6 of the largest square added, the sum is off by at most 0.4% and a weight (its inverse square) by 1%; a
//     candidate is off by 2^-19.  A combination above 5% of its terms' magnitudes and 2^-17 of the weights keeps its
//     sign in FP64.
// The second test takes 5% of the FP64 instructions off a rippled 128^3 field (168 to 160 a warp and stage).
__device__ __forceinline__ int weno_sign(float d0, float d1, float d2, float d3, float d4) {
    const float tol = 1.9073486e-6f;
    const float a = d0 * (1.f / 3.f), b = d1 * (-7.f / 6.f), c = d2 * (11.f / 6.f);
    const float p1 = a + b + c, e1 = (fabsf(a) + fabsf(b) + fabsf(c)) * tol;
    const float f = d1 * (-1.f / 6.f), g = d2 * (5.f / 6.f), h = d3 * (1.f / 3.f);
    const float p2 = f + g + h, e2 = (fabsf(f) + fabsf(g) + fabsf(h)) * tol;
    const float l = d2 * (1.f / 3.f), m = d3 * (5.f / 6.f), n = d4 * (-1.f / 6.f);
    const float p3 = l + m + n, e3 = (fabsf(l) + fabsf(m) + fabsf(n)) * tol;
    if (p1 > e1 && p2 > e2 && p3 > e3) return 1;
    if (p1 < -e1 && p2 < -e2 && p3 < -e3) return -1;
    const float top = fmaxf(fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(d2), fabsf(d3))), fabsf(d4));
    const float sc = __uint_as_float((254u << 23) - (__float_as_uint(top) & 0x7f800000u));  // 2^-exponent
    const float x0 = d0 * sc, x1 = d1 * sc, x2 = d2 * sc, x3 = d3 * sc, x4 = d4 * sc;
    const float eps = 1e-6f * (top * sc) * (top * sc);
    const float t1 = x0 - 2.f * x1 + x2, q1 = x0 - 4.f * x1 + 3.f * x2;
    const float t2 = x1 - 2.f * x2 + x3, q2 = x1 - x3;
    const float t3 = x2 - 2.f * x3 + x4, q3 = 3.f * x2 - 4.f * x3 + x4;
    const float s1 = t1 * t1 * (13.f / 12.f) + q1 * q1 * .25f + eps;
    const float s2 = t2 * t2 * (13.f / 12.f) + q2 * q2 * .25f + eps;
    const float s3 = t3 * t3 * (13.f / 12.f) + q3 * q3 * .25f + eps;
    const float a1 = __fdividef(.1f, s1 * s1), a2 = __fdividef(.6f, s2 * s2), a3 = __fdividef(.3f, s3 * s3);
    const float n1 = a1 * (p1 * sc), n2 = a2 * (p2 * sc), n3 = a3 * (p3 * sc);
    const float num = n1 + n2 + n3;
    const float err = .05f * (fabsf(n1) + fabsf(n2) + fabsf(n3)) + 7.6293945e-6f * (a1 + a2 + a3);
    return num > err ? 1 : (num < -err ? -1 : 0);
}

// Tile of the step kernel: 16 (z) x 4 (y) x 4 (x) cells, one thread each.  The differences along the three axes that
// its stencils read are formed once, into shared memory: 9 x 4 x 16 along x, 4 x 9 x 16 along y, 4 x 4 x 21 along z,
// 5.8 a cell instead of 18.
constexpr int kRx = 4, kRy = 4, kRz = 16;
constexpr int kRdx = (kRx + 5) * kRy * kRz, kRdy = kRx * (kRy + 5) * kRz, kRdz = kRx * kRy * (kRz + 5);

__device__ __forceinline__ int clamp_to(int v, int last) { return v < 0 ? 0 : (v > last ? last : v); }

// Reinitialization::Advance (core/Reinitialization.cpp:48-74): one explicit step of the reinitialisation equation
// with Godunov upwinding of the WENO5 derivatives (clamped stencils at the grid ends), and the TVD-RK3 combination
// that follows it (core/Reinitialization.cpp:41-44): STAGE 0 the step alone, 1 (3 phi + step) / 4, 2 (phi + 2 step) / 3.
//
// A derivative enters only with one sign (Godunov): where its sign is known without evaluating it and is the other
// one, it adds +0 to a sum that is never negative, and is left out.  On a smooth field that is one of the two sides
// of each axis; the few cells that need both (2% an axis next to kinks, but half of the warps hold one) leave the
// second to a queue that the block's threads then share.  `plain` (h outside [2^-60, 2^60]) sends every derivative
// to the plain form.
//
// Bound by the FP64 pipe, then by the integer pipes; DRAM carries 16-24 bytes a cell, 1% of its rate.  A stage at
// 128^3: 4.39 ms with every operation on the FP64 pipe (1043 a cell, half of them inside divisions), 1.11 ms with
// quotients off it, 0.69 ms with products off it too (168 instructions a warp), 0.48 ms with the differences shared, the
// second sides queued and magnitudes taken on the words (108; the pipe 77% busy).  64 registers: four blocks an SM
// instead of three are worth 2.5%.
template <int STAGE>
__global__ void __launch_bounds__(256, 4) k_reinit_advance(Dims d, double h, double invdx, double dt, int plain,
                                                        const double *__restrict__ f, const double *phi, double *out) {
    __shared__ double diff[kRdx + kRdy + kRdz];
    __shared__ double part[6][256];  // squares of the derivatives taken, minus (or only) and plus side of each axis
    __shared__ uint16_t queue[3 * 256];
    __shared__ int queued;
    const int tid = threadIdx.x, lz = tid & 15, ly = (tid >> 4) & 3, lx = tid >> 6;
    const int k0 = blockIdx.x * kRz, j0 = blockIdx.y * kRy, i0 = blockIdx.z * kRx;
    const int lastx = d.nx - 1, lasty = d.ny - 1, lastz = d.nz - 1;
    if (tid == 0) queued = 0;
    for (int e = tid; e < kRdx; e += 256) {  // [m][y][z], m the lower x plane + 3
        const int m = i0 + (e >> 6) - 3;
        const long long r = cid(d, 0, clamp_to(j0 + ((e >> 4) & 3), lasty), clamp_to(k0 + (e & 15), lastz));
        const long long sx = (long long)d.ny * d.nz;
        diff[e] = f[r + clamp_to(m + 1, lastx) * sx] - f[r + clamp_to(m, lastx) * sx];
    }
    for (int e = tid; e < kRdy; e += 256) {  // [x][m][z]
        const int r = e >> 4, x = r / (kRy + 5), m = j0 + r - x * (kRy + 5) - 3;
        const long long c = cid(d, clamp_to(i0 + x, lastx), 0, clamp_to(k0 + (e & 15), lastz));
        diff[kRdx + e] = f[c + (long long)clamp_to(m + 1, lasty) * d.nz] - f[c + (long long)clamp_to(m, lasty) * d.nz];
    }
    for (int e = tid; e < kRdz; e += 256) {  // [x][y][m]
        const int r = e / (kRz + 5), m = k0 + e - r * (kRz + 5) - 3;
        const long long c = cid(d, clamp_to(i0 + (r >> 2), lastx), clamp_to(j0 + (r & 3), lasty), 0);
        diff[kRdx + kRdy + e] = f[c + clamp_to(m + 1, lastz)] - f[c + clamp_to(m, lastz)];
    }
    __syncthreads();
    const int k = k0 + lz, j = j0 + ly, i = i0 + lx;
    const bool cell = i <= lastx && j <= lasty && k <= lastz;
    const long long c = cid(d, i, j, k);
    const double fc = cell ? f[c] : 0.;
    const bool neg = below0(fc);
    if (cell) {
#pragma unroll 1
        for (int a = 0; a < 3; a++) {
            const double *dd = diff + (a == 0 ? tid : (a == 1 ? kRdx + (lx * (kRy + 5) + ly) * kRz + lz
                                                              : kRdx + kRdy + (lx * kRy + ly) * (kRz + 5) + lz));
            const int st = a == 0 ? kRy * kRz : (a == 1 ? kRz : 1);
            double dv[6];
            float w[6];
            bool fast = !plain;
#pragma unroll
            for (int q = 0; q < 6; q++) {
                dv[q] = dd[q * st];
                fast = fast && f64_in_range(dv[q], -100, 60);
                w[q] = f32_near(dv[q]);
            }
            double p0 = 0., p1 = 0.;
            if (fast) {
                const int drops = neg ? 1 : -1;  // the sign with which the minus derivative drops out
                const bool left = weno_sign(w[0], w[1], w[2], w[3], w[4]) != drops &&
                                  !(w[0] == 0.f && w[1] == 0.f && w[2] == 0.f && w[3] == 0.f && w[4] == 0.f);
                const bool right = weno_sign(w[5], w[4], w[3], w[2], w[1]) != -drops &&
                                   !(w[5] == 0.f && w[4] == 0.f && w[3] == 0.f && w[2] == 0.f && w[1] == 0.f);
                if (left || right) {
                    // read again rather than selected: a select of doubles takes the FP64 pipe
                    const double *s0 = left ? dd : dd + 5 * st;
                    const int sst = left ? st : -st;
                    const double dev[5] = {s0[0], s0[sst], s0[2 * sst], s0[3 * sst], s0[4 * sst]};
                    const double v = weno_fast(dev, invdx);
                    // min(v, 0) or std::max(v, 0) by the side and the sign of phi; tested on the bits
                    if (below0(v) == (left == neg)) p0 = f64_sqr(v);
                }
                if (left && right) queue[atomicAdd(&queued, 1)] = (uint16_t)(a * 256 + tid);
            } else {
                double v = weno_plain(dv[0], dv[1], dv[2], dv[3], dv[4], invdx);
                if (below0(v) == neg) p0 = v * v;
                v = weno_plain(dv[5], dv[4], dv[3], dv[2], dv[1], invdx);
                if (below0(v) != neg) p1 = v * v;
            }
            part[2 * a][tid] = p0;
            part[2 * a + 1][tid] = p1;
        }
    }
    __syncthreads();
    for (int e = tid; e < queued; e += 256) {
        const int a = queue[e] >> 8, t = queue[e] & 255;
        const int tz = t & 15, ty = (t >> 4) & 3, tx = t >> 6;
        const double *dd = diff + (a == 0 ? t : (a == 1 ? kRdx + (tx * (kRy + 5) + ty) * kRz + tz
                                                        : kRdx + kRdy + (tx * kRy + ty) * (kRz + 5) + tz));
        const int st = a == 0 ? kRy * kRz : (a == 1 ? kRz : 1);
        const double dev[5] = {dd[5 * st], dd[4 * st], dd[3 * st], dd[2 * st], dd[st]};
        const double v = weno_fast(dev, invdx);
        const double fo = f[cid(d, i0 + tx, j0 + ty, k0 + tz)];
        if (below0(v) != below0(fo)) part[2 * a + 1][t] = f64_sqr(v);
    }
    __syncthreads();
    if (!cell) return;
    double sum = part[0][tid];  // minus side first, as the reference adds them; a zero would leave the sum as it is
#pragma unroll
    for (int q = 1; q < 6; q++)
        if (!f64_is_zero(part[q][tid])) sum += part[q][tid];
    sum = f64_in_range(sum, -600, 600) && !f64_is_zero(sum) ? f64_sqrt(sum) : sqrt(sum);
    const double sp = h * sum;
    const double len2 = fc * fc + sp * sp;
    const double len = f64_in_range(len2, -600, 600) && !f64_is_zero(len2) ? f64_sqrt(len2) : sqrt(len2);
    const double sgn = f64_in_range(fc, -300, 300) && f64_in_range(len, -300, 300) && !f64_is_zero(len)
                           ? f64_div(fc, len)
                           : fc / len;
    const double step = fc + dt * sgn * (1. - sum);
    if (STAGE == 0) {
        out[c] = step;
    } else if (STAGE == 1) {
        out[c] = (phi[c] * 3 + step) / 4;
    } else {
        const double s = phi[c] + step * 2;
        out[c] = f64_in_range(s, -1000, 1000) ? f64_third(s) : s / 3;
    }
}

inline dim3 reinit_grid(const Dims &d) {
    return dim3((d.nz + kRz - 1) / kRz, (d.ny + kRy - 1) / kRy, (d.nx + kRx - 1) / kRx);
}

inline dim3 cell_grid(const Dims &d) { return dim3((d.nz + 31) / 32, (d.ny + 7) / 8, d.nx); }
}  // namespace

void launch_advect_levelset(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &u,
                            double dt, const double *phi, double *out) {
    Origin og{{origin[0], origin[1], origin[2]}};
    k_advect_levelset<<<cell_grid(d), blk2(), 0, st>>>(d, og, h, 1 / h, u, dt, phi, out);
}

void launch_advect_velocity(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &u,
                            double dt, double *const out[3]) {
    Origin og{{origin[0], origin[1], origin[2]}};
    for (int a = 0; a < 3; a++)
        k_advect_velocity<<<face_grid(d, a), blk2(), 0, st>>>(d, a, og, h, 1 / h, u, u.p[a], dt, out[a]);
}

void launch_reinitialize(cudaStream_t st, const Dims &d, double h, double *phi, double *p1, double *p2,
                         int max_steps) {
    const double dt = h * .5, invdx = 1 / h;
    const int plain = !(h >= 0x1p-60 && h <= 0x1p60);
    for (int it = 0; it < max_steps; it++) {
        k_reinit_advance<0><<<reinit_grid(d), 256, 0, st>>>(d, h, invdx, dt, plain, phi, nullptr, p1);
        k_reinit_advance<1><<<reinit_grid(d), 256, 0, st>>>(d, h, invdx, dt, plain, p1, phi, p2);
        k_reinit_advance<2><<<reinit_grid(d), 256, 0, st>>>(d, h, invdx, dt, plain, p2, phi, phi);
    }
}

void launch_vertex_pressures(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &H,
                             double chi, const double *pos, const double *nrm, long long nv, double *out) {
    if (nv <= 0) return;
    Origin og{{origin[0], origin[1], origin[2]}};
    long long blocks = (nv + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_vertex_pressures<<<(unsigned)blocks, 256, 0, st>>>(d, og, h, 1 / h, H, chi, pos, nrm, nv, out);
}

void launch_pressure_jump(cudaStream_t st, const Dims &d, const int32_t *const edge_mark[3], const double *kappa,
                          const double *pm, double sigma, double rho, double h, double dt, double *const jump[3]) {
    EdgeMarks em{{edge_mark[0], edge_mark[1], edge_mark[2]}};
    for (int a = 0; a < 3; a++)
        k_pressure_jump<<<face_grid(d, a), blk2(), 0, st>>>(d, a, em, kappa, pm, sigma, rho, 1 / h, dt, jump[a]);
}

void launch_extrapolate(cudaStream_t st, const Dims &d, const double *phi, const Faces &frac, double *const u[3],
                        uint8_t *const valid[3], uint8_t *const valid1[3], double clear_val, int max_steps) {
    for (int a = 0; a < 3; a++) {
        k_extrap_init<<<face_grid(d, a), blk2(), 0, st>>>(d, a, phi, frac.p[a], valid[a]);
        uint8_t *v0 = valid[a], *v1 = valid1[a];
        for (int it = 0; it < max_steps; it++) {
            k_extrap_step<<<face_grid(d, a), blk2(), 0, st>>>(d, a, u[a], v0, v1, clear_val);
            uint8_t *t = v0;
            v0 = v1;
            v1 = t;
        }
    }
}

void launch_enforce(cudaStream_t st, const Dims &d, const double origin[3], double h, const Faces &old,
                    const Faces &us, const Faces &normal, const Faces &frac, double *const u[3]) {
    Origin og{{origin[0], origin[1], origin[2]}};
    const double invh = 1 / h;  // Grid::m_InvSpacing
    for (int a = 0; a < 3; a++)
        k_enforce<<<face_grid(d, a), blk2(), 0, st>>>(d, a, og, h, invh, old, us, normal, frac.p[a], u[a]);
}

}  // namespace sf
